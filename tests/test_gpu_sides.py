"""The mesh passes at every kind of mesh side, against the CPU oracle: one tile cut so that PM2
and PM3 take sides of 2^a 3^b (the specialised FFT passes, fused planes up to 144 and rows
above) and sides outside the list (the general passes); ghost depths ncb and ngb that do not
match; boxes few enough that the deposit cuts them in z, ragged in every direction; cells of
more than 511 particles (the deposit's 32-bit sums with carries) and subtiles of several
classes, so that the FP64 mass sums and the deposit see class boundaries.

Tolerances (FP32 rounding u = 2^-24):
  * fixed-point density: bit-exact.  FP32 density: a mesh cell is a sum of at most M terms,
    M the particles of the fullest 2x2x2 coarse cells, so within (M + 8) u of itself; PM2 and
    PM3 round each term to a multiple of 2^-40 (M 2^-41 particle masses).
  * potential, velocities and f2max: the bounds that test_gpu_parity.py states and reasons.
  * mass: FP64 sums of FP32 terms, each within 4 u: 1e-6 of the total.
"""
import numpy as np
import pytest

from cube_nu_b200.params import DEPOSIT_FIXED, DEPOSIT_FP32, Params
from tests.helpers import state_from_positions

pytestmark = pytest.mark.gpu

#        ng nnt nns ncb ngb     PM2 side; PM3 sides of the classes that occur
SIDES = [(64, 1, 8, 4, 16),    # 96; 32, 64, 96
         (96, 1, 4, 4, 16),    # 128; 64, 128; PM1 24 (general passes)
         (96, 1, 6, 4, 24),    # 144; 48, 96: ngb deeper than ncb coarse cells
         (144, 1, 6, 6, 24),   # 192; 64, 128
         (192, 1, 8, 8, 32),   # 256; 64, 128
         (128, 2, 8, 4, 16)]   # 96; 32, 64, 96: eight tiles, neighbours across their faces


N = 18001  # particles


def _params(ng, nnt, nns, ncb, ngb, fixed):
    p = Params(ng=ng, nnt=nnt, nns=nns, np_nc=2, ncb=ncb, ngb=ngb, izipx=1 + fixed, box=100.0)
    p.deposit_mode = DEPOSIT_FIXED if fixed else DEPOSIT_FP32
    p.mass_p_cdm = float(p.ng) ** 3 / N
    return p


def _state(p, seed):
    """A sparse background and cells that hold a clump: on a tile's face, and inside; the
    fullest cell of a subtile sets its class (3 from 1536 particles, 4 from 7296)."""
    rng = np.random.default_rng(seed)
    clumps = [1600, 7400] if p.ngp // p.nns == 8 else [1600]
    at = [np.array([0, p.nc // 2, p.nc - 1]), np.array([p.nc // 3, p.nc // 3 + 1, p.nc // 2])]
    X = [c + rng.random((k, 3)) for c, k in zip(at, clumps)]
    X = np.concatenate(X + [rng.random((N - sum(clumps), 3)) * p.nc])
    return state_from_positions(p, X, rng.normal(size=X.shape) * 0.3)


def _fullest_corner(p, rhoc):
    g = np.zeros((p.nc,) * 3, dtype=np.int64)
    c = np.arange(p.ncells)
    l, t = c % p.nt ** 3, c // p.nt ** 3
    co = [(t // p.nnt ** d % p.nnt) * p.nt + l // p.nt ** d % p.nt for d in range(3)]
    g[co[2], co[1], co[0]] = rhoc
    for ax in range(3):
        g = g + np.roll(g, 1, axis=ax)
    return int(g.max())


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("sides", SIDES, ids=lambda s: "-".join(map(str, s)))
def test_meshes_at_every_kind_of_side(oracle_lib, sides, fixed):
    from cube_nu_b200._lib import Context

    p = _params(*sides, fixed)
    st = _state(p, seed=sides[0] + sides[2])
    assert st[3].max() > 511
    ires, _ = oracle_lib.classify(p, st[3])
    fields = [(1, 0, p.nc), (2, p.ntiles - 1, p.ngt)]
    fields += [(3, int(np.flatnonzero(ires == cl)[0]), p.nft(cl)) for cl in np.unique(ires)[:None if fixed else 1]]
    u, m = 2.0 ** -24, _fullest_corner(p, st[3])
    dt, a_mid = 0.2, 0.05
    for level, box, side in fields:
        for what in (0, 1) if fixed else (0,):
            _, ref = oracle_lib.kick(p, st[0], st[1].copy(), st[3], dt, a_mid, fixed=fixed, only=1 << (level - 1),
                                     debug=(level, box, what, side ** 3))
            with Context(p) as ctx:
                ctx.upload(*st)
                ctx.capture(level, box, what)
                ctx.kick(dt, a_mid)
                got = ctx.captured(side ** 3)
            where = "level %d box %d side %d" % (level, box, side)
            if what == 1:
                assert np.abs(got - ref).max() < 2e-5 * np.abs(ref).max(), "potential, " + where
            elif fixed:
                assert np.array_equal(got, ref), "density, " + where
            else:
                bound = (m + 8) * u * ref + m * 2.0 ** -41 * max(1.0, p.mass_p_cdm)
                assert np.all(np.abs(got - ref) <= bound), "density, " + where
    v_ref = st[1].copy()
    out = oracle_lib.kick(p, st[0], v_ref, st[3], dt, a_mid, fixed=fixed)
    with Context(p) as ctx:
        ctx.upload(*st)
        so = ctx.kick(dt, a_mid)
        v = ctx.download()[1]
    dref = v_ref - st[1]
    assert np.abs((v - st[1]) - dref).max() < 2e-4 * np.abs(dref).max()
    for level in (1, 2, 3):
        a, b = getattr(so, "f2max_pm%d" % level), getattr(out, "f2max_pm%d" % level)
        assert abs(a - b) <= 1e-4 * abs(b), level
    if not fixed:
        for a, b in zip((so.mass_pm1, so.mass_pm2, so.mass_pm3), out.mass):
            assert abs(a - b) <= 1e-6 * abs(b)


@pytest.mark.parametrize("izipx,fullest", [(1, 64), (1, 65), (2, 65), (2, 700)])
def test_plain_pp_equals_the_queue(izipx, fullest):
    """The plain form's PP gives a thread to each particle, and its cells of more than 16 to
    the queue's heavy kernel once a cell holds more than 64: on both sides of that line its
    velocities, pairs and largest force are the queue's, bit for bit."""
    from cube_nu_b200._lib import Context

    rng = np.random.default_rng(fullest)
    got = []
    for queue in (False, True):
        p = Params(ng=64, nnt=2, nns=2, np_nc=2, izipx=izipx, box=100.0, deposit_mode=DEPOSIT_FIXED, pp_queue=queue)
        if not got:  # a cell of `fullest`, one of 17, one of 16 beside it, and a background of one to a cell
            cells = [(c, k) for c, k in (((5, 9, 2), fullest), ((7, 7, 8), 17), ((8, 7, 8), 16))]
            X = [np.array(c) + rng.random((k, 3)) for c, k in cells]
            bg = np.stack(np.meshgrid(*[np.arange(p.nc)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
            taken = {c for c, _ in cells}
            bg = np.array([b for b in bg if tuple(b) not in taken])
            X = np.concatenate(X + [bg + rng.random(bg.shape)])
            st = state_from_positions(p, X, rng.normal(size=X.shape) * 0.3)
            assert st[3].max() == fullest
        p.mass_p_cdm = float(p.ng) ** 3 / X.shape[0]
        with Context(p) as ctx:
            if queue:
                for cls in range(4):
                    ctx.pp_shape(cls, 4096, 256, 256)  # every cell light
            ctx.upload(*st)
            so = ctx.kick(0.2, 0.05)
            got.append((ctx.download()[1], so.pp_pairs, so.pp_candidates, so.f2max_pp))
    assert np.array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]


@pytest.mark.parametrize("n,odd", [(16, 0), (48, 0), (18, 1)])
def test_mesh_density_at_row_ends(n, odd):
    """The differentiable step's density with its rows in pairs of cells and, in an array that
    starts on an odd word, cell by cell; particles in every residue of a pair and on the rows'
    ends, where the cells wrap: against a float64 sum, each FP32 term within 4 u of itself and
    M of them to a cell, and the weights' own rounding (u/2 each, three factors)."""
    import torch

    from cube_nu_b200 import adjoint as A

    rng = np.random.default_rng(n)
    x = rng.random((4000, 3)) * n
    x[:2000, 0] = np.mod(rng.integers(-2, 3, 2000) + rng.random(2000), n)
    x = np.minimum(x.astype(np.float32), np.nextafter(np.float32(n), np.float32(0)))
    dpm = A.DPM(n, 1.5, 2.0)
    xd = torch.from_numpy(x).cuda()
    buf = torch.full((n ** 3 + 2,), -1.0, device="cuda")
    torch.cuda.synchronize()
    rho = buf[odd:odd + n ** 3]
    assert rho.data_ptr() % 8 == 4 * odd
    assert dpm._lib.cube_dpm_density(dpm._h, xd.data_ptr(), x.shape[0], rho.data_ptr()) == 0
    dpm.close()
    buf = buf.cpu().numpy()
    assert np.all(buf[:odd] == -1.0) and np.all(buf[odd + n ** 3:] == -1.0)
    got = buf[odd:odd + n ** 3].reshape(n, n, n).astype(np.float64)
    ref, count = np.zeros((n, n, n)), np.zeros((n, n, n), dtype=np.int64)
    f = np.floor(x.astype(np.float64)).astype(np.int64)
    w = x.astype(np.float64) - f
    w = np.stack([0.5 * (1 - w) ** 2, 1 - 0.5 * (1 - w) ** 2 - 0.5 * w ** 2, 0.5 * w ** 2])
    for c in range(3):
        for b in range(3):
            for a in range(3):
                at = tuple((f + np.array([a - 1, b - 1, c - 1]))[:, d] % n for d in (2, 1, 0))
                np.add.at(ref, at, 2.0 * w[a, :, 0] * w[b, :, 1] * w[c, :, 2])
                np.add.at(count, at, 1)
    u = 2.0 ** -24
    assert np.all(np.abs(got - ref) <= (count + 4) * u * ref + 3 * u * count)
    assert abs(got.sum() - 8000.0) < 8000.0 * 4 * u * 27


@pytest.mark.parametrize("n", [64, 162])
def test_force_mesh_at_both_depths(n):
    """The force of the differentiable step where the force mesh takes one cell a thread (64)
    and four along z with a remainder of two (162), against FP64 (the bound of
    test_gpu_adjoint.py's force test)."""
    import torch

    from cube_nu_b200 import adjoint as A
    from tests.test_gpu_adjoint import ref_force

    g = torch.Generator(device="cuda").manual_seed(n)
    x = (torch.rand((20000, 3), generator=g, device="cuda") * n).contiguous()
    dpm = A.DPM(n, 1.5, 8.0)
    green = torch.from_numpy(dpm.green()).double().cuda()
    got = dpm.force(x).double()
    dpm.close()
    ref = ref_force(x.double(), n, 8.0, green)
    assert float((got - ref).norm() / ref.norm()) < 1e-5
