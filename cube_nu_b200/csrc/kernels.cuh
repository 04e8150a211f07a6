// Step kernels (header-only, included once by cube_gpu.cu) for one CUBE image on one B200 (sm_100a).
//
// All particle data stays in the reference's order (tile z,y,x; coarse cell z,y,x;
// arrival).  Ghost cells of the reference (buffer_grid.f90, buffer_particle.f90) are
// periodic copies when nn=1, so every kernel reads neighbour cells through periodic
// cell indexing instead of materialised ghost copies.
#pragma once
#include <type_traits>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "fft.cuh"

namespace cube {

// =================================================================================
// Exclusive scan int32 -> int64 (cell starts); out has n+1 entries.
// =================================================================================
static constexpr int SCAN_T = 256, SCAN_I = 8, SCAN_TILE = SCAN_T * SCAN_I;

__device__ __forceinline__ int64_t warp_incl_scan(int64_t v) {
  for (int o = 1; o < 32; o <<= 1) {
    int64_t u = __shfl_up_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) >= o) v += u;
  }
  return v;
}

// Block-wide exclusive scan of one value per thread; returns exclusive prefix, total in *tot.
__device__ int64_t block_excl_scan(int64_t v, int64_t* tot) {
  __shared__ int64_t ws[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int64_t inc = warp_incl_scan(v);
  if (lane == 31) ws[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    int64_t s = (lane < nw) ? ws[lane] : 0;
    s = warp_incl_scan(s);
    if (lane < nw) ws[lane] = s;
  }
  __syncthreads();
  const int64_t base = (wid > 0) ? ws[wid - 1] : 0;
  *tot = ws[nw - 1];
  __syncthreads();
  return base + inc - v;
}

__global__ void k_scan_tiles(const int32_t* __restrict__ in, int64_t n, int64_t* __restrict__ tile_sums) {
  const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_I;
  int64_t s = 0;
#pragma unroll
  for (int i = 0; i < SCAN_I; ++i)
    if (base + i < n) s += in[base + i];
  int64_t tot;
  block_excl_scan(s, &tot);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = tot;
}

__global__ void k_scan_sums(int64_t* __restrict__ sums, int64_t nt) {
  // single block: exclusive scan of nt tile sums in place
  __shared__ int64_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t b0 = 0; b0 < nt; b0 += blockDim.x) {
    const int64_t i = b0 + threadIdx.x;
    const int64_t v = (i < nt) ? sums[i] : 0;
    int64_t tot;
    const int64_t ex = block_excl_scan(v, &tot);
    if (i < nt) sums[i] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[nt] = carry;
}

__global__ void k_scan_apply(const int32_t* __restrict__ in, int64_t n, const int64_t* __restrict__ tile_sums,
                             int64_t* __restrict__ out, int64_t ntiles) {
  const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_I;
  int64_t v[SCAN_I];
  int64_t s = 0;
#pragma unroll
  for (int i = 0; i < SCAN_I; ++i) {
    v[i] = (base + i < n) ? in[base + i] : 0;
    s += v[i];
  }
  int64_t tot;
  int64_t ex = block_excl_scan(s, &tot) + tile_sums[blockIdx.x];
#pragma unroll
  for (int i = 0; i < SCAN_I; ++i) {
    if (base + i < n) out[base + i] = ex;
    ex += v[i];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = tile_sums[ntiles];
}

inline void exclusive_scan(const int32_t* in, int64_t* out, int64_t n, int64_t* tmp, cudaStream_t s) {
  const int64_t nt = (n + SCAN_TILE - 1) / SCAN_TILE;
  k_scan_tiles<<<(unsigned)nt, SCAN_T, 0, s>>>(in, n, tmp);
  k_scan_sums<<<1, 1024, 0, s>>>(tmp, nt);
  k_scan_apply<<<(unsigned)nt, SCAN_T, 0, s>>>(in, n, tmp, out, nt);
}

// Particle -> storage cell index, from the cell starts.
__global__ void k_fill_pcell(const int64_t* __restrict__ cstart, int64_t ncells, int32_t* __restrict__ pcell) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  for (int64_t i = cstart[c]; i < cstart[c + 1]; ++i) pcell[i] = (int32_t)c;
}

// =================================================================================
// Drift (drift.f90:1-233), bit-exact.
// =================================================================================
// Destination cell, arrival key and count.  The reference scans, per destination
// tile, source cells of the tile's ncb-deep extended region in order
// (ilayer, k, j, i, l) with ilayer=(k-(1-ncb)) mod nlayer (drift.f90:96-115).  The key
// packs that order relative to the destination tile:
//   ilayer:16 | k+ncb-1:8 | j+ncb-1:8 | i+ncb-1:8 | l:24.
// A particle that would move beyond the ghost depth raises CUBE_DEVERR_DRIFT_RANGE (the
// reference stops, drift.f90:64-73) and is kept in its own cell, so the drifted state stays
// a consistent permutation that later kernels can read safely until the host sees the error.
__global__ void k_drift_dest(Geo G, int64_t np, const void* __restrict__ xp, const float* __restrict__ vp,
                             const int32_t* __restrict__ pcell, const int64_t* __restrict__ cstart,
                             const StepDev* __restrict__ sd, int32_t* __restrict__ dest, uint64_t* __restrict__ key,
                             int32_t* __restrict__ count_new, unsigned* err) {
  const int64_t ip = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= np) return;
  const float dt_mid = sd->dt_mid;
  const int nlayer = sd->nlayer;
  const int c = pcell[ip];
  int g[3];
  cell_coords(G, c, g[0], g[1], g[2]);
  const int64_t l = ip - cstart[c];
  int dn[3];
  bool bad = false;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int code = load_code(xp, G.izipx, 3 * ip + d);
    const float p = __fmul_rn(dt_mid, vp[3 * ip + d]);
    const double deltax = (double)__fdiv_rn(p, (float)G.rcs);       // drift.f90:57
    const int li = g[d] % G.nt;                                      // i-1 in the source tile
    const double xq = (double)li + zfrac(code, G);                   // drift.f90:59
    const double ig = ceil(__dadd_rn(xq, deltax));                   // drift.f90:63
    if (!(ig >= (double)(1 - 2 * G.ncb) && ig <= (double)(G.nt + 2 * G.ncb))) bad = true;
    dn[d] = bad ? 0 : (int)ig - (li + 1);
  }
  // Source coordinate (i-1) in the destination tile's frame: the ghost copy that lands
  // in the destination's physical cell is the one at (destination - displacement).  When a
  // tile's ghost region wraps onto itself (nc < nt+2ncb) a cell has two copies there and
  // only this one reaches a physical cell.
  int dst[3], rel[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    dst[d] = wrapi(g[d] + dn[d], G.nc);
    const int dloc = dst[d] % G.nt;
    rel[d] = dloc - dn[d];
    if (rel[d] < -G.ncb || rel[d] >= G.nt + G.ncb) bad = true;  // source outside the dest tile's ghost region
  }
  if (bad) {
    set_err(err, CUBE_DEVERR_DRIFT_RANGE);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      dst[d] = g[d];
      rel[d] = g[d] % G.nt;
    }
  }
  const int64_t dc = cell_index(G, dst[0], dst[1], dst[2]);
  if (!owned_cell(G, dc)) {  // lands in another rank's slab, which keeps it
    dest[ip] = -1;
    return;
  }
  const uint64_t kz = (uint64_t)(rel[2] + G.ncb), ky = (uint64_t)(rel[1] + G.ncb), kx = (uint64_t)(rel[0] + G.ncb);
  const uint64_t il = kz % (uint64_t)nlayer;
  // l < 2^24: a cell holds fewer particles than the capacity check on upload allows
  key[ip] = (il << 48) | (kz << 40) | (ky << 32) | (kx << 24) | (uint64_t)(l & 0xffffff);
  dest[ip] = (int32_t)dc;
  atomicAdd(&count_new[dc], 1);
}

__global__ void k_drift_scatter(int64_t np, const int32_t* __restrict__ dest, const uint64_t* __restrict__ key,
                                const int64_t* __restrict__ cstart_new, int32_t* __restrict__ fill,
                                uint64_t* __restrict__ skey, uint32_t* __restrict__ ssrc) {
  const int64_t ip = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= np) return;
  const int dc = dest[ip];
  if (dc < 0) return;
  const int slot = atomicAdd(&fill[dc], 1);
  const int64_t pos = cstart_new[dc] + slot;
  skey[pos] = key[ip];
  ssrc[pos] = (uint32_t)ip;
}

// Ascending bitonic sort of (key, value) pairs across groups of W lanes (W = 16 or 32);
// lanes pass their index within the group.  Keys are unique; padding lanes hold ~0.
template <int W>
__device__ __forceinline__ void group_bitonic(uint64_t& k, uint32_t& v, int gl) {
#pragma unroll
  for (int size = 2; size <= W; size <<= 1)
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      const uint64_t ok = __shfl_xor_sync(0xffffffffu, k, stride);
      const uint32_t ov = __shfl_xor_sync(0xffffffffu, v, stride);
      const bool up = ((gl & size) == 0);
      const bool lower = ((gl & stride) == 0);
      const bool take = lower ? (up ? (ok < k) : (ok > k)) : (up ? (ok > k) : (ok < k));
      if (take) {
        k = ok;
        v = ov;
      }
    }
}

// Two destination cells per warp, one per 16-lane half: segments of <=16 (nearly all at
// 8 particles per cell) are sorted in registers by the half; segments of 17..32 are then
// sorted by the whole warp, one at a time; longer ones are listed for the block sorter.
// Launch (ncells + 1) / 2 warps.
__global__ void k_drift_sort_small(int64_t ncells, const int32_t* __restrict__ count_new,
                                   const int64_t* __restrict__ cstart_new, uint64_t* __restrict__ skey,
                                   uint32_t* __restrict__ ssrc, int32_t* __restrict__ biglist,
                                   int32_t* __restrict__ nbig) {
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (2 * w >= ncells) return;  // warp-uniform
  const int lane = threadIdx.x & 31;
  const int hl = lane & 15;
  const int64_t c = 2 * w + (lane >> 4);
  const int n = (c < ncells) ? count_new[c] : 0;
  if (n > 32 && hl == 0) biglist[atomicAdd(nbig, 1)] = (int32_t)c;
  const bool small = n > 1 && n <= 16;
  if (__any_sync(0xffffffffu, small)) {
    const int64_t base = small ? cstart_new[c] : 0;
    const bool live = small && hl < n;
    uint64_t k = live ? skey[base + hl] : ~0ull;
    uint32_t v = live ? ssrc[base + hl] : 0u;
    group_bitonic<16>(k, v, hl);
    if (live) {
      skey[base + hl] = k;
      ssrc[base + hl] = v;
    }
  }
  unsigned mid = __ballot_sync(0xffffffffu, n > 16 && n <= 32 && hl == 0);
  while (mid) {
    const int h = __ffs(mid) - 1;
    mid &= mid - 1;
    const int64_t cm = 2 * w + (h >> 4);
    const int nm = count_new[cm];
    const int64_t base = cstart_new[cm];
    uint64_t k = (lane < nm) ? skey[base + lane] : ~0ull;
    uint32_t v = (lane < nm) ? ssrc[base + lane] : 0u;
    group_bitonic<32>(k, v, lane);
    if (lane < nm) {
      skey[base + lane] = k;
      ssrc[base + lane] = v;
    }
  }
}

// Block per long segment: bitonic sort in shared memory (keys are unique), which holds
// max_seg rounded up to a power of two keys and values (drift_sort_smem).  Segments
// longer than max_seg are listed in hugelist for k_drift_rank_huge.
__global__ void k_drift_sort_big(const int32_t* __restrict__ biglist, const int32_t* __restrict__ nbig,
                                 const int32_t* __restrict__ count_new, const int64_t* __restrict__ cstart_new,
                                 uint64_t* __restrict__ skey, uint32_t* __restrict__ ssrc, int max_seg,
                                 int32_t* __restrict__ hugelist, int32_t* __restrict__ nhuge) {
  extern __shared__ uint64_t smk[];
  const int nb = *nbig;
  for (int b = blockIdx.x; b < nb; b += gridDim.x) {  // block-uniform loop over the listed cells
  __syncthreads();  // the previous segment's write-out is done with the shared arrays
  const int c = biglist[b];
  const int n = count_new[c];
  if (n > max_seg) {
    if (threadIdx.x == 0) hugelist[atomicAdd(nhuge, 1)] = c;
    continue;
  }
  int m = 1;
  while (m < n) m <<= 1;  // m <= max_seg rounded up to a power of two: the keys' capacity
  int cap = 1;
  while (cap < max_seg) cap <<= 1;
  uint32_t* smv = reinterpret_cast<uint32_t*>(smk + cap);
  const int64_t base = cstart_new[c];
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    smk[i] = (i < n) ? skey[base + i] : ~0ull;
    smv[i] = (i < n) ? ssrc[base + i] : 0u;
  }
  __syncthreads();
  for (int size = 2; size <= m; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int j = i ^ stride;
        if (j > i) {
          const bool up = ((i & size) == 0);
          const uint64_t a = smk[i], b = smk[j];
          if ((a > b) == up) {
            smk[i] = b;
            smk[j] = a;
            const uint32_t t = smv[i];
            smv[i] = smv[j];
            smv[j] = t;
          }
        }
      }
      __syncthreads();
    }
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    skey[base + i] = smk[i];
    ssrc[base + i] = smv[i];
  }
  }
}

// Dynamic shared memory of k_drift_sort_big for a given max_seg.
inline size_t drift_sort_smem(int max_seg) {
  size_t cap = 1;
  while (cap < (size_t)max_seg) cap <<= 1;
  return cap * 12;
}

// Segments longer than the shared-memory sorter holds (dense halo cores at late times):
// the rank of each key is the number of smaller keys in its segment (keys are unique), so
// it is written straight to its sorted place in (tkey, tsrc); k_drift_copy_huge copies the
// segment back.  Every block walks the listed cells and takes the tiles of 512 elements
// with index = blockIdx.x mod gridDim.x; the segment's keys stream through shared memory in
// chunks.  Quadratic in the segment length (0.3 ms for 5e4 keys), and only such cells run.
constexpr int HUGE_T = 512, HUGE_CHUNK = 4096;
__global__ void __launch_bounds__(HUGE_T) k_drift_rank_huge(const int32_t* __restrict__ hugelist,
                                                            const int32_t* __restrict__ nhuge,
                                                            const int32_t* __restrict__ count_new,
                                                            const int64_t* __restrict__ cstart_new,
                                                            const uint64_t* __restrict__ skey,
                                                            const uint32_t* __restrict__ ssrc,
                                                            uint64_t* __restrict__ tkey, uint32_t* __restrict__ tsrc) {
  __shared__ uint64_t chunk[HUGE_CHUNK];
  const int nh = *nhuge;
  int item = 0;  // running tile index over all listed cells
  for (int h = 0; h < nh; ++h) {
    const int c = hugelist[h];
    const int n = count_new[c];
    const int64_t base = cstart_new[c];
    const int ntile = (n + HUGE_T - 1) / HUGE_T;
    for (int t = 0; t < ntile; ++t, ++item) {
      if (item % gridDim.x != blockIdx.x) continue;  // block-uniform
      const int i = t * HUGE_T + threadIdx.x;
      const bool live = i < n;
      const uint64_t k = live ? skey[base + i] : 0ull;
      int rank = 0;
      for (int j0 = 0; j0 < n; j0 += HUGE_CHUNK) {
        const int cnt = min(HUGE_CHUNK, n - j0);
        __syncthreads();
        for (int j = threadIdx.x; j < cnt; j += HUGE_T) chunk[j] = skey[base + j0 + j];
        __syncthreads();
        if (live)
          for (int j = 0; j < cnt; ++j) rank += chunk[j] < k;
      }
      if (live) {
        tkey[base + rank] = k;
        tsrc[base + rank] = ssrc[base + i];
      }
    }
  }
}

__global__ void k_drift_copy_huge(const int32_t* __restrict__ hugelist, const int32_t* __restrict__ nhuge,
                                  const int32_t* __restrict__ count_new, const int64_t* __restrict__ cstart_new,
                                  const uint64_t* __restrict__ tkey, const uint32_t* __restrict__ tsrc,
                                  uint64_t* __restrict__ skey, uint32_t* __restrict__ ssrc) {
  const int nh = *nhuge;
  for (int h = 0; h < nh; ++h) {
    const int c = hugelist[h];
    const int64_t base = cstart_new[c];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count_new[c];
         i += (int64_t)gridDim.x * blockDim.x) {
      skey[base + i] = tkey[base + i];
      ssrc[base + i] = tsrc[base + i];
    }
  }
}

// New arrays in the sorted order, with the ZIPX update xp+nint(dt_mid*vp/(x_res*ratio_cs))
// in the integer kind (drift.f90:117).
__global__ void k_drift_gather(Geo G, int64_t np, const uint32_t* __restrict__ ssrc, const int32_t* __restrict__ dest,
                               const void* __restrict__ xp, const float* __restrict__ vp,
                               const int64_t* __restrict__ pid, const StepDev* __restrict__ sd, void* __restrict__ xo,
                               float* __restrict__ vo, int64_t* __restrict__ po, int32_t* __restrict__ pcell_o,
                               const int64_t* __restrict__ ntot) {
  // ntot: particles the drift kept (fewer than np when some left this rank's slab)
  const int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= (ntot ? *ntot : np)) return;
  const float dt_mid = sd->dt_mid;
  const int64_t src = ssrc[pos];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float v = vp[3 * src + d];
    const int code = load_code(xp, G.izipx, 3 * src + d);
    const long long dn = llround(__dmul_rn((double)__fmul_rn(dt_mid, v), G.inv_step));
    store_code(xo, G.izipx, 3 * pos + d, (int)(code + (int)dn));
    vo[3 * pos + d] = v;
  }
  if (pid) po[pos] = pid[src];  // null: the ids are permuted later (k_permute_ids)
  pcell_o[pos] = dest[src];
}

// The drift's permutation applied to the particle ids on their own: ids_out[pos] =
// ids_in[ssrc[pos]], for a caller whose ids arrive after the rest of the drift has run.
__global__ void k_permute_ids(int64_t np, const uint32_t* __restrict__ ssrc, const int64_t* __restrict__ ids_in,
                              int64_t* __restrict__ ids_out) {
  const int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (pos < np) ids_out[pos] = ids_in[ssrc[pos]];
}

// =================================================================================
// Deposit (particle_mesh.f90:20-109, kick.f90:611-691).
// =================================================================================

// Mass sums of the deposited density over the physical cells of a level (the reference
// forms them in real(8): particle_mesh.f90:106 testrho, kick.f90:687-688 ptotal), in
// particle units.  The fixed-point form sums the int64 contributions exactly (order
// independent, so deterministic); the FP32 form sums the float weights in FP64.  Warps
// add into one of MASS_SLOTS accumulators picked by block, each on its own 128-byte line
// (MASS_STRIDE words apart), so the atomics spread over many L2 lines; the host adds the
// slots.  A fixed-point slot is 128 bits: word 0 takes the sums, word 1 counts its carries
// (2^40 per particle overflows 64 bits beyond 2^24 particles).
constexpr int MASS_SLOTS = 64, MASS_STRIDE = 16;

__device__ __forceinline__ void warp_sum_to(unsigned long long v, unsigned long long* out) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v && out) {
    unsigned long long* slot = out + (blockIdx.x & (MASS_SLOTS - 1)) * MASS_STRIDE;
    const unsigned long long old = atomicAdd(slot, v);
    if (old + v < old) atomicAdd(slot + 1, 1ull);
  }
}

__device__ __forceinline__ void warp_sum_to(double v, double* out) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v != 0.0 && out) atomicAdd(out + (blockIdx.x & (MASS_SLOTS - 1)) * MASS_STRIDE, v);
}

// One thread's running mass sum in the arithmetic of its deposit form.
template <bool FIXED>
struct MassAcc {
  using T = typename std::conditional<FIXED, unsigned long long, double>::type;
  T v = 0;
  __device__ __forceinline__ void add(float w) {
    if constexpr (FIXED) v += fixed40(w);
    else v += (double)w;
  }
  // out: MASS_SLOTS accumulators of type T (nullptr: no sum wanted)
  __device__ __forceinline__ void flush(void* out) { warp_sum_to(v, static_cast<T*>(out)); }
};

// PM1 deposit.  A particle of coarse cell g has floor(xpos) = g, so every particle of the cell
// deposits into the same 27 cells, and particles are stored cell by cell.  A warp takes 32
// consecutive particles: each lane works out one particle's weights, then lane o < 27 takes
// mesh cell o of the 27 and goes over the 32 particles, summing its contribution (int64 fixed
// point, or FP32) while the coarse cell stays the same and adding the sum with one reduction
// when it changes.  Integer sums do not depend on the order.  Sums by shuffles (27 segmented
// suffix sums of 64-bit values) took three times the instructions: 0.92 ms for 256^3 particles
// at 8 a cell, 0.69 now.
template <bool FIXED>
__global__ void __launch_bounds__(256) k_deposit_pm1(Geo G, int64_t np, const void* __restrict__ xp,
                                                     const int32_t* __restrict__ pcell, void* __restrict__ rho, int pr,
                                                     int64_t pl, void* msum) {
  using T = typename std::conditional<FIXED, unsigned long long, float>::type;
  __shared__ float ws[8][9][33];
  T* const mesh = static_cast<T*>(rho);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t p0 = (int64_t)blockIdx.x * blockDim.x + wid * 32;
  if (p0 >= np) return;  // warp-uniform
  const int n = (int)min((int64_t)32, np - p0);
  const int64_t ip = p0 + min(lane, n - 1);
  const int cell = pcell[ip];
  int g[3];
  cell_coords(G, cell, g[0], g[1], g[2]);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    float w[3];
    tsc_weights((double)g[d] + zfrac(load_code(xp, G.izipx, 3 * ip + d), G), w);  // floor(xpos) = g
#pragma unroll
    for (int a = 0; a < 3; ++a) ws[wid][3 * d + a][lane] = w[a];
  }
  __syncwarp();
  const int o = min(lane, 26), a1 = o % 3, a2 = o / 3 % 3, a3 = o / 9;
  const float *wx = ws[wid][a1], *wy = ws[wid][3 + a2], *wz = ws[wid][6 + a3];
  MassAcc<FIXED> mass;
  T sum = 0;
  for (int p = 0; p < n; ++p) {
    const float ww = __fmul_rn(__fmul_rn(wx[p], wy[p]), wz[p]);
    if constexpr (FIXED) {
      sum += fixed40(ww);
    } else {
      sum += ww;
      if (lane < 27) mass.add(ww);
    }
    const int here = __shfl_sync(0xffffffffu, cell, p), next = __shfl_sync(0xffffffffu, cell, (p + 1) & 31);
    if (p + 1 == n || next != here) {  // the run ends
      const int gx = __shfl_sync(0xffffffffu, g[0], p), gy = __shfl_sync(0xffffffffu, g[1], p),
                gz = __shfl_sync(0xffffffffu, g[2], p);
      if (lane < 27) {
        atomicAdd(mesh + (int64_t)wrap1(gz - 1 + a3, G.nc) * pl + (int64_t)wrap1(gy - 1 + a2, G.nc) * pr +
                      wrap1(gx - 1 + a1, G.nc), sum);
        if constexpr (FIXED) mass.v += sum;
      }
      sum = 0;
    }
  }
  mass.flush(msum);
}

// Candidate subtiles along one dimension (PM3 nloop=1): own subtile and, in the
// first/last coarse cell of a subtile, the neighbour subtile (possibly in the
// neighbour tile).  Returns count; writes tile, subtile, and local coordinate (i-1)
// in that tile.
__device__ __forceinline__ int sub_cands(const Geo& G, int g, int* t, int* u, int* li) {
  const int tt = g / G.nt, l = g - tt * G.nt;
  const int uu = l / G.ntt, r = l - uu * G.ntt;
  t[0] = tt;
  u[0] = uu;
  li[0] = l;
  // With ntt >= 2 at most one of the two faces is adjacent; constant slot indices keep
  // the caller's arrays in registers.
  const bool lo = r == 0, hi = r == G.ntt - 1;
  if (lo) {
    const bool wrap = uu == 0;
    t[1] = wrap ? wrapi(tt - 1, G.nnt) : tt;
    u[1] = wrap ? G.nns - 1 : uu - 1;
    li[1] = wrap ? l + G.nt : l;
  } else {
    const bool wrap = uu == G.nns - 1;
    t[1] = wrap ? wrapi(tt + 1, G.nnt) : tt;
    u[1] = wrap ? 0 : uu + 1;
    li[1] = wrap ? l - G.nt : l;
  }
  return (lo || hi) ? 2 : 1;
}

__device__ __forceinline__ int subtile_id(const Geo& G, const int t[3], const int u[3]) {
  const int T = (t[2] * G.nnt + t[1]) * G.nnt + t[0];
  return ((T * G.nns + u[2]) * G.nns + u[1]) * G.nns + u[0];
}

// PM3 meshes of one class: slot = box_slot[subtile] (or -1), mesh [slot][nft^3];
// refined index i maps to array i-(1-nfb).
// xpos of kick.f90:628-629, ((l + f) * ratio_cs) / gridsize - u * nfp in real(8), with
// gridsize = real(1/rsf, 4).  For rsf a power of two gridsize is exact and the division
// equals the multiplication by rsf (exact scaling by a power of two).
__device__ __forceinline__ double pm3_xpos(double lf, const Geo& G, double gs, int rsf, int unfp) {
  const double a = lf * (double)G.rcs;
  return (((rsf & (rsf - 1)) == 0) ? a * (double)rsf : a / gs) - (double)unfp;
}

// PM3 mass over the physical cells of every subtile box (kick.f90:687-688 ptotal), summed
// per particle: for each box the deposit puts the particle in (its own subtile and, in the
// first or last coarse cell of a subtile, the neighbour; each at that box's class), the
// contributions that land in the box's physical cells.  The deposit adds exactly these
// contributions to those cells, so with the fixed-point deposit this is the mesh sum
// itself, exactly; the deposit kernels need no extra work for it.
// A neighbour box of the same class has the own box's weights shifted by whole cells, so
// its physical contributions are the own box's contributions that leave the own physical
// region in its direction: the sum of all 27 own contributions covers both, and
// k_interp_pm3 adds it while it holds the weights.  Only a neighbour of another class (a
// class boundary, rare) needs its own weights: its share of the 27 is replaced by its
// physical contributions at its class (k_mass_pm3).
template <bool FIXED>
__device__ __forceinline__ void mass_box(const Geo& G, int iapm, const double lf[3], const int u[3], int i2[3],
                                         float w[3][3]) {
  const int rsf = rsf_of(iapm), nfp = G.nfp[iapm];
  const double gs = (double)(1.f / (float)rsf);
#pragma unroll
  for (int d = 0; d < 3; ++d) i2[d] = tsc_weights(pm3_xpos(lf[d], G, gs, rsf, u[d] * nfp), w[d]);
}

// direction (-1, 0, +1) of 0-based cell index i relative to the physical range 0..nfp-1
__device__ __forceinline__ int mass_dir(int i, int nfp) { return i < 0 ? -1 : (i >= nfp ? 1 : 0); }

// The class-boundary part.  A cell in a face layer of its subtile whose neighbour subtile
// across that face has another class corrects the own-box sums that k_interp_pm3 added for
// its particles.  A block looks at gpb groups of 32 consecutive coarse cells, one cell per
// thread, and its threads then share out the particles of a group's cells to correct (a
// prefix of the counts and a binary search), so a cell of tens of thousands of particles is
// not walked by one thread: that made the kernel as long as its fullest boundary cell, 112 ms
// of a 147 ms kick of 128^3 clustered particles (largest cell 3e4), 0.2 ms now.  A group's
// sum is added to the mass slots as one value.
constexpr int MASS3_T = 256;
template <bool FIXED>
__global__ void __launch_bounds__(MASS3_T) k_mass_pm3(Geo G, const int64_t* __restrict__ cstart,
                                                      const void* __restrict__ xp, const int32_t* __restrict__ ires,
                                                      int gpb, void* msum) {
  using Acc = typename MassAcc<FIXED>::T;
  __shared__ unsigned flags[MASS3_T / 32];  // cells to correct, a bit each, per group
  __shared__ int64_t pre[33];               // prefix of their particle counts
  __shared__ int32_t list[32];
  __shared__ Acc part[MASS3_T / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t cell0 = (int64_t)blockIdx.x * gpb * 32;
  if (wid < gpb) {
    const int64_t cell = cell0 + threadIdx.x;
    bool any = false;
    if (cell < G.ncells && owned_cell(G, cell) && cstart[cell + 1] > cstart[cell]) {
      int g[3], tc[3][2], uc[3][2], lc[3][2], nca[3];
      cell_coords(G, cell, g[0], g[1], g[2]);
#pragma unroll
      for (int d = 0; d < 3; ++d) nca[d] = sub_cands(G, g[d], tc[d], uc[d], lc[d]);
      if (nca[0] * nca[1] * nca[2] > 1) {
        const int t0[3] = {tc[0][0], tc[1][0], tc[2][0]}, u0[3] = {uc[0][0], uc[1][0], uc[2][0]};
        const int own = ires[subtile_id(G, t0, u0)];
        for (int cz = 0; cz < nca[2]; ++cz)
          for (int cy = 0; cy < nca[1]; ++cy)
            for (int cx = 0; cx < nca[0]; ++cx) {
              const int t[3] = {tc[0][cx], tc[1][cy], tc[2][cz]}, u[3] = {uc[0][cx], uc[1][cy], uc[2][cz]};
              any |= ires[subtile_id(G, t, u)] != own;
            }
      }
    }
    const unsigned bits = __ballot_sync(0xffffffffu, any);
    if (lane == 0) flags[wid] = bits;
  }
  __syncthreads();
  for (int grp = 0; grp < gpb; ++grp) {
  const unsigned bits = flags[grp];
  if (bits == 0) continue;  // block-uniform
  const int nl = __popc(bits);
  __syncthreads();  // list, pre and part are free again
  if (wid == 0) {
    const bool mine = (bits >> lane) & 1u;
    const int r = __popc(bits & ((1u << lane) - 1u));
    const int64_t cell = cell0 + grp * 32 + lane;
    const int64_t cnt = mine ? cstart[cell + 1] - cstart[cell] : 0;
    const int64_t incl = warp_incl_scan(cnt);
    if (mine) {
      list[r] = (int32_t)cell;
      pre[r] = incl - cnt;
    }
    if (lane == 31) pre[nl] = incl;
  }
  __syncthreads();
  const int64_t total = pre[nl];
  MassAcc<FIXED> mass;
  for (int64_t v = threadIdx.x; v < total; v += MASS3_T) {
    int lo = 0, hi = nl;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (pre[mid] <= v) lo = mid;
      else hi = mid;
    }
    const int64_t ip = cstart[list[lo]] + (v - pre[lo]);
    int g[3], tc[3][2], uc[3][2], lc[3][2], nca[3];
    cell_coords(G, list[lo], g[0], g[1], g[2]);
#pragma unroll
    for (int d = 0; d < 3; ++d) nca[d] = sub_cands(G, g[d], tc[d], uc[d], lc[d]);
    const int t0[3] = {tc[0][0], tc[1][0], tc[2][0]}, u0[3] = {uc[0][0], uc[1][0], uc[2][0]};
    const int own = ires[subtile_id(G, t0, u0)];
    const int nfp0 = G.nfp[own];
    double f[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) f[d] = zfrac(load_code(xp, G.izipx, 3 * ip + d), G);
    const double lf0[3] = {(double)lc[0][0] + f[0], (double)lc[1][0] + f[1], (double)lc[2][0] + f[2]};
    int i2[3];
    float w[3][3];
    mass_box<FIXED>(G, own, lf0, u0, i2, w);
    for (int cz = 0; cz < nca[2]; ++cz)
      for (int cy = 0; cy < nca[1]; ++cy)
        for (int cx = 0; cx < nca[0]; ++cx) {
          if (cx + cy + cz == 0) continue;
          const int t[3] = {tc[0][cx], tc[1][cy], tc[2][cz]};
          const int u[3] = {uc[0][cx], uc[1][cy], uc[2][cz]};
          const int nb = ires[subtile_id(G, t, u)];
          if (nb == own) continue;
          int dir[3];
          const int cc[3] = {cx, cy, cz};
#pragma unroll
          for (int d = 0; d < 3; ++d)  // sub_cands: the first coarse cell of a subtile reaches down, the last up
            dir[d] = cc[d] == 0 ? 0 : ((lc[d][0] % G.ntt) == 0 ? -1 : 1);
          // the own contributions in that direction leave the sum ...
          MassAcc<FIXED> sub;
#pragma unroll
          for (int a3 = 0; a3 < 3; ++a3)
#pragma unroll
            for (int a2 = 0; a2 < 3; ++a2)
#pragma unroll
              for (int a1 = 0; a1 < 3; ++a1)
                if (mass_dir(i2[0] - 2 + a1, nfp0) == dir[0] && mass_dir(i2[1] - 2 + a2, nfp0) == dir[1] &&
                    mass_dir(i2[2] - 2 + a3, nfp0) == dir[2])
                  sub.add(__fmul_rn(__fmul_rn(w[0][a1], w[1][a2]), w[2][a3]));
          mass.v -= sub.v;
          // ... and the neighbour's own physical contributions at its class come in
          const double lf[3] = {(double)lc[0][cx] + f[0], (double)lc[1][cy] + f[1], (double)lc[2][cz] + f[2]};
          int j2[3];
          float v3[3][3];
          mass_box<FIXED>(G, nb, lf, u, j2, v3);
          const int nfp = G.nfp[nb];
#pragma unroll
          for (int a3 = 0; a3 < 3; ++a3)
#pragma unroll
            for (int a2 = 0; a2 < 3; ++a2)
#pragma unroll
              for (int a1 = 0; a1 < 3; ++a1)
                if ((unsigned)(j2[0] - 2 + a1) < (unsigned)nfp && (unsigned)(j2[1] - 2 + a2) < (unsigned)nfp &&
                    (unsigned)(j2[2] - 2 + a3) < (unsigned)nfp)
                  mass.add(__fmul_rn(__fmul_rn(v3[0][a1], v3[1][a2]), v3[2][a3]));
        }
  }
  for (int o = 16; o > 0; o >>= 1) mass.v += __shfl_xor_sync(0xffffffffu, mass.v, o);
  if (lane == 0) part[wid] = mass.v;
  __syncthreads();
  if (wid == 0) {
    MassAcc<FIXED> sum;
    if (lane < MASS3_T / 32) sum.v = part[lane];
    sum.flush(msum);
  }
  }
}

// Groups of 32 cells per block of k_mass_pm3: one where the box has few cells (at most 2^18,
// a few blocks per SM), so that its full cells spread over the SMs; eight (a cell per
// thread) where most blocks only look.
inline int mass3_groups(int64_t ncells) { return ncells <= (1 << 18) ? 1 : MASS3_T / 32; }

// =================================================================================
// PM2 and PM3 deposit, owner-computes, both deposit forms.  A box (a PM2 tile or a PM3
// subtile) is S coarse cells a side and a halo of `halo`, q mesh cells a coarse cell, and its
// mesh is padded by `pad` cells (halo*q, unless ngb says otherwise): the particles of coarse
// cell k (relative to the box, -halo .. S+halo-1) lie in array cells k*q+pad .. +q-1 and reach
// one cell further.  A block owns a column of cx x cy cells of a
// box and planes [p0, p1) of it, and walks the coarse layers along z once: the contributions
// of a layer's particles are summed in shared memory, in a ring of the q+2 planes a layer
// reaches, and the planes no later layer reaches are written out (zeros included) and their
// slots cleared.  So a particle is looked at by the columns it touches only (1.4 to 2.5 times
// as a whole), the mesh needs no memset, and nothing is read back.
//
// Sums are int64 in units of 2^-40, round(w * 2^40) per contribution, so they are exact and
// independent of the order; cells are written as the float they round to (unscaled; the FFT
// multiplies by the particle mass).  Where no coarse cell the part reads holds more than
// DEPB_CELL particles, a contribution is added as two independent 32-bit halves, a multiple
// of 2^20 and a signed remainder, made by adding and subtracting 1.5 * 2^23 (round to
// nearest) instead of a 64-bit conversion.  Else the low word is added first and its carry
// goes into the high word: the 64-bit shared-memory atomic is a loop of compare-and-swap,
// which made tiles with 64 particles a cell take 2.5 times as long.
//
// The halves lie in arrays of their own, so that a warp's additions fall on all 32 banks and
// the write-out reads and clears them without conflicts (side by side, bank conflicts took
// half of the shared-memory pipe's time, which was 72% busy).  One region of 24^3 cells per block, which looked at 4.6 times
// its particles and took the whole 27-cell loop in nearly every warp, took 4.64 ms for 512
// boxes of 144^3, 3.13 now, and the PM2 reductions into memory 2.19 ms for eight of 288^3,
// 1.55 now.
// =================================================================================
constexpr int DEPB_T = 320, DEPB_SEG = 96;
constexpr int DEPB_SMEM = 96 * 1024;  // ring of one block: two blocks per SM
// A cell takes contributions from 2^3 coarse cells (3^3 when a mesh cell is as large as one):
// with at most 4095 of them, remainders of at most 2^19 stay below 2^31.
constexpr int DEPB_CELL = 511, DEPB_CELL_Q1 = 151;

struct DepBox {
  int S, halo, q, pad, n;        // coarse cells, halo, mesh cells per coarse cell, padding and side of the mesh
  int iapm;                      // PM3 class, 0 for PM2
  int cx, cy, cz, ncx, ncy, ncz;  // cells of a block's part and the parts per dimension
};

__device__ __forceinline__ int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

template <typename CODE>
__global__ void __launch_bounds__(DEPB_T, 2) k_deposit_box(Geo G, DepBox B, const CODE* __restrict__ xp,
                                                           const int32_t* __restrict__ pcell,
                                                           const int64_t* __restrict__ cstart,
                                                           const int32_t* __restrict__ box_sub, int box0,
                                                           float* __restrict__ rho, int pr, int64_t pl, bool fixed,
                                                           void* msum) {
  extern __shared__ __align__(16) int ring[];  // low words [q+2][cy][cx], then the high words
  __shared__ int64_t seg_ip[2][DEPB_SEG];                     // a segment's first particle,
  __shared__ int32_t seg_cell[2][DEPB_SEG], seg_k[2][DEPB_SEG], seg_pre[2][DEPB_SEG + 1];  // first cell, its k, prefix
  __shared__ int dense;
  const int tid = threadIdx.x;
  const int nparts = B.ncx * B.ncy * B.ncz;
  const int64_t j = blockIdx.x / nparts;
  const int part = (int)(blockIdx.x - j * nparts);
  // origin of the box in coarse cells
  int org[3], u[3] = {0, 0, 0};
  if (box_sub) {  // a class list of subtiles; -1 pads it beyond its count (the slot is never read)
    const int s = box_sub[j];
    if (s < 0) return;
    const int nns3 = G.nns * G.nns * G.nns, T = s / nns3, f = s - T * nns3;
    u[0] = f % G.nns;
    u[1] = (f / G.nns) % G.nns;
    u[2] = f / (G.nns * G.nns);
    org[0] = (T % G.nnt) * G.nt + u[0] * G.ntt;
    org[1] = ((T / G.nnt) % G.nnt) * G.nt + u[1] * G.ntt;
    org[2] = (T / (G.nnt * G.nnt)) * G.nt + u[2] * G.ntt;
  } else {
    const int T = box0 + (int)j;
    org[0] = (T % G.nnt) * G.nt;
    org[1] = ((T / G.nnt) % G.nnt) * G.nt;
    org[2] = (T / (G.nnt * G.nnt)) * G.nt;
  }
  const int q = B.q, rd = q + 2, cx = B.cx, cy = B.cy;
  const int hi_at = rd * cy * cx;  // offset of the high words (a multiple of 4)
  const int ox = (part % B.ncx) * cx, oy = ((part / B.ncx) % B.ncy) * cy, p0 = (part / (B.ncx * B.ncy)) * B.cz;
  const int ex = min(cx, B.n - ox), ey = min(cy, B.n - oy), p1 = min(B.n, p0 + B.cz);
  // coarse cells l = k + halo whose particles can reach the part: cells l*q+off-1 .. l*q+off+q
  const int off = B.pad - B.halo * q, nl = B.S + 2 * B.halo;
  const int kx0 = max(0, floor_div(ox - off - 1, q)) - B.halo, kx1 = min(nl - 1, floor_div(ox + ex - off, q)) - B.halo;
  const int ky0 = max(0, floor_div(oy - off - 1, q)) - B.halo, ky1 = min(nl - 1, floor_div(oy + ey - off, q)) - B.halo;
  const int l0 = min(nl - 1, max(0, floor_div(p0 - off - 1, q))), l1 = max(l0, min(nl - 1, floor_div(p1 - off, q)));
  const int nseg = 3 * max(0, ky1 - ky0 + 1);  // per layer: rows of cells, cut where they leave the box's own cells
  auto segment = [&](int i, int l, int& cell, int& kx) {  // first cell and k of segment i; returns its cells
    const int row = i / 3, piece = i - 3 * row;
    const int lo = piece == 0 ? kx0 : piece == 1 ? max(kx0, 0) : max(kx0, B.S);
    const int hi = piece == 0 ? min(kx1, -1) : piece == 1 ? min(kx1, B.S - 1) : kx1;
    kx = lo;
    if (lo > hi) return 0;
    cell = (int)cell_index(G, org[0] + lo, org[1] + ky0 + row, org[2] + l - B.halo);
    return hi - lo + 1;
  };
  auto table = [&](int buf, int l) {  // one warp: the segments of layer l
    const int lane = tid & 31;
    int carry = 0;
    for (int i0 = 0; i0 < nseg; i0 += 32) {
      const int i = i0 + lane;
      int cell = 0, kx = 0, cnt = 0;
      int64_t ip = 0;
      if (i < nseg) {
        const int m = segment(i, l, cell, kx);
        if (m) {
          ip = cstart[cell];
          cnt = (int)(cstart[cell + m] - ip);
        }
      }
      int incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (i < nseg) {
        seg_ip[buf][i] = ip;
        seg_cell[buf][i] = cell;
        seg_k[buf][i] = (kx + B.halo) | ((i / 3 + ky0 + B.halo) << 16);
        seg_pre[buf][i + 1] = carry + incl;
      }
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) seg_pre[buf][0] = 0;
  };
  if (tid == 0) dense = 0;
  {
    int4* z = reinterpret_cast<int4*>(ring);
    for (int i = tid; i < rd * cy * cx / 2; i += DEPB_T) z[i] = make_int4(0, 0, 0, 0);
  }
  __syncthreads();
  for (int i = tid; i < (l1 - l0 + 1) * nseg; i += DEPB_T) {
    const int l = i / nseg;
    int cell, kx;
    const int m = segment(i - l * nseg, l0 + l, cell, kx);
    for (int k = 0; k < m; ++k)
      if (cstart[cell + k + 1] - cstart[cell + k] > (q > 1 ? DEPB_CELL : DEPB_CELL_Q1)) dense = 1;
  }
  if (tid < 32) table(0, l0);
  __syncthreads();
  const bool split = dense == 0;
  const bool pow2 = (q & (q - 1)) == 0;
  const int rsf = B.iapm ? rsf_of(B.iapm) : 1;
  const double gs = (double)(1.f / (float)rsf);
  const int bits = 8 * (int)sizeof(CODE);
  const float M = 12582912.f;  // 1.5 * 2^23
  // write-out: a thread's 4 cells of a plane, planes dealt to groups of threads
  const int cxq = cx / 4, per = cxq * cy, ngrp = max(1, DEPB_T / per), gstep = ngrp % rd;
  int done = p0;  // planes written
  unsigned long long mloc = 0;
  for (int l = l0; l <= l1; ++l) {
    const int buf = (l - l0) & 1;
    if (tid < 32 && l < l1) table(buf ^ 1, l + 1);
    const int total = seg_pre[buf][nseg];
    const int zb = l * q + off - 1;  // first plane the layer reaches; the last is zb + q + 1
    const int zslot = (zb % rd + rd) % rd;
    auto visits = [&](auto split_tag) {
      constexpr bool SPLIT = decltype(split_tag)::value;
      for (int v = tid; v < total; v += DEPB_T) {
        int lo = 0, hi = nseg;
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (seg_pre[buf][mid] <= v) lo = mid;
          else hi = mid;
        }
        const int64_t ip = seg_ip[buf][lo] + (v - seg_pre[buf][lo]);
        const int kk = seg_k[buf][lo];
        const int k[3] = {(kk & 0xffff) + (pcell[ip] - seg_cell[buf][lo]), kk >> 16, l};  // k + halo
        int c0[3];  // part-local cell of the footprint's first weight
        float w[3][3];
        const int o[3] = {ox, oy, zb};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const unsigned code = (unsigned)xp[3 * ip + d];
          if (pow2) {
            // (code + 1/2) q / 2^bits: whole part and, exactly, the rest
            const unsigned t = (2u * code + 1u) * (unsigned)q;
            const float f = (float)(t & ((2u << bits) - 1u)) * (0.5f / (float)(1u << bits));
            const float a = __fsub_rn(1.f, f);
            w[d][0] = __fmul_rn(__fmul_rn(a, a), 0.5f);
            w[d][2] = __fmul_rn(__fmul_rn(f, f), 0.5f);
            w[d][1] = __fsub_rn(__fsub_rn(1.f, w[d][0]), w[d][2]);
            c0[d] = k[d] * q + off + (int)(t >> (bits + 1)) - 1 - o[d];
          } else {
            const int nfp = B.S * q;
            const double xpos = pm3_xpos((double)(u[d] * G.ntt + k[d] - B.halo) + zfrac((int)code, G), G, gs, rsf, u[d] * nfp);
            c0[d] = tsc_weights(xpos, w[d]) + B.pad - 2 - o[d];  // kick.f90:628-629
          }
        }
        if (c0[0] + 2 < 0 || c0[0] >= ex || c0[1] + 2 < 0 || c0[1] >= ey) continue;
#pragma unroll
        for (int a3 = 0; a3 < 3; ++a3) {
          const int zr = c0[2] + a3;  // 0 .. q+1: plane zb + zr
          if (zb + zr < p0 || zb + zr >= p1) continue;
          int slot = zslot + zr;
          slot = slot >= rd ? slot - rd : slot;
          // a power of two commutes with the products' rounding
          const float wz = SPLIT ? __fmul_rn(w[2][a3], 1048576.f) : w[2][a3];
#pragma unroll
          for (int a2 = 0; a2 < 3; ++a2) {
            const int y = c0[1] + a2;
            if ((unsigned)y >= (unsigned)ey) continue;
            int* const row = ring + (slot * cy + y) * cx + c0[0];
#pragma unroll
            for (int a1 = 0; a1 < 3; ++a1) {
              if ((unsigned)(c0[0] + a1) >= (unsigned)ex) continue;
              const float ww = __fmul_rn(__fmul_rn(w[0][a1], w[1][a2]), wz);
              if (SPLIT) {
                const float h = __fadd_rn(ww, M);
                const float r = __fmaf_rn(__fsub_rn(ww, __fsub_rn(h, M)), 1048576.f, M);
                atomicAdd(row + a1, __float_as_int(r) - __float_as_int(M));
                atomicAdd(row + hi_at + a1, __float_as_int(h) - __float_as_int(M));
              } else {
                const unsigned long long v64 = fixed40(ww);
                unsigned* const word = reinterpret_cast<unsigned*>(row + a1);
                const unsigned old = atomicAdd(word, (unsigned)v64);
                const unsigned up = (unsigned)(v64 >> 32) + (old + (unsigned)v64 < old ? 1u : 0u);
                if (up) atomicAdd(word + hi_at, up);
              }
            }
          }
        }
      }
    };
    if (split) visits(std::true_type{});
    else visits(std::false_type{});
    __syncthreads();
    const int upto = l == l1 ? p1 : min(p1, zb + q);
    for (int t = tid; t < per * ngrp; t += DEPB_T) {
      const int grp = t / per, i = t - grp * per, y = i / cxq, x = 4 * (i - y * cxq);
      if (y >= ey) continue;
      int p = done + grp, slot = p % rd;
      float* out = rho + (j * B.n + p) * pl + (int64_t)(oy + y) * pr + ox + x;
      const bool vec = x + 4 <= ex && (reinterpret_cast<uintptr_t>(out) & 15) == 0 && (pl & 3) == 0;
      for (; p < upto; p += ngrp, out += ngrp * pl) {
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        if (p >= zb && p <= zb + q + 1) {  // else no layer reaches the plane
          int4* a = reinterpret_cast<int4*>(ring + (slot * cy + y) * cx + x);
          int4* b = reinterpret_cast<int4*>(ring + hi_at + (slot * cy + y) * cx + x);
          const int4 l4 = *a, h4 = *b;
          *a = make_int4(0, 0, 0, 0);
          *b = make_int4(0, 0, 0, 0);
          const int lo[4] = {l4.x, l4.y, l4.z, l4.w}, hi[4] = {h4.x, h4.y, h4.z, h4.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const long long sum = split ? (long long)hi[k] * 1048576 + lo[k]
                                        : (long long)(((unsigned long long)(unsigned)hi[k] << 32) | (unsigned)lo[k]);
            f[k] = __fmul_rn(__ll2float_rn(sum), 9.094947017729282e-13f);  // 2^-40
            // the physical cells: pad .. n-pad-1
            if (msum && (unsigned)(ox + x + k - B.pad) < (unsigned)(B.S * q) &&
                (unsigned)(oy + y - B.pad) < (unsigned)(B.S * q) && (unsigned)(p - B.pad) < (unsigned)(B.S * q))
              mloc += (unsigned long long)sum;
          }
        }
        if (vec) {
          __stcs(reinterpret_cast<float4*>(out), make_float4(f[0], f[1], f[2], f[3]));
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (x + k < ex) out[k] = f[k];
        }
        slot += gstep;
        slot = slot >= rd ? slot - rd : slot;
      }
    }
    done = max(done, upto);
    __syncthreads();
  }
  if (msum) {
    if (fixed) warp_sum_to(mloc, static_cast<unsigned long long*>(msum));
    else warp_sum_to((double)(long long)mloc * 9.094947017729282e-13, static_cast<double*>(msum));
  }
}

// The parts of a box: of the splits along x, y and z whose ring fits DEPB_SMEM, the one that
// an estimate of the time (in rounds of the resident blocks) favours: a layer costs its
// barriers and dependent loads (DEPB_C0 clocks), its particles (`per_cell` a coarse cell,
// DEPB_C1 clocks per round of the block's threads) and its write-out (DEPB_C2 per round of 4
// cells a thread); fewer, larger parts look at fewer particles twice, and few boxes want more
// parts than fit the ring.
constexpr double DEPB_C0 = 3000, DEPB_C1 = 4500, DEPB_C2 = 600;
inline DepBox dep_box(int S, int halo, int q, int pad, int iapm, int64_t nbox, double per_cell, int nsm) {
  DepBox B{};
  B.S = S;
  B.halo = halo;
  B.q = q;
  B.pad = pad;
  B.iapm = iapm;
  B.n = S * q + 2 * pad;
  const int nl = S + 2 * halo;
  double best = -1;
  int lastx = 0;
  for (int nx = 1; nx <= 32; ++nx) {
    const int cx = ((B.n + nx - 1) / nx + 3) / 4 * 4, ncx = (B.n + cx - 1) / cx;
    if (cx == lastx || (cx < 8 && nx > 1 && best >= 0)) continue;
    lastx = cx;
    int lasty = 0;
    for (int ny = 1, tried = 0; ny <= B.n && tried < 4; ++ny) {
      const int cy = (B.n + ny - 1) / ny, ncy = (B.n + cy - 1) / cy;
      if (cy == lasty || (int64_t)cx * cy * (q + 2) * 8 > DEPB_SMEM || cy > 28 * q) continue;
      lasty = cy;
      ++tried;
      const double kx = std::min(nl, (cx + 1) / q + 2), ky = std::min(nl, (cy + 1) / q + 2);
      const double layer = DEPB_C0 + DEPB_C1 * std::max(1.0, kx * ky * per_cell / DEPB_T) +
                           DEPB_C2 * std::max(1.0, (double)cx * cy * q / (4 * DEPB_T));
      for (int lz = nl; lz >= 1; lz = lz > 1 ? (lz + 1) / 2 : 0) {  // layers a part
        const int cz = std::min(B.n, lz * q), ncz = (B.n + cz - 1) / cz;
        const double blocks = (double)nbox * ncx * ncy * ncz, slots = 2.0 * nsm;
        const double rounds = blocks <= 8 * slots ? std::ceil(blocks / slots) : blocks / slots;
        const double cost = rounds * std::min(nl, lz + 2) * layer;
        if (best < 0 || cost < best) {
          best = cost;
          B.cx = cx;
          B.cy = cy;
          B.cz = cz;
          B.ncx = ncx;
          B.ncy = ncy;
          B.ncz = ncz;
        }
      }
    }
  }
  return B;
}
inline size_t dep_box_smem(const DepBox& B) { return (size_t)B.cx * B.cy * (B.q + 2) * 8; }

// =================================================================================
// Force from potential (particle_mesh.f90:224-247, kick.f90:839-862) and max |F|^2.
// =================================================================================
__device__ __forceinline__ float grad4(float pm2, float pm1, float pp1, float pp2) {
  const float w0 = (CUBE_W_ALPHA - 1.f) / 4.f, w1 = -CUBE_W_ALPHA / 2.f, w2 = CUBE_W_ALPHA / 2.f,
              w3 = (1.f - CUBE_W_ALPHA) / 4.f;
  float s = __fmul_rn(pm2, w0);
  s = __fadd_rn(s, __fmul_rn(pm1, w1));
  s = __fadd_rn(s, __fmul_rn(pp1, w2));
  s = __fadd_rn(s, __fmul_rn(pp2, w3));
  return s;
}

__device__ __forceinline__ float sumsq3(float a, float b, float c) {
  return __fadd_rn(__fadd_rn(__fmul_rn(a, a), __fmul_rn(b, b)), __fmul_rn(c, c));
}

__device__ __forceinline__ float warp_max(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide max of non-negative values; one atomic per block.  Every thread of the
// block must call it (no early returns before it).
__device__ __forceinline__ void block_max_to(float v, float* out) {
  __shared__ float sm[32];
  v = warp_max(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sm[w] = v;
  __syncthreads();
  if (w == 0) {
    v = (lane < (int)(blockDim.x >> 5)) ? sm[lane] : 0.f;
    v = warp_max(v);
    if (lane == 0 && v > 0.f) atomic_max_pos(out, v);
  }
}

// PM1: periodic nc^3 phi[z][y][x].  One warp per x-row, grid-stride over rows.
__global__ void k_f2max_periodic(const float* __restrict__ phi, int nc, float* __restrict__ f2out, int pf, int64_t pl) {
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  float v = 0.f;
  const int nrows = nc * nc;
  for (int row = blockIdx.x * wpb + (threadIdx.x >> 5); row < nrows; row += gridDim.x * wpb) {
    const int z = row / nc, y = row - z * nc;
    const int zm2 = wrapi(z - 2, nc), zm1 = wrapi(z - 1, nc), zp1 = wrapi(z + 1, nc), zp2 = wrapi(z + 2, nc);
    const int ym2 = wrapi(y - 2, nc), ym1 = wrapi(y - 1, nc), yp1 = wrapi(y + 1, nc), yp2 = wrapi(y + 2, nc);
    auto R = [&](int zz, int yy) { return phi + (size_t)zz * pl + (size_t)yy * pf; };
    const float* r0 = R(z, y);
    for (int x = lane; x < nc; x += 32) {
      const int xm2 = wrapi(x - 2, nc), xm1 = wrapi(x - 1, nc), xp1 = wrapi(x + 1, nc), xp2 = wrapi(x + 2, nc);
      const float fx = grad4(r0[xm2], r0[xm1], r0[xp1], r0[xp2]);
      const float fy = grad4(R(z, ym2)[x], R(z, ym1)[x], R(z, yp1)[x], R(z, yp2)[x]);
      const float fz = grad4(R(zm2, y)[x], R(zm1, y)[x], R(zp1, y)[x], R(zp2, y)[x]);
      v = fmaxf(v, sumsq3(fx, fy, fz));
    }
  }
  block_max_to(v, f2out);
}

// f2max over box meshes phi[b] (row pitch pf, plane pitch pl floats; coordinate i is
// array index i - m1phi; physical cells 1..nforce), z stencil in registers.  Block: a 32x32 (x,y) tile of one
// box, 256 threads; thread (lx, ly) owns cells y = 4*ly .. 4*ly+3 at x = lx.  Halo
// planes (36x36) of phi stream through a 4-stage shared-memory ring filled with cp.async,
// three planes ahead of the one being reduced.  From a plane a thread takes one column
// of 8 values (own phi and the y stencils of its 4 cells) and 4 x stencils, 6 loads per
// cell.  Own phi values of the last 5 planes and fx, fy of the last 3 stay in registers,
// so the force at plane zc-2 completes when plane zc arrives.
constexpr int F3_T = 32, F3_P = F3_T + 4, F3_HALO = F3_P * F3_P, F3_LOADS = (F3_HALO + 255) / 256, F3_STAGES = 4;
__device__ __forceinline__ void f3_cp_async4(float* smem, const float* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__global__ void __launch_bounds__(256, 3) k_f2max_box2(const float* __restrict__ phi, int n, int nforce, int m1phi,
                                                       int nbox, float* __restrict__ f2out, int pf, int64_t pl,
                                                       const int32_t* __restrict__ box_sub) {
  __shared__ float pln[F3_STAGES][F3_HALO];
  const int nt = (nforce + F3_T - 1) / F3_T;
  const int tile = blockIdx.x % (nt * nt);
  const int b = blockIdx.x / (nt * nt);
  if (box_sub && box_sub[b] < 0) return;  // padding slot of a class list: block-uniform, nothing to reduce
  const int tx0 = (tile % nt) * F3_T + 1, ty0 = (tile / nt) * F3_T + 1;  // first physical x, y
  const float* pb = phi + (size_t)b * n * pl;
  const int lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
  int off[F3_LOADS];
#pragma unroll
  for (int k = 0; k < F3_LOADS; ++k) {
    const int i = threadIdx.x + k * 256;
    off[k] = -2;  // not a halo element of this thread
    if (i < F3_HALO) {
      const int py = i / F3_P, px = i - py * F3_P;
      const int x = tx0 - 2 + px - m1phi, y = ty0 - 2 + py - m1phi;  // array coordinates, >= 0
      off[k] = (x < n && y < n) ? y * pf + x : -1;
      if (off[k] < 0)
#pragma unroll
        for (int st = 0; st < F3_STAGES; ++st) pln[st][i] = 0.f;  // outside the box: zero, never copied
    }
  }
  const int zlast = nforce + 2;
  auto issue = [&](int zc) {  // copy plane zc into its stage; always commits a group
    if (zc <= zlast) {
      const float* pz = pb + (size_t)(zc - m1phi) * pl;
      float* dst = pln[(zc + 1) & (F3_STAGES - 1)];
#pragma unroll
      for (int k = 0; k < F3_LOADS; ++k)
        if (off[k] >= 0) f3_cp_async4(dst + threadIdx.x + k * 256, pz + off[k]);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  const bool xin = tx0 + lx <= nforce;
  bool own[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) own[j] = xin && (ty0 + 4 * ly + j <= nforce);
  float P[4][5], FX[4][3], FY[4][3];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
#pragma unroll
    for (int q = 0; q < 5; ++q) P[j][q] = 0.f;
#pragma unroll
    for (int q = 0; q < 3; ++q) FX[j][q] = FY[j][q] = 0.f;
  }
  float v = 0.f;
  issue(-1);
  issue(0);
  issue(1);
  for (int zc = -1; zc <= zlast; ++zc) {
    asm volatile("cp.async.wait_group 2;\n" ::: "memory");  // this thread's copies of plane zc landed
    __syncthreads();  // everyone's copies landed; the stage of plane zc-1 is free again
    issue(zc + 3);
    const float* c = pln[(zc + 1) & (F3_STAGES - 1)];
    // own column: rows 4*ly .. 4*ly+7 of the halo plane at x = lx + 2
    float col[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) col[r] = c[(4 * ly + r) * F3_P + lx + 2];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int q = 0; q < 4; ++q) P[j][q] = P[j][q + 1];
      P[j][4] = col[j + 2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        FX[j][q] = FX[j][q + 1];
        FY[j][q] = FY[j][q + 1];
      }
      const float* row = c + (4 * ly + j + 2) * F3_P + lx + 2;
      FX[j][2] = grad4(row[-2], row[-1], row[1], row[2]);
      FY[j][2] = grad4(col[j], col[j + 1], col[j + 3], col[j + 4]);
      if (zc >= 3 && own[j]) {  // plane zc-2 is complete: phi(zc-4..zc) in P, fx, fy in slot 0
        const float fz = grad4(P[j][0], P[j][1], P[j][3], P[j][4]);
        v = fmaxf(v, sumsq3(FX[j][0], FY[j][0], fz));
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  block_max_to(v, f2out);
}

// The same over rows read in whole vectors, for layouts that k_f2max_box3_fits accepts: a
// thread owns 4 cells along x of one row, so a plane costs it 7 vector loads from shared memory
// (own cells, the 2 on either side, the rows at +-1 and +-2) and the planes arrive by 16-byte
// copies.  The differences go first, phi(+1) - phi(-1) and phi(+2) - phi(-2), then their
// weights, two cells to an instruction: 9 floating-point instructions per cell instead of 27.
// phi of the last five planes stays in registers for the z stencil, and of the x and y
// components only the sum of squares.  Halo planes are 36 rows of 40 values, the own cells
// from column 4.  2.12 ms for 512 boxes of 144^3 in the form above, bound by instruction issue;
// 1.39 ms now (reading phi once: 0.92).
constexpr int F3_Q = 40;
__device__ __forceinline__ void f3_cp_async16(float* smem, const float* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
inline bool f2max_box3_fits(int n, int nforce, int m1phi, int pf, int64_t pl, const float* phi) {
  return n % 4 == 0 && nforce % 4 == 0 && (1 - m1phi) % 4 == 0 && 1 - m1phi >= 4 && pf % 4 == 0 && pl % 4 == 0 &&
         (reinterpret_cast<uintptr_t>(phi) & 15) == 0;
}
__global__ void __launch_bounds__(256, 3) k_f2max_box3(const float* __restrict__ phi, int n, int nforce, int m1phi,
                                                       int nbox, float* __restrict__ f2out, int pf, int64_t pl,
                                                       const int32_t* __restrict__ box_sub) {
  __shared__ __align__(16) float pln[F3_STAGES][F3_P * F3_Q];
  const int nt = (nforce + F3_T - 1) / F3_T;
  const int tile = blockIdx.x % (nt * nt);
  const int b = blockIdx.x / (nt * nt);
  if (box_sub && box_sub[b] < 0) return;  // padding slot of a class list: block-uniform, nothing to reduce
  const int tx0 = (tile % nt) * F3_T + 1, ty0 = (tile / nt) * F3_T + 1;  // first physical x, y
  const float* pb = phi + (size_t)b * n * pl;
  const int xq = threadIdx.x & 7, ly = threadIdx.x >> 3;
  // this thread's 16-byte copies of a halo plane (36 rows of 10)
  constexpr int NC = F3_P * F3_Q / 4, LOADS = (NC + 255) / 256;
  int off[LOADS];
#pragma unroll
  for (int k = 0; k < LOADS; ++k) {
    const int i = threadIdx.x + k * 256;
    off[k] = -2;  // not a piece of this thread
    if (i < NC) {
      const int py = i / (F3_Q / 4), px = 4 * (i - py * (F3_Q / 4));
      const int x = tx0 - 4 + px - m1phi, y = ty0 - 2 + py - m1phi;  // array coordinates, x a multiple of 4
      off[k] = (x + 4 <= n && y < n) ? y * pf + x : -1;
      if (off[k] < 0)
#pragma unroll
        for (int st = 0; st < F3_STAGES; ++st)
          *reinterpret_cast<float4*>(&pln[st][4 * i]) = make_float4(0.f, 0.f, 0.f, 0.f);  // outside the box: never copied
    }
  }
  const int zlast = nforce + 2;
  auto issue = [&](int zc) {  // copy plane zc into its stage; always commits a group
    if (zc <= zlast) {
      const float* pz = pb + (size_t)(zc - m1phi) * pl;
      float* dst = pln[(zc + 1) & (F3_STAGES - 1)];
#pragma unroll
      for (int k = 0; k < LOADS; ++k)
        if (off[k] >= 0) f3_cp_async16(dst + 4 * (threadIdx.x + k * 256), pz + off[k]);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  const bool own = tx0 + 4 * xq <= nforce && ty0 + ly <= nforce;
  const float2 g1 = make_float2(CUBE_W_ALPHA / 2.f, CUBE_W_ALPHA / 2.f);
  const float2 g2 = make_float2((1.f - CUBE_W_ALPHA) / 4.f, (1.f - CUBE_W_ALPHA) / 4.f);
  const float2 neg = make_float2(-1.f, -1.f);
  auto diff = [&](float2 a, float2 b2) { return fma2(b2, neg, a); };                       // a - b
  auto grad = [&](float2 d1, float2 d2) { return fma2(g2, d2, mul2(g1, d1)); };
  float2 P[5][2], S[3][2];
#pragma unroll
  for (int k = 0; k < 5; ++k) P[k][0] = P[k][1] = make_float2(0.f, 0.f);
#pragma unroll
  for (int k = 0; k < 3; ++k) S[k][0] = S[k][1] = make_float2(0.f, 0.f);
  float v = 0.f;
  issue(-1);
  issue(0);
  issue(1);
  for (int zc = -1; zc <= zlast; ++zc) {
    asm volatile("cp.async.wait_group 2;\n" ::: "memory");  // this thread's copies of plane zc landed
    __syncthreads();  // everyone's copies landed; the stage of plane zc-1 is free again
    issue(zc + 3);
    const float* c = pln[(zc + 1) & (F3_STAGES - 1)] + (ly + 2) * F3_Q + 4 + 4 * xq;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      P[k][0] = P[k + 1][0];
      P[k][1] = P[k + 1][1];
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      S[k][0] = S[k + 1][0];
      S[k][1] = S[k + 1][1];
    }
    const float4 r = *reinterpret_cast<const float4*>(c);
    const float2 rl = *reinterpret_cast<const float2*>(c - 2), rr = *reinterpret_cast<const float2*>(c + 4);
    const float4 um2 = *reinterpret_cast<const float4*>(c - 2 * F3_Q), um1 = *reinterpret_cast<const float4*>(c - F3_Q);
    const float4 up1 = *reinterpret_cast<const float4*>(c + F3_Q), up2 = *reinterpret_cast<const float4*>(c + 2 * F3_Q);
    const float2 r01 = make_float2(r.x, r.y), r23 = make_float2(r.z, r.w);
    P[4][0] = r01;
    P[4][1] = r23;
    const float2 fx0 = grad(make_float2(r.y - rl.y, r.z - r.x), diff(r23, rl));
    const float2 fx1 = grad(make_float2(r.w - r.y, rr.x - r.z), diff(rr, r01));
    const float2 fy0 = grad(diff(make_float2(up1.x, up1.y), make_float2(um1.x, um1.y)),
                            diff(make_float2(up2.x, up2.y), make_float2(um2.x, um2.y)));
    const float2 fy1 = grad(diff(make_float2(up1.z, up1.w), make_float2(um1.z, um1.w)),
                            diff(make_float2(up2.z, up2.w), make_float2(um2.z, um2.w)));
    S[2][0] = fma2(fy0, fy0, mul2(fx0, fx0));
    S[2][1] = fma2(fy1, fy1, mul2(fx1, fx1));
    if (zc >= 3 && own) {  // plane zc-2 is complete: phi(zc-4..zc) in P, fx^2 + fy^2 in slot 0
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float2 fz = grad(diff(P[3][k], P[1][k]), diff(P[4][k], P[0][k]));
        const float2 f2 = fma2(fz, fz, S[0][k]);
        v = fmaxf(v, fmaxf(f2.x, f2.y));
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  block_max_to(v, f2out);
}

__host__ inline unsigned f2max_box2_grid(int nforce, int nbox) {
  const int nt = (nforce + F3_T - 1) / F3_T;
  return (unsigned)(nt * nt * nbox);
}

// =================================================================================
// Interpolation and kick (particle_mesh.f90:148-217, kick.f90:745-834).  The force
// at each of the 27 TSC cells is differenced from phi on the fly; the values equal
// those of a stored force grid because each uses the same four phi values.
// =================================================================================
// For each component the 27 TSC terms are summed in the reference order
// (i3 outer, i2, i1 inner; kick.f90:789-795); components are independent sums, so
// they are accumulated one after another to keep the loads to 3 x 63.
template <class PhiFn>
__device__ __forceinline__ void tsc_gather_force(const int i2[3], const float w[3][3], PhiFn P, float dv[3]) {
  const int x0 = i2[0] - 1, y0 = i2[1] - 1, z0 = i2[2] - 1;
  // x component: rows of 7 values along x
  float s = 0.f;
#pragma unroll
  for (int a3 = 0; a3 < 3; ++a3)
#pragma unroll
    for (int a2 = 0; a2 < 3; ++a2) {
      float r[7];
#pragma unroll
      for (int k = 0; k < 7; ++k) r[k] = P(x0 - 2 + k, y0 + a2, z0 + a3);
#pragma unroll
      for (int a1 = 0; a1 < 3; ++a1) {
        const float F = grad4(r[a1], r[a1 + 1], r[a1 + 3], r[a1 + 4]);
        s = __fadd_rn(s, __fmul_rn(__fmul_rn(__fmul_rn(F, w[0][a1]), w[1][a2]), w[2][a3]));
      }
    }
  dv[0] = s;
  // y component: per a3, a 7 (y) x 3 (x) block
  s = 0.f;
#pragma unroll
  for (int a3 = 0; a3 < 3; ++a3) {
    float r[7][3];
#pragma unroll
    for (int k = 0; k < 7; ++k)
#pragma unroll
      for (int a1 = 0; a1 < 3; ++a1) r[k][a1] = P(x0 + a1, y0 - 2 + k, z0 + a3);
#pragma unroll
    for (int a2 = 0; a2 < 3; ++a2)
#pragma unroll
      for (int a1 = 0; a1 < 3; ++a1) {
        const float F = grad4(r[a2][a1], r[a2 + 1][a1], r[a2 + 3][a1], r[a2 + 4][a1]);
        s = __fadd_rn(s, __fmul_rn(__fmul_rn(__fmul_rn(F, w[0][a1]), w[1][a2]), w[2][a3]));
      }
  }
  dv[1] = s;
  // z component: the 27 values first (columns of 7 along z), then the ordered sum
  float F2[3][3][3];
#pragma unroll
  for (int a2 = 0; a2 < 3; ++a2)
#pragma unroll
    for (int a1 = 0; a1 < 3; ++a1) {
      float r[7];
#pragma unroll
      for (int k = 0; k < 7; ++k) r[k] = P(x0 + a1, y0 + a2, z0 - 2 + k);
#pragma unroll
      for (int a3 = 0; a3 < 3; ++a3) F2[a3][a2][a1] = grad4(r[a3], r[a3 + 1], r[a3 + 3], r[a3 + 4]);
    }
  s = 0.f;
#pragma unroll
  for (int a3 = 0; a3 < 3; ++a3)
#pragma unroll
    for (int a2 = 0; a2 < 3; ++a2)
#pragma unroll
      for (int a1 = 0; a1 < 3; ++a1)
        s = __fadd_rn(s, __fmul_rn(__fmul_rn(__fmul_rn(F2[a3][a2][a1], w[0][a1]), w[1][a2]), w[2][a3]));
  dv[2] = s;
}

__device__ __forceinline__ void apply_kick(float* vp, int64_t ip, const float dv[3], float a_mid, float dt,
                                           float av[3]) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float v = kick_add(vp[3 * ip + d], dv[d], a_mid, dt);
    vp[3 * ip + d] = v;
    av[d] = fabsf(v);
  }
}

__device__ __forceinline__ void block_vmax(const float av[3], float* vmax) {
  block_max_to(av[0], vmax + 0);
  block_max_to(av[1], vmax + 1);
  block_max_to(av[2], vmax + 2);
}

__global__ void k_interp_pm1(Geo G, int64_t np, const void* __restrict__ xp, const int32_t* __restrict__ pcell,
                             const float* __restrict__ phi, float* __restrict__ vp, const StepDev* __restrict__ sd,
                             int pf, int64_t pl) {
  const int64_t ip = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= np) return;
  const float a_mid = sd->a_mid, dt = sd->dt;
  int g[3];
  cell_coords(G, pcell[ip], g[0], g[1], g[2]);
  int i2[3];
  float w[3][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double xpos = (double)g[d] + zfrac(load_code(xp, G.izipx, 3 * ip + d), G);
    i2[d] = tsc_weights(xpos, w[d]);
  }
  const int nc = G.nc;
  // force index i (1-based, periodic) reads phi(i-2..i+2); array index (i-1) mod nc.
  // Wrapped indices of the 7 positions i2-3..i2+3 per dimension, computed once.
  int wx[7], wy[7], wz[7];
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    wx[k] = wrapi(i2[0] - 4 + k, nc);
    wy[k] = wrapi(i2[1] - 4 + k, nc) * pf;
    wz[k] = wrapi(i2[2] - 4 + k, nc) * (int)pl;
  }
  const int x0 = i2[0] - 1, y0 = i2[1] - 1, z0 = i2[2] - 1;
  auto P = [&](int a, int b, int c) { return __ldg(&phi[wz[c - z0 + 2] + wy[b - y0 + 2] + wx[a - x0 + 2]]); };
  float dv[3], av[3];
  tsc_gather_force(i2, w, P, dv);
  apply_kick(vp, ip, dv, a_mid, dt, av);
}

// PM1 force mesh, as potential_to_force builds it before the interpolation
// (particle_mesh.f90:224-247): at every coarse cell j (0-based, periodic) the three
// components grad4(phi(j-2), phi(j-1), phi(j+1), phi(j+2)), with the same FP32
// operations as tsc_gather_force, stored as float4 (fx, fy, fz, 0), x fastest.
// Grid (blocks along x, y, z): FORCE_T cells along x and, per thread, ZS along z.  Bound by the
// write of 16 bytes a cell; with one cell a thread the blocks of a large mesh come and go too
// fast to keep enough loads in flight: 0.119 ms at 256^3 cells, 0.090 with four (the write and
// the read of phi alone: 0.050).  A mesh whose blocks of four cells are fewer than two rounds
// of the chip's (2 x 16 x 148) keeps one (64^3: 4.0 us against 4.5).
constexpr int FORCE_T = 128, FORCE_Z = 4;
inline dim3 force_grid(int nc, int zs = 1) {
  return dim3((unsigned)((nc + FORCE_T - 1) / FORCE_T), (unsigned)nc, (unsigned)((nc + zs - 1) / zs));
}
inline bool force_deep(int nc) {
  const dim3 g = force_grid(nc, FORCE_Z);
  return (int64_t)g.x * g.y * g.z >= 2 * 16 * 148;
}
template <int ZS>
__global__ void __launch_bounds__(FORCE_T) k_force_pm1(int nc, const float* __restrict__ phi, int pf, int64_t pl,
                                                       float4* __restrict__ force) {
  const int x = blockIdx.x * FORCE_T + threadIdx.x, y = blockIdx.y, z0 = blockIdx.z * ZS;
  if (x >= nc) return;
  const int xm2 = wrap1(x - 2, nc), xm1 = wrap1(x - 1, nc), xp1 = wrap1(x + 1, nc), xp2 = wrap1(x + 2, nc);
  const float* const row = phi + (int64_t)y * pf;
  const float* const ym2 = phi + (int64_t)wrap1(y - 2, nc) * pf + x;
  const float* const ym1 = phi + (int64_t)wrap1(y - 1, nc) * pf + x;
  const float* const yp1 = phi + (int64_t)wrap1(y + 1, nc) * pf + x;
  const float* const yp2 = phi + (int64_t)wrap1(y + 2, nc) * pf + x;
  float line[ZS + 4];  // phi(x, y, z0 - 2 ..)
#pragma unroll
  for (int k = 0; k < ZS + 4; ++k) line[k] = __ldg(row + x + (int64_t)wrapi(z0 - 2 + k, nc) * pl);
#pragma unroll
  for (int k = 0; k < ZS; ++k) {
    const int z = z0 + k;
    if (z >= nc) break;
    const int64_t o = (int64_t)z * pl;
    force[((int64_t)z * nc + y) * nc + x] =
        make_float4(grad4(__ldg(row + o + xm2), __ldg(row + o + xm1), __ldg(row + o + xp1), __ldg(row + o + xp2)),
                    grad4(__ldg(ym2 + o), __ldg(ym1 + o), __ldg(yp1 + o), __ldg(yp2 + o)),
                    grad4(line[k], line[k + 1], line[k + 3], line[k + 4]), 0.f);
  }
}

// PM1 interpolation + kick from the force mesh: the 27 TSC points of a particle are the
// cells fl-1..fl+1 around its coarse cell; each component is summed in the order of
// tsc_gather_force (a3 outer, a2, a1 inner) with the same products, so the result is
// bit-identical to differencing phi on the fly.
__global__ void k_interp_pm1_force(Geo G, int64_t np, const void* __restrict__ xp, const int32_t* __restrict__ pcell,
                                   const float4* __restrict__ force, float* __restrict__ vp,
                                   const StepDev* __restrict__ sd) {
  const int64_t ip = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= np) return;
  const float a_mid = sd->a_mid, dt = sd->dt;
  int g[3];
  cell_coords(G, pcell[ip], g[0], g[1], g[2]);
  int i2[3];
  float w[3][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double xpos = (double)g[d] + zfrac(load_code(xp, G.izipx, 3 * ip + d), G);
    i2[d] = tsc_weights(xpos, w[d]);
  }
  const int nc = G.nc;
  int64_t jx[3], jy[3], jz[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    jx[a] = wrap1(i2[0] - 2 + a, nc);
    jy[a] = (int64_t)wrap1(i2[1] - 2 + a, nc) * nc;
    jz[a] = (int64_t)wrap1(i2[2] - 2 + a, nc) * nc * nc;
  }
  float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
  for (int a3 = 0; a3 < 3; ++a3)
#pragma unroll
    for (int a2 = 0; a2 < 3; ++a2)
#pragma unroll
      for (int a1 = 0; a1 < 3; ++a1) {
        const float4 F = __ldg(&force[jz[a3] + jy[a2] + jx[a1]]);
        sx = __fadd_rn(sx, __fmul_rn(__fmul_rn(__fmul_rn(F.x, w[0][a1]), w[1][a2]), w[2][a3]));
        sy = __fadd_rn(sy, __fmul_rn(__fmul_rn(__fmul_rn(F.y, w[0][a1]), w[1][a2]), w[2][a3]));
        sz = __fadd_rn(sz, __fmul_rn(__fmul_rn(__fmul_rn(F.z, w[0][a1]), w[1][a2]), w[2][a3]));
      }
  const float dv[3] = {sx, sy, sz};
  float av[3];
  apply_kick(vp, ip, dv, a_mid, dt, av);
}

__global__ void __launch_bounds__(256, 3) k_interp_pm2(Geo G, int64_t np, const void* __restrict__ xp, const int32_t* __restrict__ pcell,
                             const float* __restrict__ phi, int tile0, int ntile, float* __restrict__ vp,
                             const StepDev* __restrict__ sd, float* vmax, unsigned* err, int pf, int64_t pl) {
  const int64_t ip = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const float a_mid = sd->a_mid, dt = sd->dt;
  float av[3] = {0.f, 0.f, 0.f};
  if (ip < np) {
    int g[3];
    cell_coords(G, pcell[ip], g[0], g[1], g[2]);
    const int T = ((g[2] / G.nt) * G.nnt + g[1] / G.nt) * G.nnt + g[0] / G.nt;
    if (T >= tile0 && T < tile0 + ntile) {
      int i2[3];
      float w[3][3];
      bool oob = false;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double xpos = ((double)(g[d] % G.nt) + zfrac(load_code(xp, G.izipx, 3 * ip + d), G)) * (double)G.rcs;
        i2[d] = tsc_weights(xpos, w[d]);
        if (i2[d] - 1 < 0 || i2[d] + 1 > G.ngp + 1) oob = true;
      }
      if (oob) {
        set_err(err, CUBE_DEVERR_INTERP_RANGE);
      } else {
        const int n = G.ngt, m1 = 1 - G.ngb;
        const float* pb = phi + (size_t)(T - tile0) * n * pl;
        const int ipl = (int)pl;
        auto P = [&](int a, int b, int c) { return __ldg(&pb[(c - m1) * ipl + (b - m1) * pf + (a - m1)]); };
        float dv[3];
        tsc_gather_force(i2, w, P, dv);
        apply_kick(vp, ip, dv, a_mid, dt, av);
      }
    }
  }
  block_vmax(av, vmax);
}

// msum: PM3 mass slots; each particle adds its own box's 27 contributions (the mass sums
// described at k_mass_pm3), in the arithmetic of the deposit form.
template <bool FIXED>
__global__ void __launch_bounds__(256, 3) k_interp_pm3(Geo G, int64_t np, const void* __restrict__ xp, const int32_t* __restrict__ pcell,
                             const float* __restrict__ phi, const int32_t* __restrict__ box_slot, int iapm,
                             float* __restrict__ vp, const StepDev* __restrict__ sd, float* vmax, unsigned* err,
                             int pf, int64_t pl, void* msum) {
  const int64_t ip = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const float a_mid = sd->a_mid, dt = sd->dt;
  float av[3] = {0.f, 0.f, 0.f};
  MassAcc<FIXED> mass;
  if (ip < np) {
    int g[3];
    cell_coords(G, pcell[ip], g[0], g[1], g[2]);
    int t[3], u[3], l[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      t[d] = g[d] / G.nt;
      l[d] = g[d] - t[d] * G.nt;
      u[d] = l[d] / G.ntt;
    }
    const int slot = box_slot[subtile_id(G, t, u)];
    if (slot >= 0) {
      const int nft = G.nft[iapm], nfp = G.nfp[iapm], nfb = G.nfb[iapm];
      const double gs = (double)(1.f / (float)rsf_of(iapm));
      int i2[3];
      float w[3][3];
      bool oob = false;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double xpos = pm3_xpos((double)l[d] + zfrac(load_code(xp, G.izipx, 3 * ip + d), G), G, gs, rsf_of(iapm), u[d] * nfp);
        i2[d] = tsc_weights(xpos, w[d]);
        if (i2[d] - 1 < 0 || i2[d] + 1 > nfp + 1) oob = true;
      }
      if (oob) {
        set_err(err, CUBE_DEVERR_INTERP_RANGE);
      } else {
        const int m1 = 1 - nfb;
        const float* pb = phi + (size_t)slot * nft * pl;
        const int ipl = (int)pl;
        auto P = [&](int a, int b, int c) { return __ldg(&pb[(c - m1) * ipl + (b - m1) * pf + (a - m1)]); };
        float dv[3];
        tsc_gather_force(i2, w, P, dv);
        apply_kick(vp, ip, dv, a_mid, dt, av);
#pragma unroll
        for (int a3 = 0; a3 < 3; ++a3)
#pragma unroll
          for (int a2 = 0; a2 < 3; ++a2)
#pragma unroll
            for (int a1 = 0; a1 < 3; ++a1) mass.add(__fmul_rn(__fmul_rn(w[0][a1], w[1][a2]), w[2][a3]));
      }
    }
  }
  block_vmax(av, vmax);
  mass.flush(msum);
}

// =================================================================================
// Subtile classes (kick.f90:108-133) and the box slot map of one class.
// =================================================================================
// One block per subtile: its threads read the subtile's rows of cells side by side.  (One
// thread per subtile read ntt^3 counts one after the other: 0.74 ms at ntt = 16, whatever
// the number of subtiles, against 0.01 ms for 512 of them now.)
constexpr int CLASSIFY_T = 128;
__global__ void __launch_bounds__(CLASSIFY_T) k_classify(Geo G, const int32_t* __restrict__ rhoc,
                                                         int32_t* __restrict__ ires, int32_t* __restrict__ napm) {
  __shared__ int part[CLASSIFY_T / 32];
  const int s = blockIdx.x;
  if (s < G.s0 || s >= G.s1) {  // another rank's subtile: its class arrives by a max-reduction
    if (threadIdx.x == 0) ires[s] = 0;
    return;
  }
  const int nns3 = G.nns * G.nns * G.nns, ntt = G.ntt, nt = G.nt;
  const int T = s / nns3, f = s - T * nns3;
  const int ux = f % G.nns, uy = (f / G.nns) % G.nns, uz = f / (G.nns * G.nns);
  // first cell of the subtile; a tile's cells are stored together, x fastest
  const int32_t* base = rhoc + (int64_t)T * nt * nt * nt + ((int64_t)uz * ntt * nt + (int64_t)uy * ntt) * nt + ux * ntt;
  int mx = 0;
  for (int c = threadIdx.x; c < ntt * ntt * ntt; c += CLASSIFY_T) {
    const int row = c / ntt, i = c - row * ntt, k = row / ntt, j = row - k * ntt;
    mx = max(mx, base[((int64_t)k * nt + j) * nt + i]);
  }
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < CLASSIFY_T / 32; ++w) mx = max(mx, part[w]);
  const float npc = (float)mx / 64.f;
  const int r = (npc < 24.f) ? 2 : (npc < 114.f) ? 3 : (npc < 320.f) ? 4 : 5;
  ires[s] = r;
  atomicAdd(&napm[r], 1);
}

// Chunk plan of the PM3 boxes: of the subtiles of class c (2..5) in ascending order, the
// first skip[c] are left out and the next cap[c] at most are listed, in chunks of per[c]
// boxes; chunk j of class c is list kbase[c] + j.  The host sizes it (exactly, or with
// headroom for a captured step; skip > 0 lists what a captured step could not hold) and
// the device fills it from ires.
struct PM3Plan {
  int cap[8], per[8], kbase[8], skip[8];
  int nk, per_max;
};

// Class lists on the device (kick.f90:108-138 classes, kick.f90:141-201 order by class):
// the subtiles of class c in ascending order take slots 0, 1, ... of the chunks of c.
// box_sub[k][slot] = subtile (-1 pads unused slots), box_slot[k][s] = slot (-1: not in
// list k); both arrays arrive filled with -1.  *overflow is set when a class has more
// subtiles than skip + capacity (the ones beyond are not listed).  One block of 1024
// threads; thread t owns a contiguous run of subtiles, so ranks follow subtile order.
__global__ void __launch_bounds__(1024) k_build_lists(const int32_t* __restrict__ ires, int ns3, int s_lo, int s_hi,
                                                      PM3Plan pl, int32_t* __restrict__ box_slot,
                                                      int32_t* __restrict__ box_sub, unsigned* __restrict__ overflow) {
  __shared__ int sc[4][1024];
  const int T = blockDim.x, tid = threadIdx.x;
  const int nown = s_hi - s_lo;  // this rank's subtiles [s_lo, s_hi)
  const int per_t = (nown + T - 1) / T;
  const int s0 = s_lo + min(nown, tid * per_t), s1 = s_lo + min(nown, tid * per_t + per_t);
  int cnt[4] = {0, 0, 0, 0};
  for (int s = s0; s < s1; ++s) cnt[(ires[s] - 2) & 3] += 1;
#pragma unroll
  for (int k = 0; k < 4; ++k) sc[k][tid] = cnt[k];
  __syncthreads();
  for (int off = 1; off < T; off <<= 1) {
    int v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = tid >= off ? sc[k][tid - off] : 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) sc[k][tid] += v[k];
    __syncthreads();
  }
  int r[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) r[k] = sc[k][tid] - cnt[k];
  for (int s = s0; s < s1; ++s) {
    const int c = ires[s], k = (c - 2) & 3;
    const int rank = r[k]++ - pl.skip[c];
    if (rank >= 0 && rank < pl.cap[c]) {
      const int chunk = rank / pl.per[c], slot = rank - chunk * pl.per[c];
      const int64_t kk = pl.kbase[c] + chunk;
      box_slot[kk * ns3 + s] = slot;
      box_sub[kk * pl.per_max + slot] = s;
    }
  }
  if (tid == 0)
    for (int k = 0; k < 4; ++k)
      if (sc[k][T - 1] > pl.skip[k + 2] + pl.cap[k + 2]) *overflow = 1u;
}

// =================================================================================
// PP (kick.f90:376-588).  Each physical particle sums 0<r^2<range^2 pairs over the
// coarse cells its range can reach; equivalent to the reference's PP-cell lists
// (the PP cell 4/rsf fine cells is wider than the range 3.5/rsf).
// =================================================================================
// F_ra of kick.f90 at r = e * apm / 2 <= apm, over apm's coefficient c = (1/35)/apm^2 (the S2
// cloud's force; 1/r^2 beyond).  The outer branch is the polynomial of kick.f90 written in
// t = 2 - e, whose terms are of the sum's size: in e they are a hundred times it and their
// rounding made the force's largest error.
// Rounded step by step (no contraction), so that every kernel gives the same bits.
__device__ __forceinline__ float F_s2_near(float e) {  // e <= 1
  return __fmul_rn(
      e, __fmaf_rn(__fmul_rn(e, e), __fmaf_rn(e, __fmaf_rn(e, __fmaf_rn(e, -21.f, 48.f), 70.f), -224.f), 224.f));
}
__device__ __forceinline__ float F_s2(float e, float twelve_over_e2) {
  const float t = __fsub_rn(2.f, e);
  const float far = __fmaf_rn(
      t, __fmaf_rn(t, __fmaf_rn(t, __fmaf_rn(t, __fmaf_rn(t, __fmaf_rn(t, 7.f, -36.f), 10.f), 16.f), 24.f), 32.f), 32.f);
  // the terms in e up to t^6; 12/e^2 is apart
  return e > 1.f ? __fadd_rn(far, twelve_over_e2) : F_s2_near(e);
}
// 1/r^2 less F_s2, over c, for 1 < e: 140/e^2 less the two terms above.  Its terms cancel up to
// t^4 (140/e^2 - 12/e^2 = 128/e^2 is a power series in t with the same ones), and what is left
// is a product, with no cancellation.
__device__ __forceinline__ float F_s2_rest(float e, float one_over_e2) {
  const float t = __fsub_rn(2.f, e), t2 = __fmul_rn(t, t);
  return __fmul_rn(__fmul_rn(__fmul_rn(t2, t2), t),
                   __fmaf_rn(__fmaf_rn(t, -10.f, 24.f), one_over_e2, __fmaf_rn(t, -7.f, 36.f)));
}

// Candidate coordinate (xq in kick.f90:424): ((lq + (u+0.5)*x_res) * ratio_cs) rounded to
// float.  FAST: lq + (u+0.5)*x_res has at most 8*izipx+1+log2|lq| significant bits; when
// that is <= 24 (int8 codes, or int16 codes with |lq| < 128) every coordinate is an exact
// FP32 number on one grid, and so are the differences of coordinates of neighbouring cells,
// in any order of the sums.
template <bool FAST>
__device__ __forceinline__ float pp_xq(const Geo& G, int lq, int code) {
  static_assert(!FAST, "the FAST form folds the decode into the difference");
  return __fmul_rn((float)((double)lq + zfrac(code, G)), (float)G.rcs);
}

// One particle's PP state: its tile-local position xf (fine cells), the candidate cell
// range per dimension, its range and the accumulated force.
struct PPi {
  float xf[3];
  int l[3], lo[3], hi[3];
  float range, range2;
  float k_range, c_range, p_range;  // 2/range, (1/35)/range^2, range^2/4: F_s2 of the range
  float k_app, c_app, p_app;        // 2/app, (1/35)/app^2, 3 app^2: of the softening (k_app infinite: none)
  float acc[3];
  unsigned pairs, cand;  // of this particle (item): well below 2^32

  __device__ __forceinline__ void init(const Geo& G, const int g[3], const float4 fin, int iapm) {
    const float fi[3] = {fin.x, fin.y, fin.z};
    range = __fdiv_rn(3.5f, (float)rsf_of(iapm));  // apm3(iapm)
    range2 = __fmul_rn(range, range);
    k_range = __fdiv_rn(2.f, range);
    c_range = __fdiv_rn(__fdiv_rn(1.f, 35.f), range2);
    p_range = 0.25f * range2;
    k_app = G.app > 0.f ? __fdiv_rn(2.f, G.app) : __int_as_float(0x7f800000);
    c_app = G.app > 0.f ? __fdiv_rn(__fdiv_rn(1.f, 35.f), __fmul_rn(G.app, G.app)) : 0.f;
    p_app = 3.f * G.app * G.app;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      l[d] = g[d] % G.nt;
      xf[d] = __fadd_rn((float)(l[d] * G.rcs), fi[d]);
      lo[d] = (fi[d] < range) ? -1 : 0;
      hi[d] = ((float)G.rcs - fi[d] < range) ? 1 : 0;
      acc[d] = 0.f;
    }
    pairs = cand = 0;
  }

  __device__ __forceinline__ bool needs(int dx, int dy, int dz) const {
    return dx >= lo[0] && dx <= hi[0] && dy >= lo[1] && dy <= hi[1] && dz >= lo[2] && dz <= hi[2];
  }

  // The force of one pair in range (separation rv, r2 = |rv|^2) added to acc, in the order
  // the callers call it (candidate order).  1/r is the hardware's approximate reciprocal
  // square root and one Newton step (y + y (1/2 - r2 y^2 / 2)), good to about one unit in the
  // last place; the force law and the projection multiply by it.  With IEEE square root and
  // divisions (up to eight a pair) the law took three times the instructions (with the packed
  // separations, the heavy-cell PP of 128^3 clustered particles: 24.8 -> 13.6 ms).  The force
  // of the outer pairs as a product without cancellation (F_s2_rest) costs 0.5 ms of that again
  // and takes the velocities' error against 64 bits below the IEEE form's (a kick of three
  // tiles a side: 3.8e-7, 4.1e-7 before F_s2_rest, 3.1e-7 now).
  __device__ __forceinline__ void accum(float rv0, float rv1, float rv2, float r2) {
    const float y = rsqrtf(r2);
    const float inv = __fmaf_rn(y, __fmaf_rn(__fmul_rn(__fmul_rn(-0.5f, r2), y), y, 0.5f), y);
    const float inv2 = __fmul_rn(inv, inv), r = __fmul_rn(r2, inv);
    const float ea = __fmul_rn(r, k_app), e = __fmul_rn(r, k_range);
    float near = inv2, extra = 0.f;
    if (ea <= 2.f) {
      near = __fmul_rn(c_app, F_s2(ea, __fmul_rn(p_app, inv2)));
      extra = __fsub_rn(near, inv2);
    }
    // both sides of e = 1, without a branch
    const float rest = __fmaf_rn(c_range, F_s2_rest(e, __fmul_rn(p_range, inv2)), extra);
    const float inner = __fmaf_rn(-c_range, F_s2_near(e), near);
    float sc = e > 1.f ? rest : inner;
    sc = __fmul_rn(sc, inv);
    acc[0] = __fmaf_rn(rv0, sc, acc[0]);
    acc[1] = __fmaf_rn(rv1, sc, acc[1]);
    acc[2] = __fmaf_rn(rv2, sc, acc[2]);
  }
};

// The plain form: one thread per particle of the cells of at most heavy_t particles, over the
// coarse cells its range reaches, reading the candidates' codes (fuller cells go to
// k_ppq_heavy).  Candidates go four at a time as independent chains; pairs in range
// are kept in the thread's own shared-memory column and added with PPi::accum in candidate
// order when it may run full and at the end, so that the lanes of a warp evaluate their
// pairs together (128^3 particles at 8 a cell: 0.76 -> 0.42 ms).
constexpr int PP_T = 128, PP_H = 8, PP_U = 4;
template <bool FAST, typename CODE>
__global__ void __launch_bounds__(PP_T) k_pp(Geo G, int64_t np, const CODE* __restrict__ xp,
                                             const int32_t* __restrict__ pcell, const int64_t* __restrict__ cstart,
                                             const int32_t* __restrict__ ires, float* __restrict__ vp,
                                             const StepDev* __restrict__ sd, int heavy_t, float* f2max, float* vmax,
                                             unsigned long long* npairs, unsigned long long* ncand,
                                             const unsigned* __restrict__ abort) {
  __shared__ float4 hb[PP_H][PP_T];
  const int64_t ip = (int64_t)blockIdx.x * PP_T + threadIdx.x;
  // abort: the class lists of a captured step were too short; PM3 is finished for the
  // unlisted subtiles afterwards and PP must follow it, so PP leaves vp alone here
  bool live = ip < np && !(abort && *abort);
  int c = 0;
  if (live) {
    c = pcell[ip];
    live = owned_cell(G, c) && cstart[c + 1] - cstart[c] <= heavy_t;
  }
  float f2 = 0.f, av[3] = {0.f, 0.f, 0.f};
  PPi P;
  P.pairs = P.cand = 0;
  if (live) {
    int g[3];
    cell_coords(G, c, g[0], g[1], g[2]);
    int t[3], u[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      t[d] = g[d] / G.nt;
      u[d] = (g[d] - t[d] * G.nt) / G.ntt;
    }
    float fin[3], xf[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double fr = zfrac((int)xp[3 * ip + d], G);
      fin[d] = __fmul_rn((float)fr, (float)G.rcs);  // offset inside the coarse cell, fine units
      xf[d] = __fmul_rn((float)((double)(g[d] - t[d] * G.nt) + fr), (float)G.rcs);  // xvec*ratio_cs (kick.f90:424)
    }
    P.init(G, g, make_float4(fin[0], fin[1], fin[2], 0.f), ires[subtile_id(G, t, u)]);
    if (!FAST) {
#pragma unroll
      for (int d = 0; d < 3; ++d) P.xf[d] = xf[d];
    }
    const float step = (float)(G.x_res * (double)G.rcs);  // fine cells per code unit, a power of two
    int nh = 0;
    for (int dz = P.lo[2]; dz <= P.hi[2]; ++dz)
      for (int dy = P.lo[1]; dy <= P.hi[1]; ++dy)
        for (int dx = P.lo[0]; dx <= P.hi[0]; ++dx) {
          const int64_t n = nbr_cell(G, c, P.l, g, dx, dy, dz);
          const int64_t s = cstart[n], e = cstart[n + 1];
          P.cand += (unsigned)(e - s);
          const int lq[3] = {P.l[0] + dx, P.l[1] + dy, P.l[2] + dz};
          float base[3];  // cell corner plus half a code unit, less xf: exact when FAST
#pragma unroll
          for (int d = 0; d < 3; ++d) base[d] = (float)(lq[d] * G.rcs) - P.xf[d] + 0.5f * step;
          for (int64_t q0 = s; q0 < e; q0 += PP_U) {
            float rv[PP_U][3], r2[PP_U];
            bool hit[PP_U];
#pragma unroll
            for (int k = 0; k < PP_U; ++k) {
              const bool valid = q0 + k < e;
              const CODE* cp = xp + 3 * (valid ? q0 + k : q0);
#pragma unroll
              for (int d = 0; d < 3; ++d)
                rv[k][d] = FAST ? fmaf((float)cp[d], step, base[d]) : __fsub_rn(pp_xq<false>(G, lq[d], (int)cp[d]), P.xf[d]);
              r2[k] = sumsq3(rv[k][0], rv[k][1], rv[k][2]);
              hit[k] = valid && r2[k] > 0.f && r2[k] < P.range2;
            }
#pragma unroll
            for (int k = 0; k < PP_U; ++k)
              if (hit[k]) {
                if (nh == PP_H) {
#pragma unroll 1
                  for (int h = 0; h < PP_H; ++h) {
                    const float4 r = hb[h][threadIdx.x];
                    P.accum(r.x, r.y, r.z, r.w);
                  }
                  nh = 0;
                }
                hb[nh][threadIdx.x] = make_float4(rv[k][0], rv[k][1], rv[k][2], r2[k]);
                ++nh;
                ++P.pairs;
              }
          }
        }
#pragma unroll 1
    for (int h = 0; h < nh; ++h) {
      const float4 r = hb[h][threadIdx.x];
      P.accum(r.x, r.y, r.z, r.w);
    }
    float f1[3];
    const float mass_scale = sd->pp_mass, v_scale = sd->pp_vscale;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      f1[d] = __fmul_rn(P.acc[d], mass_scale);
      const float v = __fadd_rn(vp[3 * ip + d], __fmul_rn(f1[d], v_scale));
      vp[3 * ip + d] = v;
      av[d] = fabsf(v);
    }
    f2 = sumsq3(f1[0], f1[1], f1[2]);
  }
  block_max_to(f2, f2max);
  block_vmax(av, vmax);
  unsigned long long a = P.pairs, b = P.cand;  // warp sums in 64 bits
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if ((threadIdx.x & 31) == 0 && a) atomicAdd(npairs, a);
  if ((threadIdx.x & 31) == 0 && b) atomicAdd(ncand, b);
}

// =================================================================================
// Total momentum (sum of vp over the particles, per component) in FP64, deterministic:
// each block sums a fixed grid-stride share in a fixed order and a shared-memory tree,
// and writes its partial; the host adds the partials in block order.  MOM_BLOCKS blocks.
// =================================================================================
constexpr int MOM_BLOCKS = 592, MOM_THREADS = 256;
__global__ void __launch_bounds__(MOM_THREADS) k_momentum(const float* __restrict__ vp, int64_t np,
                                                          double* __restrict__ partial) {
  __shared__ double sh[3][MOM_THREADS];
  double s0 = 0.0, s1 = 0.0, s2 = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * MOM_THREADS + threadIdx.x; i < np; i += (int64_t)gridDim.x * MOM_THREADS) {
    s0 += (double)vp[3 * i];
    s1 += (double)vp[3 * i + 1];
    s2 += (double)vp[3 * i + 2];
  }
  sh[0][threadIdx.x] = s0;
  sh[1][threadIdx.x] = s1;
  sh[2][threadIdx.x] = s2;
  __syncthreads();
  for (int h = MOM_THREADS / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h)
#pragma unroll
      for (int d = 0; d < 3; ++d) sh[d][threadIdx.x] += sh[d][threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x < 3) partial[3 * blockIdx.x + threadIdx.x] = sh[threadIdx.x][0];
}

// =================================================================================
// ZIPV int16 velocity codec (utilities/pp_subtile.f90:61 decode, :125 encode), izipv=2:
//   v = tan(pi*vp/(nvbin-1)) / (sqrt(pi/2)/(sigma_vi*vrel_boost))
//   vp = nint((nvbin-1)*atan(sqrt(pi/2)/(sigma_vi*vrel_boost)*v)/pi)
// with nvbin = 2^16 and vrel_boost = 2.5 (parameters.f90:90,135); FP64 as the reference.
// =================================================================================
__device__ __forceinline__ double zipv_scale(float sigma_vi) {
  return sqrt(3.141592653589793 / 2.0) / ((double)sigma_vi * 2.5);
}

__global__ void k_zipv_decode(const int16_t* __restrict__ code, float* __restrict__ v, int64_t n, float sigma_vi) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double arg = 3.141592653589793 * (double)(float)code[i] / (double)65535.f;
  v[i] = (float)(tan(arg) / zipv_scale(sigma_vi));
}

__global__ void k_zipv_encode(const float* __restrict__ v, int16_t* __restrict__ code, int64_t n, float sigma_vi) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = (double)65535.f * atan(zipv_scale(sigma_vi) * (double)v[i]) / 3.141592653589793;
  code[i] = (int16_t)llround(x);
}

// =================================================================================
// int2real (utilities/int2real.f90:68-86): xv(3,np) real(4) = ZIPX offset + cell index in
// coarse-cell units; the real(8) sum is exact, so one rounding to float.
// =================================================================================
__global__ void k_int2real(Geo G, int64_t np, const void* __restrict__ xp, const int32_t* __restrict__ pcell,
                           float* __restrict__ xv) {
  const int64_t ip = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= np) return;
  int g[3];
  cell_coords(G, pcell[ip], g[0], g[1], g[2]);
#pragma unroll
  for (int d = 0; d < 3; ++d)
    xv[3 * ip + d] = __double2float_rn(zfrac(load_code(xp, G.izipx, 3 * ip + d), G) + (double)g[d]);
}

// =================================================================================
// Green's function (Green/Green.f90:1-80) in FP64, stored real32.
// =================================================================================
__global__ void k_green(float* __restrict__ Gk, int n, float apm_soft, float apm_range, float gridsize) {
  const int nh = n / 2 + 1;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)nh * n * n) return;
  const int k1 = (int)(i % nh), k2 = (int)((i / nh) % n), k3 = (int)(i / ((int64_t)nh * n));
  const float inv_n = 1.f / (float)n;
  const double PI = 3.141592653589793;
  auto fs = [&](int k) {  // fftspace(k+1)
    const int m = ((k + 1 + n / 2 - 1) % n) - n / 2;
    return (2.0 * PI) * (double)inv_n * (double)m;
  };
  const double kv[3] = {fs(k1), fs(k2), fs(k3)};
  const float alpha = 4.f / 3.f;
  double Dv[3], ur[3] = {0, 0, 0};
  for (int d = 0; d < 3; ++d) Dv[d] = (double)alpha * sin(kv[d]) + (double)(1.f - alpha) * sin(2 * kv[d]) / 2;
  for (int i3 = -2; i3 <= 2; ++i3)
    for (int i2 = -2; i2 <= 2; ++i2)
      for (int i1 = -2; i1 <= 2; ++i1) {
        const double kn[3] = {kv[0] + 2 * PI * i1, kv[1] + 2 * PI * i2, kv[2] + 2 * PI * i3};
        const double kmag = sqrt(kn[0] * kn[0] + kn[1] * kn[1] + kn[2] * kn[2]);
        if (kmag == 0) continue;  // only k=0, zeroed below
        double prod = 1;
        for (int d = 0; d < 3; ++d) prod *= (kn[d] == 0) ? 1.0 : sin(kn[d] / 2) / (kn[d] / 2);
        const double p2 = prod * prod;
        const double Uk2 = p2 * p2 * p2;
        double y = (double)apm_soft * kmag / 2;
        const double Ss = 12 / (y * y * y * y) * (2 - 2 * cos(y) - y * sin(y));
        double Sr;
        if (apm_range == 0.f) Sr = 0;
        else {
          y = (double)apm_range * kmag / 2;
          Sr = 12 / (y * y * y * y) * (2 - 2 * cos(y) - y * sin(y));
        }
        for (int d = 0; d < 3; ++d) ur[d] += Uk2 * (kn[d] * (Ss * Ss - Sr * Sr) / (kmag * kmag));
      }
  double u2n = 1;
  const double two15 = (double)(2.f / 15.f);
  for (int d = 0; d < 3; ++d) {
    const double s = sin(kv[d] / 2);
    u2n *= 1 - s * s + two15 * s * s * s * s;
  }
  const double num = Dv[0] * ur[0] + Dv[1] * ur[1] + Dv[2] * ur[2];
  const double den = Dv[0] * Dv[0] + Dv[1] * Dv[1] + Dv[2] * Dv[2];
  const float gs2 = gridsize * gridsize;
  double val = (den == 0) ? 0.0 : 4 * PI * num / den / (u2n * u2n) / (double)gs2;
  const int h = n / 2;
  if ((k1 % h == 0) && (k2 % h == 0) && (k3 % h == 0)) val = 0.0;  // Green.f90:71
  Gk[i] = (float)val;
}

// =================================================================================
// Neutrino linear response of the force kernels (kick.f90:23-29; power_nu.f90:179-219
// interp_tf_F, :449-476 nu_correction): tf(k) = interp_tf_F(|k|) * Gk(k) for every mode
// of a Green table, the zero mode set to 1 as nu_correction leaves it.  k of mode
// (i, j, k) (1-based) is (mod(i + n/2, n) - n/2 - 1) * 2 pi / size with `size` the level's
// box side in Mpc/h (box for PM1, box/nnt for PM2, box/nnt/nns for PM3), rounded to real
// as the reference stores kx.  The interpolation is quadratic in log-log through the three
// table points nearest log|k|, in FP32 as the reference computes it.
// =================================================================================
__device__ float nu_interp_tf(const float* __restrict__ klog, const float* __restrict__ tlog, int nb, float kr) {
  const float kn = logf(kr);
  int i1 = 1, i2 = nb;  // 1-based as the reference
  while (i2 - i1 > 1) {
    const int mid = (i1 + i2) / 2;
    if (kn > klog[mid - 1]) i1 = mid;
    else i2 = mid;
  }
  int i3;
  if (kn - klog[i1 - 1] < klog[i2 - 1] - kn) {
    i3 = i2;
    i2 = i1;
    i1 = i1 - 1;
  } else {
    i3 = i2 + 1;
  }
  if (i3 > nb) {
    --i1;
    --i2;
    --i3;
  }
  if (i1 < 1) {  // |k| below the table's second point: the first three points
    i1 = 1;
    i2 = 2;
    i3 = 3;
  }
  const float K1 = klog[i1 - 1], K2 = klog[i2 - 1], K3 = klog[i3 - 1];
  const float T1 = tlog[i1 - 1], T2 = tlog[i2 - 1], T3 = tlog[i3 - 1];
  const float a1 = (T1 - T2) / (K1 - K2);
  const float a2 = (T2 - T3) / (K2 - K3);
  const float k2 = (a1 - a2) / (K1 - K3);
  const float b2 = a1 - k2 * (K1 + K2);
  const float c2 = T1 - k2 * K1 * K1 - b2 * K1;
  return expf(k2 * kn * kn + b2 * kn + c2);
}

__global__ void k_nu_rescale(int n, double size, const float* __restrict__ gk, float* __restrict__ tf,
                             const float* __restrict__ klog, const float* __restrict__ tlog, int nb, float scale) {
  const int nh = n / 2 + 1;
  const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= (int64_t)nh * n * n) return;
  if (nb < 3) {  // no table: the constant (1 - f_nu) of initialize.f90:316-322
    tf[m] = scale * gk[m];
    return;
  }
  const int i = (int)(m % nh) + 1, j = (int)((m / nh) % n) + 1, k = (int)(m / ((int64_t)nh * n)) + 1;
  if (i == 1 && j == 1 && k == 1) {  // zero frequency
    tf[m] = 1.f;
    return;
  }
  const double f = 2.0 * 3.141592653589793 / size;
  const float kx = (float)(((i + n / 2) % n - n / 2 - 1) * f);
  const float ky = (float)(((j + n / 2) % n - n / 2 - 1) * f);
  const float kz = (float)(((k + n / 2) % n - n / 2 - 1) * f);
  const float kr = sqrtf(kx * kx + ky * ky + kz * kz);
  tf[m] = nu_interp_tf(klog, tlog, nb, kr) * gk[m];
}

}  // namespace cube
