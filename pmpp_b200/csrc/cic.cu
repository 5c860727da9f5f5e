// Cell sort, deterministic CIC scatter, CIC gather and their adjoints.
//
// Reference semantics: cic/enmesh.py:34-165 (binning, weights, weight
// gradients), cic/scatter.py:315-437 and cic/gather.py:452-548 (forward and
// hand-written VJPs), cic/pallas.py:268-409 (the GPU kernels this replaces).
//
// B200 design:
//  * particles are counting-sorted by the mesh row (x, y) of their lower CIC
//    corner.  Bin order is the reference's raveled cell-key order
//    ((x*My + y)*Mz + z, core/utils.py:292-326) at row granularity;
//  * the scatter is a pull kernel: one CTA owns an RX x RY block of output
//    rows, reads the particles of the (RX+1) x (RY+1) source rows that can
//    reach it, and accumulates in shared memory in 64-bit fixed point (split
//    over two 32-bit planes).  The
//    result is independent of accumulation order (bit-deterministic), every
//    output cell is written exactly once with coalesced stores, and no
//    global atomics or mesh zero-fill pass are needed;
//  * gathers and adjoint position terms walk particles in sorted order so the
//    eight corner loads of neighbouring threads hit the same cache lines.
#include <cstdio>
#include <tuple>
#include <type_traits>

#include "pmb_cic_device.cuh"
#include "pmb_common.cuh"
#include "pmb_kernels.cuh"
#include "pmb_tma.cuh"

namespace pmb {

// Sticky device-wide flags (DeviceFlag bits), read and cleared by
// pmb_device_status.
__device__ unsigned int g_device_flags = 0;

// Raises flag f in the sorted buffer's status word (if any) and device-wide.
__device__ __forceinline__ void raise_flag(uint32_t* status, unsigned int f) {
  if (status != nullptr) atomicOr(status, f);
  atomicOr(&g_device_flags, f);
}

// Consumers of a sorted buffer whose sort was flagged write nothing.
__device__ __forceinline__ bool flagged(const uint32_t* status) { return status != nullptr && *status != 0u; }

// ---------------------------------------------------------------------------
// Binning
// ---------------------------------------------------------------------------
// Count particles per row.  Optionally applies the drift disp += vel * D
// first (integrator.py:223-225, two roundings as in the reference) and writes
// the drifted displacement back.  With a shift the mesh origin moves
// (BinShift); particles with valid[i] == 0 go to the extra bin after the last
// row (their records trail the sorted array with kMaskedKey).
//
// Ranks come from one atomic per run of equal rows in the warp: particles come
// in lattice order, z fastest, so neighbouring lanes mostly share a row, and a
// run is found with one shuffle and one ballot.  (Grouping all equal rows of
// the warp with __match_any_sync saves some atomics but its own issue was the
// bound: 342 us for 256^3 and 2.71 ms for 512^3 clustered particles, 174 us
// and 1.26 ms by runs; the bytes take 0.07 and 0.6 ms.)  kSortPer particles a
// thread, a block apart, so that their loads overlap.
//
// On meshes of few rows (FEW) a warp of particles in no order, more than eight
// runs of rows that repeat, groups equal rows all the same: the atomics on those
// rows are the bound there (sorts of 2^22 shuffled particles by runs / grouped, us:
// 4^3 cells 730 / 243, 8^3 1146 / 770, 16^3 1056 / 980, 24^3 631 / 617, 32^3 434 / 432).
constexpr int kSortThreads = 256;
constexpr int kSortPer = 4;
constexpr int64_t kFewRows = 1024;

__device__ __forceinline__ uint32_t row_bin(const int16_t* __restrict__ pmid, float d0, float d1, float d2, int64_t i,
                                            Mesh3 m, float cell, const BinShift& sh,
                                            const uint8_t* __restrict__ valid) {
  if (valid != nullptr && !valid[i]) return (uint32_t)m.rows();
  const Binned b = bin_particle(pmid, d0, d1, d2, i, m, cell, sh);
  return (uint32_t)b.cx * (uint32_t)m.ny + (uint32_t)b.cy;
}

template <bool FEW>
__global__ void __launch_bounds__(kSortThreads) bin_count_kernel(const int16_t* pmid,
                                                                 float* __restrict__ disp,
                                                                 const float* vel, float drift, int64_t n,
                                                                 Mesh3 m, float cell, BinShift sh,
                                                                 const uint8_t* valid,
                                                                 uint32_t* __restrict__ counts,
                                                                 uint32_t* __restrict__ row_of,
                                                                 uint32_t* __restrict__ rank_of,
                                                                 uint32_t* __restrict__ flag) {
  wait_for_previous();
  let_next_start();
  const int64_t base = (int64_t)blockIdx.x * (kSortThreads * kSortPer) + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const unsigned upto = 0xFFFFFFFFu >> (31 - lane);  // lanes 0 .. lane
  float d[kSortPer][3];
#pragma unroll
  for (int k = 0; k < kSortPer; ++k) {
    const int64_t i = base + k * kSortThreads;
#pragma unroll
    for (int a = 0; a < 3; ++a) d[k][a] = i < n ? disp[3 * i + a] : 0.f;
  }
  if (vel != nullptr) {
#pragma unroll
    for (int k = 0; k < kSortPer; ++k) {
      const int64_t i = base + k * kSortThreads;
      if (i < n) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          d[k][a] = __fadd_rn(d[k][a], __fmul_rn(vel[3 * i + a], drift));
          disp[3 * i + a] = d[k][a];
        }
      }
    }
  }
  uint32_t head_base[kSortPer];
  int head[kSortPer], after_head[kSortPer];
  bool bad = false;
#pragma unroll
  for (int k = 0; k < kSortPer; ++k) {
    const int64_t i = base + k * kSortThreads;
    bad |= !(isfinite(d[k][0]) && isfinite(d[k][1]) && isfinite(d[k][2]));
    uint32_t row = 0xFFFFFFFFu;
    if (i < n) row_of[i] = row = row_bin(pmid, d[k][0], d[k][1], d[k][2], i, m, cell, sh, valid);
    const uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, row, 1);
    const unsigned heads = __ballot_sync(0xFFFFFFFFu, lane == 0 || row != prev);
    head[k] = 31 - __clz(heads & upto);
    after_head[k] = lane - head[k];
    const unsigned after = heads & ~upto;
    int len = (after ? __ffs(after) - 1 : 32) - lane;
    if (FEW && __popc(heads) > 8) {
      const unsigned equal = __match_any_sync(0xFFFFFFFFu, row);
      head[k] = __ffs(equal) - 1;
      after_head[k] = __popc(equal & upto) - 1;
      len = __popc(equal);
    }
    head_base[k] = 0;
    if (head[k] == lane && i < n) head_base[k] = atomicAdd(&counts[row], (uint32_t)len);
  }
  if (bad) raise_flag(flag, kFlagNonFiniteDisp);
#pragma unroll
  for (int k = 0; k < kSortPer; ++k) {
    const int64_t i = base + k * kSortThreads;
    const uint32_t b = __shfl_sync(0xFFFFFFFFu, head_base[k], head[k]);
    if (i < n) rank_of[i] = b + (uint32_t)after_head[k];
  }
}

// Records to their places: bound by the scattered stores (about one 128-byte
// line per run of equal rows for the record and one for the index; 0.29 ms for
// 256^3 clustered particles against 0.11 ms for the bytes).  Two or four
// particles a thread, streaming loads and forming the row again instead of
// reading row_of all measured slower (0.31 - 0.33 ms).
__global__ void __launch_bounds__(kSortThreads) bin_place_kernel(const int16_t* pmid,
                                                                 const float* disp, int64_t n, Mesh3 m,
                                                                 float cell, BinShift sh,
                                                                 const uint32_t* offs,
                                                                 const uint32_t* row_of,
                                                                 const uint32_t* rank_of,
                                                                 Rec* __restrict__ rec, uint32_t* __restrict__ perm) {
  wait_for_previous();
  let_next_start();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t row = row_of[i];
  const uint32_t dst = offs[row] + rank_of[i];
  Rec r;
  if (row == (uint32_t)m.rows()) {
    r.fx = r.fy = r.fz = 0.f;
    r.key = kMaskedKey;
  } else {
    const Binned b = bin_particle(pmid, disp[3 * i], disp[3 * i + 1], disp[3 * i + 2], i, m, cell, sh);
    r.fx = b.fx;
    r.fy = b.fy;
    r.fz = b.fz;
    r.key = row * (uint32_t)m.nz + (uint32_t)b.cz;
  }
  rec[dst] = r;
  perm[dst] = (uint32_t)i;
}

// Exclusive scan of row counts: one block up to kScanOne entries (the row
// counts of a 128^3 mesh; 4.6 us against 7 of the three launches it replaces, with two
// launches saved on the host), else two launches over tiles of 4096 entries,
// the second adding the sum of the tiles before its own.
constexpr int kScanThreads = 1024;
constexpr int kScanPer = 4;  // (scan_one_kernel moves these as one vector)
constexpr int kScanTile = kScanThreads * kScanPer;
constexpr int kScanOneTiles = 4;
constexpr int64_t kScanOne = kScanOneTiles * kScanTile + 1;

__device__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* sh, uint32_t* total) {
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < (blockDim.x >> 5) ? sh[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
      if (lane >= o) w += y;
    }
    sh[lane] = w;
  }
  __syncthreads();
  uint32_t warp_off = warp ? sh[warp - 1] : 0;
  if (total) *total = sh[(blockDim.x >> 5) - 1];
  uint32_t r = warp_off + x - v;
  __syncthreads();
  return r;
}

// A flag word raised by the counting pass, handed on to the sorted buffer's
// status word by the scan (both may be null).
__device__ __forceinline__ void hand_on_flag(const uint32_t* flag, uint32_t* status) {
  if (status != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *status = flag != nullptr ? *flag : 0u;
}

// All entries in one block: kScanOneTiles coalesced groups of four entries a
// thread, scanned side by side.  The last entry (n - 1) is only written: no
// exclusive sum contains its count.
__global__ void __launch_bounds__(kScanThreads) scan_one_kernel(const uint32_t* in, uint32_t* out, int64_t n,
                                                                const uint32_t* flag, uint32_t* status) {
  __shared__ uint32_t sh[kScanOneTiles][33];
  wait_for_previous();
  let_next_start();
  hand_on_flag(flag, status);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t last = n - 1;
  const bool vec = (((uintptr_t)in | (uintptr_t)out) & 15) == 0;
  uint32_t v[kScanOneTiles][kScanPer], x[kScanOneTiles], own[kScanOneTiles];
#pragma unroll
  for (int c = 0; c < kScanOneTiles; ++c) {
    const int64_t base = (int64_t)c * kScanTile + (int64_t)threadIdx.x * kScanPer;
    if (vec && base + kScanPer <= last) {
      const uint4 q = *reinterpret_cast<const uint4*>(in + base);
      v[c][0] = q.x;
      v[c][1] = q.y;
      v[c][2] = q.z;
      v[c][3] = q.w;
    } else {
#pragma unroll
      for (int j = 0; j < kScanPer; ++j) v[c][j] = base + j < last ? in[base + j] : 0u;
    }
    own[c] = x[c] = v[c][0] + v[c][1] + v[c][2] + v[c][3];
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
#pragma unroll
    for (int c = 0; c < kScanOneTiles; ++c) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x[c], o);
      if (lane >= o) x[c] += y;
    }
  if (lane == 31)
#pragma unroll
    for (int c = 0; c < kScanOneTiles; ++c) sh[c][warp] = x[c];
  __syncthreads();
  if (warp < kScanOneTiles) {
    uint32_t w = sh[warp][lane];
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
      if (lane >= o) w += y;
    }
    sh[warp][lane] = w;
  }
  __syncthreads();
  uint32_t carry = 0;
#pragma unroll
  for (int c = 0; c < kScanOneTiles; ++c) {
    const int64_t base = (int64_t)c * kScanTile + (int64_t)threadIdx.x * kScanPer;
    const uint32_t o0 = carry + (warp ? sh[c][warp - 1] : 0u) + x[c] - own[c];
    const uint32_t o1 = o0 + v[c][0], o2 = o1 + v[c][1], o3 = o2 + v[c][2];
    if (vec && base + kScanPer <= last) {
      *reinterpret_cast<uint4*>(out + base) = make_uint4(o0, o1, o2, o3);
    } else {
      const uint32_t o[kScanPer] = {o0, o1, o2, o3};
#pragma unroll
      for (int j = 0; j < kScanPer; ++j)
        if (base + j < last) out[base + j] = o[j];
    }
    carry += sh[c][31];
  }
  if (threadIdx.x == 0) out[last] = carry;
}

__global__ void __launch_bounds__(kScanThreads) scan_tiles_kernel(const uint32_t* in, uint32_t* out, int64_t n,
                                                                  uint32_t* __restrict__ tile_sums,
                                                                  const uint32_t* flag, uint32_t* status) {
  __shared__ uint32_t sh[32];
  wait_for_previous();
  let_next_start();
  hand_on_flag(flag, status);
  int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanPer;
  uint32_t v[kScanPer];
  uint32_t s = 0;
  for (int j = 0; j < kScanPer; ++j) {
    v[j] = (base + j < n) ? in[base + j] : 0u;
    s += v[j];
  }
  uint32_t total;
  uint32_t off = block_exclusive_scan(s, sh, &total);
  for (int j = 0; j < kScanPer; ++j) {
    if (base + j < n) out[base + j] = off;
    off += v[j];
  }
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// Adds the sum of the tiles before this block's own (block 0 has none).
__global__ void __launch_bounds__(kScanThreads) scan_add_kernel(uint32_t* __restrict__ out, int64_t n,
                                                                const uint32_t* tile_sums) {
  __shared__ uint32_t sh[32];
  wait_for_previous();
  let_next_start();
  const int64_t tile = (int64_t)blockIdx.x + 1;
  uint32_t s = 0;
  for (int64_t t = threadIdx.x; t < tile; t += kScanThreads) s += tile_sums[t];
  uint32_t before;
  block_exclusive_scan(s, sh, &before);
#pragma unroll
  for (int j = 0; j < kScanPer; ++j) {
    const int64_t i = tile * kScanTile + j * kScanThreads + threadIdx.x;
    if (i < n) out[i] += before;
  }
}

int64_t scan_tmp_elems(int64_t len) { return (len + kScanTile - 1) / kScanTile + 1; }

// Exclusive scan of len uint32 values (in == out allowed); tile_sums needs
// scan_tmp_elems(len) entries.  flag / status: hand_on_flag.
static int exclusive_scan(const uint32_t* in, uint32_t* out, int64_t len, uint32_t* tile_sums, const uint32_t* flag,
                          uint32_t* status, bool early, cudaStream_t s) {
  if (len <= 0) return kOk;
  if (len <= kScanOne) {
    PMB_CUDA_CHECK(launch_dependent(early, scan_one_kernel, 1, kScanThreads, 0, s, in, out, len, flag, status));
  } else {
    const int64_t ntiles = (len + kScanTile - 1) / kScanTile;
    PMB_CUDA_CHECK(launch_dependent(early, scan_tiles_kernel, (int)ntiles, kScanThreads, 0, s, in, out, len, tile_sums,
                                    flag, status));
    PMB_CUDA_CHECK(launch_dependent(early, scan_add_kernel, (int)(ntiles - 1), kScanThreads, 0, s, out, len,
                                    tile_sums));
  }
  return kOk;
}

int exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t len, uint32_t* tile_sums, cudaStream_t s) {
  return exclusive_scan(in, out, len, tile_sums, nullptr, nullptr, false, s);
}

int64_t bin_scratch_bytes(int64_t n, Mesh3 m) {
  int64_t rows = m.rows();
  int64_t ntiles = (rows + 1 + kScanTile - 1) / kScanTile;
  return align_up(4 * (rows + 1), 256) * 2 + align_up(4 * n, 256) * 2 + align_up(4 * (ntiles + 1), 256);
}

// Sort particles by lower-corner row.  Outputs rec[n], perm[n] and
// offs[rows + 1] (offs lives inside the caller's scratch, returned pointer).
int bin_particles(const int16_t* pmid, float* disp, const float* vel, float drift, int64_t n, Mesh3 m, float cell,
                  Rec* rec, uint32_t* perm, uint32_t* offs, void* scratch, cudaStream_t s, const BinShift* shift,
                  const uint8_t* valid, uint32_t* status) {
  BinShift sh{0, 0, 0, 0.f, 0.f, 0.f};
  if (shift != nullptr) sh = *shift;
  int64_t rows = m.rows();
  char* p = (char*)scratch;
  const int64_t len = rows + 1;
  uint32_t* counts = (uint32_t*)p;
  p += align_up(4 * len, 256);
  // the counting pass raises its flag in the word after the counts, cleared
  // together with them (a separate launch costs 2 us)
  uint32_t* flag = (uint32_t*)p;
  p += 256;
  uint32_t* row_of = (uint32_t*)p;
  p += align_up(4 * n, 256);
  uint32_t* rank_of = (uint32_t*)p;
  p += align_up(4 * n, 256);
  uint32_t* tile_sums = (uint32_t*)p;
  PMB_CUDA_CHECK(cudaMemsetAsync(counts, 0, align_up(4 * len, 256) + 4, s));
  const bool early = small_mesh(m.nx, m.ny, m.nz);
  const auto grid_of = [n](int per) { return (int)((n + kSortThreads * per - 1) / (kSortThreads * per)); };
  if (n > 0) {
    auto k = rows <= kFewRows ? bin_count_kernel<true> : bin_count_kernel<false>;
    PMB_CUDA_CHECK(launch_dependent(early, k, grid_of(kSortPer), kSortThreads, 0, s, pmid, disp, vel, drift, n, m, cell,
                                    sh, valid, counts, row_of, rank_of, flag));
  }
  int st = exclusive_scan(counts, offs, len, tile_sums, flag, status, early, s);
  if (st != kOk) return st;
  if (n > 0)
    PMB_CUDA_CHECK(launch_dependent(early, bin_place_kernel, grid_of(1), kSortThreads, 0, s, pmid, disp, n, m, cell, sh,
                                    offs, row_of, rank_of, rec, perm));
  return kOk;
}

// ---------------------------------------------------------------------------
// Fixed-point scale for the deterministic scatter
// ---------------------------------------------------------------------------
// Contributions val*w are converted to int64 units of 1/scale with the power
// of two scale = 2^e / 2^ceil(log2 max|val|), e = 62 - ceil(log2(n + 1)) (at
// most 52), so that the sum of up to n contributions of magnitude <= max|val|
// cannot overflow and val*w*scale is exact in float.
// Four values a load where they are aligned; one atomic a block, and only if
// it raises the maximum (an atomic per warp on the one word was the bound: 24
// us for 3.2 M values, now 5; 49 -> 36 us for 50 M).
__global__ void __launch_bounds__(256) absmax_kernel(const float* __restrict__ v, int64_t count,
                                                     unsigned int* __restrict__ out) {
  __shared__ float sh[8];
  const float inf = __int_as_float(0x7f800000);
  float mx = 0.f;
  auto take = [&](float x) {
    const float a = fabsf(x);
    if (a > mx || a != a) mx = (a != a) ? inf : a;
  };
  const int64_t step = (int64_t)gridDim.x * blockDim.x, t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t n4 = ((uintptr_t)v & 15) == 0 ? count >> 2 : 0;
  for (int64_t i = t; i < n4; i += step) {
    const float4 x = reinterpret_cast<const float4*>(v)[i];
    take(x.x);
    take(x.y);
    take(x.z);
    take(x.w);
  }
  for (int64_t i = 4 * n4 + t; i < count; i += step) take(v[i]);
  for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) mx = fmaxf(mx, sh[w]);
    const unsigned int bits = __float_as_uint(mx);
    if (bits > *reinterpret_cast<volatile unsigned int*>(out)) atomicMax(out, bits);
  }
}

__global__ void scale_from_absmax_kernel(const unsigned int* __restrict__ bits, double pow2e, double* __restrict__ scale) {
  float mx = __uint_as_float(*bits);
  // A non-finite maximum leaves no usable scale: flag it with a NaN scale.
  if (!(mx < __int_as_float(0x7f800000))) {
    *scale = __longlong_as_double(0x7ff8000000000000ll);
    return;
  }
  *scale = fixed_point_scale(pow2e, mx);
}

double fixed_point_pow2(int64_t n) {
  int e = 62;
  int64_t t = n + 1;
  int lg = 0;
  while ((int64_t(1) << lg) < t) ++lg;
  e -= lg;
  if (e > 52) e = 52;
  return ldexp(1.0, e);
}

int compute_scale(const float* val, int64_t count, int64_t n, double* scale_dev, unsigned int* tmp, cudaStream_t s) {
  PMB_CUDA_CHECK(cudaMemsetAsync(tmp, 0, sizeof(unsigned int), s));
  if (count > 0) {
    int64_t blocks = (count + 1023) / 1024;
    if (blocks > 148 * 8) blocks = 148 * 8;
    absmax_kernel<<<(unsigned)blocks, 256, 0, s>>>(val, count, tmp);
  }
  scale_from_absmax_kernel<<<1, 1, 0, s>>>(tmp, fixed_point_pow2(n), scale_dev);
  PMB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

// ---------------------------------------------------------------------------
// Pull scatter
// ---------------------------------------------------------------------------
// One block owns RX x RY output rows and pulls the particles of the
// (RX + 1) x (RY + 1) source rows that reach them.  Each contribution q =
// rint(val * w * scale) (64 bits in scatter_tile, pmb_cic_device.cuh) is split
// as q = h 2^s + l, and h and l are summed by 32-bit shared atomics on two
// planes (8 bytes per output cell); the recombined sum equals the 64-bit sum
// exactly, so the output is bit-identical to scatter_tile's and independent of
// the particle order.
//
// The kernel is bound by the shared atomics (L1 throughput 92%; the memory it
// must touch takes a third of its time), after the split was made of few
// instructions; with one corner set, conversion and address at a time it was
// bound by instruction issue (800 instructions per particle; now 380): one
// channel 24.4 -> 8.7 us for 64^3 particles on 128^3 cells, 519 -> 281 us for
// 256^3 on 512^3, 3065 -> 2190 us for 512^3 on 1024^3; three channels 1312 ->
// 822 us for 256^3 on 512^3.  The value is scaled by the power of two
// scale 2^-s 2^-49 first, so that a contribution c counts units of 2^-49 of h
// (an exact change of exponent); then t = c 2^-100 is a subnormal float whose
// bit pattern is the integer h (rounded by the multiplication itself, linear
// up to 2^24), r = c - t 2^100 is its exact remainder, and r 2^(s - 100) is a
// subnormal whose bits are l.  Two z corners go through each step as one
// packed operation (f32x2).
//   unsigned values: h = floor, so 0 <= l <= 2^s and both planes count in
//     32 unsigned bits: s >= E - 24, s >= L + E - 32, s <= 24, s <= 32 - L;
//   signed values: |val| goes through with h to nearest and l biased by
//     2^(s - 1), and the sign is applied to the integers:
//     s >= E - 24, s >= L + E - 31, 2 <= s <= 23, s <= 32 - L
// where K < 2^L particles can reach a cell of the block and |q| <= 2^E.  A
// block without such an s (very small particle counts, or a block holding very
// many particles), or a scale outside [2^-50, 2^100], adds the 64-bit q with
// 64-bit atomics on the same 8 bytes.
//
// Particles are handed out one a thread over the block's source rows: for one
// x the rows y0 - 1 .. y0 + RY - 1 are contiguous in the sorted records
// (pass 0; row ny - 1 before row 0 is pass 1), so every lane is busy whatever
// the number of particles in a row, and a record's own key says which output
// rows it reaches.  NZP: the row stride of the accumulator (nz rounded up to
// one of a few lengths), a constant so that every corner's address is one of
// two registers plus an immediate.
constexpr int kRowThreads = 256;

template <int C, int RX, int RY, int NZP, bool EXACT, bool SIGNED>
__global__ void __launch_bounds__(kRowThreads)
    scatter_rows_kernel(const Rec* rec, const uint32_t* perm,
                        const uint32_t* offs, Mesh3 m, FastDiv by_nz, FastDiv by_nby,
                        const float* val, int val_sorted, float val_const,
                        const double* scale_dev, double scale_const, int E, int dup, int mode,
                        float src_mul, float* __restrict__ out, uint32_t* __restrict__ status) {
  constexpr int CH = RX * RY * NZP;   // cells of one channel, row (lx, ly) at (lx * RY + ly) * NZP
  constexpr int PLANE = C * CH;       // cells per plane
  constexpr int GROUPS = PLANE / 4;   // groups of four cells per plane
  constexpr int T = kRowThreads;
  static_assert(NZP % 4 == 0, "rows of whole groups");
  wait_for_previous();
  let_next_start();
  if (flagged(status)) return;
  const double scale = scale_dev != nullptr ? *scale_dev : scale_const;
  if (!(scale == scale)) {  // NaN scale: a non-finite value
    if (threadIdx.x == 0) raise_flag(status, kFlagNonFiniteValue);
    return;
  }
  extern __shared__ __align__(16) unsigned int acc[];  // 2 * PLANE
  // source segments: [pass][k] for source row x0 + k - 1
  __shared__ uint32_t s_beg[2][RX + 1], s_cnt[2][RX + 1], s_row[2][RX + 1];
  const int tid = threadIdx.x;
  const int nz = EXACT ? NZP : m.nz, nz4 = (nz + 3) >> 2;
  int x0, y0;
  {
    const uint32_t bx = div_by(blockIdx.x, by_nby);
    x0 = (int)bx * RX;
    y0 = (int)(blockIdx.x - bx * (uint32_t)((m.ny + RY - 1) / RY)) * RY;
  }
  const int rxe = RX == 1 ? 1 : min(RX, m.nx - x0), rye = RY == 1 ? 1 : min(RY, m.ny - y0);  // rows in the mesh
  if (tid < 2 * (RX + 1)) {
    const int pass = tid > RX, k = tid - pass * (RX + 1);
    uint32_t b = 0, c = 0, row = 0;
    if (k - 1 < rxe && (pass == 0 || y0 == 0)) {
      const int x = k == 0 ? (x0 == 0 ? m.nx - 1 : x0 - 1) : x0 + k - 1;
      row = (uint32_t)((int64_t)x * m.ny) + (uint32_t)(pass == 0 ? y0 : m.ny);  // the record's ly = its row - this
      const int64_t lo = pass == 0 ? (int64_t)row - (y0 > 0) : (int64_t)row - 1;
      const int64_t hi = pass == 0 ? (int64_t)row + rye : (int64_t)row;
      b = offs[lo];
      c = offs[hi] - b;
    }
    s_beg[pass][k] = b;
    s_cnt[pass][k] = c;
    s_row[pass][k] = EXACT ? row * (uint32_t)NZP : row;
  }
  {
    uint4* a4 = reinterpret_cast<uint4*>(acc);
#pragma unroll 4
    for (int g = tid; g < 2 * GROUPS; g += T)
      if (EXACT || g % (NZP / 4) < nz4) a4[g] = make_uint4(0u, 0u, 0u, 0u);
  }
  __syncthreads();
  uint32_t kcell = 0;  // particles that may reach one cell: those of two neighbouring source x
#pragma unroll
  for (int k = 0; k < RX; ++k) kcell = max(kcell, s_cnt[0][k] + s_cnt[1][k] + s_cnt[0][k + 1] + s_cnt[1][k + 1]);
  int s;
  bool split;
  {
    const uint64_t kmax = (uint64_t)kcell * (uint64_t)dup;
    const int L = kmax ? 64 - __clzll((long long)kmax) : 0;  // kmax < 2^L
    const int lo = max(max(E - 24, L + E - (SIGNED ? 31 : 32)), SIGNED ? 2 : 1);
    const int hi = min(SIGNED ? 23 : 24, 32 - L);
    // half of the bits to each plane where that is allowed, so that the sums
    // of both stay within the epilogue's short conversion
    s = max(lo, min(hi, (E + 1) / 2));
    split = lo <= hi && scale >= 0x1p-50 && scale <= 0x1p100;
  }
  unsigned long long* acc64 = reinterpret_cast<unsigned long long*>(acc);
  if (!EXACT && !split) {  // the 64-bit sums lie elsewhere in the rows than the planes cleared above
    for (int g = tid; g < PLANE; g += T) acc64[g] = 0ull;
    __syncthreads();
  }
  const float y_scale = split ? __fmul_rn((float)scale, pow2f(-s - 49)) : 0.f;
  const F2 to_h = f2_pack(pow2f(-100), pow2f(-100)), back = f2_pack(-pow2f(100), -pow2f(100));
  const F2 to_l = f2_pack(pow2f(s - 100), pow2f(s - 100));
  const int bias = SIGNED ? 1 << (s - 1) : 0;
  const F2 bias2 = f2_pack(__int_as_float(bias), __int_as_float(bias));
  int* const planes = reinterpret_cast<int*>(acc);

  // One particle: r its record, at its cell in tile row (sx, ly) of channel 0
  // (RX, RY == 1: of the one row), dz the step to its upper z cell; x0in ..
  // y1in: the rows that its lower / upper corners along x and y fall into are
  // this block's.
  auto visit = [&](const Rec& r, uint32_t i, int at, int dz, int sx, bool low_y, bool x0in, bool x1in, bool y0in,
                   bool y1in, auto split_tag) {
    constexpr bool SPLIT = decltype(split_tag)::value;
    float v[C];
    int sgn[C], nbias[C];
    if (val != nullptr) {
      const int64_t src = val_sorted ? (int64_t)i : (int64_t)perm[i];
#pragma unroll
      for (int c = 0; c < C; ++c) v[c] = val[src * C + c];
    } else {
#pragma unroll
      for (int c = 0; c < C; ++c) v[c] = val_const;
    }
    if (SPLIT) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        if (SIGNED) {
          sgn[c] = v[c] < 0.f ? -1 : 1;
          nbias[c] = -bias * sgn[c];
          v[c] = fabsf(v[c]);
        }
        v[c] = __fmul_rn(v[c], y_scale);
      }
    }
    const float wx0 = axis_weight(r.fx, 0), wx1 = axis_weight(r.fx, 1);
    const float wy0 = axis_weight(r.fy, 0), wy1 = axis_weight(r.fy, 1);
    const F2 wz = f2_pack(axis_weight(r.fz, 0), axis_weight(r.fz, 1));
    // with one output row along an axis a source row reaches it by one corner
    constexpr int NX = RX == 1 ? 1 : 2, NY = RY == 1 ? 1 : 2;
    int* const a0 = planes + at;
    int* const a1 = a0 + dz;
#pragma unroll
    for (int bx = 0; bx < NX; ++bx) {
      const float wx = RX == 1 ? (sx < 0 ? wx1 : wx0) : (bx ? wx1 : wx0);
#pragma unroll
      for (int by = 0; by < NY; ++by) {
        const float wy = RY == 1 ? (low_y ? wy1 : wy0) : (by ? wy1 : wy0);
        if (!((bx ? x1in : x0in) && (by ? y1in : y0in))) continue;
        const float wxy = __fmul_rn(wx, wy);
        const F2 w = f2_mul(f2_pack(wxy, wxy), wz);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const int o = c * CH + (bx * RY + by) * NZP;
          const F2 q = f2_mul(f2_pack(v[c], v[c]), w);
          if (SPLIT) {
            const F2 t = SIGNED ? f2_mul(q, to_h) : f2_mul_rz(q, to_h);
            const F2 rem = f2_fma(t, back, q);
            const F2 u = SIGNED ? f2_fma(rem, to_l, bias2) : f2_mul(rem, to_l);
            int h0, h1, l0, l1;
            f2_bits(t, h0, h1);
            f2_bits(u, l0, l1);
            if (SIGNED) {
              h0 *= sgn[c];
              h1 *= sgn[c];
              l0 = l0 * sgn[c] + nbias[c];
              l1 = l1 * sgn[c] + nbias[c];
            }
            atomicAdd(a0 + o, h0);
            atomicAdd(a0 + o + PLANE, l0);
            atomicAdd(a1 + o, h1);
            atomicAdd(a1 + o + PLANE, l1);
          } else {
            int q0, q1;
            f2_bits(q, q0, q1);
            atomicAdd(&acc64[at + o], (unsigned long long)__double2ll_rn((double)__int_as_float(q0) * scale));
            atomicAdd(&acc64[at + dz + o], (unsigned long long)__double2ll_rn((double)__int_as_float(q1) * scale));
          }
        }
      }
    }
  };
  auto visits = [&](auto split_tag) {
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      // visits before segment k, record index = visit index + dk[k] (mod 2^32)
      uint32_t pk[RX + 2], dk[RX + 1], bk[RX + 1];
      pk[0] = 0;
#pragma unroll
      for (int k = 0; k <= RX; ++k) {
        pk[k + 1] = pk[k] + s_cnt[pass][k];
        dk[k] = s_beg[pass][k] - pk[k];
        bk[k] = s_row[pass][k];
      }
#pragma unroll 1
      for (uint32_t vi = tid; vi < pk[RX + 1]; vi += T) {
        uint32_t i = vi + dk[0], b = bk[0];
        int sx = -1;
#pragma unroll
        for (int k = 1; k <= RX; ++k)
          if (vi >= pk[k]) {
            i = vi + dk[k];
            b = bk[k];
            sx = k - 1;
          }
        const Rec r = rec[i];
        const bool x0in = RX == 1 || sx >= 0, x1in = RX == 1 || sx + 1 < rxe;
        if (EXACT) {
          // cell counted from the tile's row 0 of this x: ly * NZP + cz
          const int lin = (int)(r.key - b);
          const bool low_y = lin < 0;
          const bool top = (uint32_t)(lin + 1 + NZP) % (uint32_t)NZP == 0;
          const int at = (RX == 1 ? 0 : sx * RY * NZP) + (RY == 1 && low_y ? lin + NZP : lin);
          visit(r, i, at, top ? 1 - NZP : 1, sx, low_y, x0in, x1in, RY == 1 || !low_y,
                RY == 1 || lin < (rye - 1) * NZP, split_tag);
        } else {
          const uint32_t rowk = div_by(r.key, by_nz);
          const int ly = (int)(rowk - b), cz = (int)(r.key - rowk * (uint32_t)nz);
          const int at = ((RX == 1 ? 0 : sx * RY) + (RY == 1 ? 0 : ly)) * NZP + cz;
          visit(r, i, at, cz + 1 == nz ? 1 - nz : 1, sx, ly < 0, x0in, x1in, RY == 1 || ly >= 0,
                RY == 1 || ly + 1 < rye, split_tag);
        }
      }
    }
  };
  if (split)
    visits(std::true_type{});
  else
    visits(std::false_type{});
  __syncthreads();

  // Epilogue: (float)(sum / scale) as scatter_tile computes it; mode 0 the
  // density, mode 1 the Poisson source (rho - 1) * src_mul
  // (gravity.py:628-630).  Plane sums below 2^23 (signed: within 2^22)
  // convert exactly through the bits of 2^23 + h and one fma forms h 2^s + l
  // with a single rounding (|sum| < 2^53, so this equals the
  // double-precision route, which the other cells take).
  const double inv = __hiloint2double(0x7FE00000 - __double2hiint(scale), 0);  // 1 / scale, a power of two
  const float invf = (float)inv, two_s = pow2f(split ? s : 0);
  const bool fconv = split && invf >= 0x1p-126f;
  constexpr unsigned kOff = SIGNED ? 0x4B400000u : 0x4B000000u;  // (sums modulo 2^32, so in unsigned)
  const F2 near2 = f2_pack(-__uint_as_float(kOff), -__uint_as_float(kOff));
  const F2 two_s2 = f2_pack(two_s, two_s), inv2 = f2_pack(invf, invf);
  // exact integers in double precision through the bits of 2^52 + h (the
  // 64-bit integer conversions are ten times as dear); one fma rounds the sum
  // as the 64-bit conversion would
  auto as_double = [](int h) {
    return __hiloint2double(0x43300000, SIGNED ? h ^ (int)0x80000000 : h) - (SIGNED ? 0x1p52 + 0x1p31 : 0x1p52);
  };
  auto slow = [&](int a) -> float {
    if (split) return (float)(fma(as_double(planes[a]), (double)two_s, as_double(planes[PLANE + a])) * inv);
    return (float)((double)(long long)acc64[a] * inv);
  };
  auto pair = [&](unsigned h0, unsigned h1, unsigned l0, unsigned l1, float& a, float& b) {
    const F2 h = f2_add(f2_pack(__uint_as_float(kOff + h0), __uint_as_float(kOff + h1)), near2);
    const F2 l = f2_add(f2_pack(__uint_as_float(kOff + l0), __uint_as_float(kOff + l1)), near2);
    int ia, ib;
    f2_bits(f2_mul(f2_fma(h, two_s2, l), inv2), ia, ib);
    a = __int_as_float(ia);
    b = __int_as_float(ib);
  };
  auto finish = [&](float x) -> float { return mode == 1 ? __fmul_rn(__fsub_rn(x, 1.0f), src_mul) : x; };
  const int64_t ystride = nz, xstride = (int64_t)m.ny * nz, cstride = (int64_t)m.nx * xstride;
  float* const out0 = out + (int64_t)x0 * xstride + (int64_t)y0 * ystride;
  // output row of accumulator row c * RX * RY + lx * RY + ly (null: not in the mesh)
  auto row_out = [&](int row) -> float* {
    const int c = row / (RX * RY), lx = row / RY % RX, ly = row % RY;
    if (lx >= rxe || ly >= rye) return nullptr;
    return out0 + c * cstride + lx * xstride + ly * ystride;
  };
  if (nz % 4 == 0 && ((uintptr_t)out & 15) == 0) {
#pragma unroll 2
    for (int g = tid; g < GROUPS; g += T) {
      const int row = g / (NZP / 4), z4 = g % (NZP / 4);
      float* o = row_out(row);
      if ((!EXACT && z4 >= nz4) || o == nullptr) continue;
      float res[4];
      bool done = false;
      if (fconv) {
        const uint4 hi = reinterpret_cast<const uint4*>(acc)[g], lo = reinterpret_cast<const uint4*>(acc)[GROUPS + g];
        constexpr unsigned kTwo23 = 0x4B000000u;
        const unsigned top = ((kOff + hi.x) ^ kTwo23) | ((kOff + hi.y) ^ kTwo23) | ((kOff + hi.z) ^ kTwo23) |
                             ((kOff + hi.w) ^ kTwo23) | ((kOff + lo.x) ^ kTwo23) | ((kOff + lo.y) ^ kTwo23) |
                             ((kOff + lo.z) ^ kTwo23) | ((kOff + lo.w) ^ kTwo23);
        if (top < 0x800000u) {
          pair(hi.x, hi.y, lo.x, lo.y, res[0], res[1]);
          pair(hi.z, hi.w, lo.z, lo.w, res[2], res[3]);
          done = true;
        }
      }
      if (!done) {
#pragma unroll
        for (int q = 0; q < 4; ++q) res[q] = slow(4 * g + q);
      }
      *reinterpret_cast<float4*>(o + 4 * z4) =
          make_float4(finish(res[0]), finish(res[1]), finish(res[2]), finish(res[3]));
    }
  } else {
    for (int a = tid; a < PLANE; a += T) {
      const int row = a / NZP, z = a % NZP;
      float* o = row_out(row);
      if (z >= nz || o == nullptr) continue;
      o[z] = finish(slow(a));
    }
  }
}

int fixed_point_exponent(int64_t n) {
  int e = 0;
  const double p = fixed_point_pow2(n);
  while (ldexp(1.0, e) < p) ++e;
  return e;
}

// Output rows of one block at row stride nzp: as many as keep the accumulator
// within 33 KB (six or seven resident blocks).  More rows read each record
// fewer times (9 / 4 visits per particle at 2 x 2 rows, 25 / 16 at 4 x 4) but
// leave fewer blocks: one channel, us at 25 / 33 / 49 / 66 KB: 64^3 particles
// on 128^3 cells 8.7 / 8.7 / 8.7 / 8.8, 256^3 on 512^3 333 / 281 / 280 / 298,
// 512^3 on 1024^3 2209 / 2190 / 2189 / 2259; three channels on 512^3 822 / 822
// / 1072 / 1071, five deposits on 256^3 553 / 554 / 667 / 667.
constexpr int kTileBytes = 33 * 1024;
constexpr int tile_x(int C, int nzp) {
  const int row = 8 * C * nzp;
  return 16 * row <= kTileBytes ? 4 : 4 * row <= kTileBytes ? 2 : 1;
}
constexpr int tile_y(int C, int nzp) {
  const int rows = 8 * C * nzp * tile_x(C, nzp);
  return 4 * rows <= kTileBytes ? 4 : 2 * rows <= kTileBytes ? 2 : 1;
}

// Crowded meshes take one output row per block (ROW) instead of a tile, although
// a record is then read four times instead of 25 / 16 or 9 / 4:
//  * where the tiles are too few to share the work out evenly;
//  * where a tile would hold too many particles for the two-plane sums and a row
//    does not (at the mean density and four standard deviations);
//  * where neither fits, with three or four channels and tiles of more than four
//    rows.
// Deposits in us, tile / row (constant value | one, two, three, four channels of
// values): 16^3 cells with 32 particles each 131 / 20 | 145 / 29, 227 / 37, 304 / 45,
// 383 / 52; 64^3 with 4: 50 / 20 | 61 / 32, 95 / 39, 126 / 48, 160 / 60; 96^3 with 32,
// where neither fits: 867 / 963 | 787 / 1002, 1389 / 1668, 2486 / 2296, 3339 / 3067;
// 128^3 with 4, where the tile of a constant fits: 89 / 98 | 300 / 132, 550 / 188, 702 /
// 249, 845 / 350; 32 x 32 x 256 with 8, whose tiles of three and four channels
// are enough: 224 / 71 | 262 / 77, 226 / 180, 192 / 249, 250 / 320.
constexpr int kRowMaxNz = 512;  // longer rows have tiles of at most four

static bool planes_fit(double particles, int E, bool sgn) {
  const double k = particles + 4.0 * sqrt(particles);
  int L = 0;  // k < 2^L, as in the kernel
  while (ldexp(1.0, L) <= k) ++L;
  const int lo = E - 24 > L + E - (sgn ? 31 : 32) ? E - 24 : L + E - (sgn ? 31 : 32);
  return lo <= (32 - L < (sgn ? 23 : 24) ? 32 - L : (sgn ? 23 : 24));
}

static bool row_per_block(Mesh3 m, int C, bool sgn, int64_t n, int E) {
  if (m.nz > kRowMaxNz) return false;
  static const int strides[6] = {64, 128, 192, 256, 384, 512};
  int q = 0;
  while (strides[q] < m.nz) ++q;
  const int tx = tile_x(C, strides[q]), ty = tile_y(C, strides[q]);
  const double tiles = (double)((m.nx + tx - 1) / tx) * (double)((m.ny + ty - 1) / ty);
  if (tiles < (tx * ty > 4 ? 3 * 148 : 148) && (double)n > 5.0 * tiles * tiles) return true;
  if (n <= m.cells()) return false;
  const double line = (double)n / (double)m.cells() * (double)m.nz;  // particles in a row of the mesh
  if (planes_fit(2 * (ty + 1) * line, E, sgn)) return false;
  return planes_fit(4 * line, E, sgn) || (C >= 3 && tx * ty > 4);
}

template <int C, int NZP, bool EXACT, bool SIGNED, bool ROW = false>
static int launch_rows(const Rec* rec, const uint32_t* perm, const uint32_t* offs, Mesh3 m, const float* val,
                       int val_sorted, float val_const, const double* scale_dev, double scale_const, int E, int mode,
                       float src_mul, float* out, uint32_t* status, cudaStream_t s, int64_t n) {
  constexpr int RX = ROW ? 1 : tile_x(C, NZP), RY = ROW ? 1 : tile_y(C, NZP);
  auto k = scatter_rows_kernel<C, RX, RY, NZP, EXACT, SIGNED>;
  constexpr int smem = 8 * RX * RY * C * NZP;
  PMB_CUDA_CHECK(smem_optin((const void*)k, smem));
  const int dup = (m.nx == 1 ? 2 : 1) * (m.ny == 1 ? 2 : 1) * (m.nz == 1 ? 2 : 1);
  const int64_t nbx = (m.nx + RX - 1) / RX, nby = (m.ny + RY - 1) / RY;
  // Few blocks of long work, started early, crowd onto the SMs that the sort's
  // last blocks leave first: sort, deposit and gather of 2^18 particles on 16^3 cells
  // 93 us early, 62 plain, of 2^20 215 / 171, of 2^22 on 32^3 399 / 373; with less
  // work a block early is the faster one (2^17 on 16^3 50 / 52, 2^19 on 32^3 56 / 70).
  const bool early = small_mesh(m.nx, m.ny, m.nz) && !(ROW && nbx * nby < 8 * 148 && n >= 1024 * nbx * nby);
  PMB_CUDA_CHECK(launch_dependent(early, k, (int)(nbx * nby), kRowThreads, smem, s, rec, perm, offs, m,
                                  fast_div((uint32_t)m.nz), fast_div((uint32_t)nby), val, val_sorted, val_const,
                                  scale_dev, scale_const, E, dup, mode, src_mul, out, status));
  return kOk;
}

// A kernel for the row length itself (usual lengths; one channel of a constant
// value and three channels, the deposits of a force and its adjoint), else the
// one of the shortest row stride that holds nz cells.  row: one row per block.
template <int C, bool SIGNED, class... Args>
static int launch_rows_nz(bool row, Args... a) {
  const int nz = std::get<3>(std::tie(a...)).nz;
  if (row) {
    if (nz <= 64) return launch_rows<C, 64, false, SIGNED, true>(a...);
    if (nz <= 128) return launch_rows<C, 128, false, SIGNED, true>(a...);
    if (nz <= 256) return launch_rows<C, 256, false, SIGNED, true>(a...);
    return launch_rows<C, kRowMaxNz, false, SIGNED, true>(a...);
  }
  if constexpr (C == 3 || (C == 1 && !SIGNED)) {
    switch (nz) {
      case 128: return launch_rows<C, 128, true, SIGNED>(a...);
      case 192: return launch_rows<C, 192, true, SIGNED>(a...);
      case 256: return launch_rows<C, 256, true, SIGNED>(a...);
      case 384: return launch_rows<C, 384, true, SIGNED>(a...);
      case 512: return launch_rows<C, 512, true, SIGNED>(a...);
      case 768: return launch_rows<C, 768, true, SIGNED>(a...);
      case 1024: return launch_rows<C, 1024, true, SIGNED>(a...);
      default: break;
    }
  }
#define PMB_ROWS(N) \
  if (nz <= N) return launch_rows<C, N, false, SIGNED>(a...)
  PMB_ROWS(64);
  PMB_ROWS(128);
  PMB_ROWS(192);
  PMB_ROWS(256);
  PMB_ROWS(384);
  PMB_ROWS(512);
  PMB_ROWS(768);
  PMB_ROWS(1024);
  PMB_ROWS(2048);
  PMB_ROWS(4096);
#undef PMB_ROWS
  return kUnsupported;
}

// scale_dev null: the scale of the constant value val_const.
int scatter_sorted(const Rec* rec, const uint32_t* perm, const uint32_t* offs, Mesh3 m, int C, const float* val,
                   int val_sorted, float val_const, const double* scale_dev, int mode, float src_mul, float* out,
                   cudaStream_t s, int64_t n, uint32_t* status) {
  const int E = fixed_point_exponent(n);
  const double scale = fixed_point_scale(fixed_point_pow2(n), fabsf(val_const));
  const bool uns = val == nullptr && val_const >= 0.f;
#define PMB_SCATTER(CC, SG)                                                                                       \
  launch_rows_nz<CC, SG>(row_per_block(m, CC, SG, n, E), rec, perm, offs, m, val, val_sorted, val_const, scale_dev, \
                         scale, E, mode, src_mul, out, status, s, n)
  switch (C) {
    case 1: return uns ? PMB_SCATTER(1, false) : PMB_SCATTER(1, true);
    case 2: return PMB_SCATTER(2, true);
    case 3: return PMB_SCATTER(3, true);
    case 4: return PMB_SCATTER(4, true);
    default: return kUnsupported;
  }
#undef PMB_SCATTER
}

// ---------------------------------------------------------------------------
// Gather and adjoint position terms
// ---------------------------------------------------------------------------
// out[src, c] = sum_b mesh_c[i_b] w_b (gather.py:452-472, pallas.py:305-318).
// With vel the half-kick vel += out * kick is applied in place (integrator.py:536),
// and with kick2 != 0 the next step's opening half-kick after it, saving passes
// over the particles.
template <int C>
__global__ void gather_kernel(const Rec* __restrict__ rec, const uint32_t* __restrict__ perm, int64_t n, Mesh3 m,
                              const float* __restrict__ mesh, float* __restrict__ out, float* __restrict__ vel,
                              float kick, float kick2, const uint32_t* __restrict__ status) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || flagged(status)) return;
  gather_one<C>(rec[i], perm[i], m, mesh, out, vel, kick, kick2);
}

// ---------------------------------------------------------------------------
// Staged gathers: the mesh rows a tile of particle rows touches are copied
// into shared memory with bulk asynchronous copies, then every particle of
// the tile interpolates from shared memory.
// ---------------------------------------------------------------------------
__device__ unsigned int g_wait_timeouts_cic = 0;

// 0: direct corner loads (default); 1: stage the rows of tiles with enough
// particles; 2: stage every non-empty tile.  Staging wins on spread-out
// particles and loses on clustered ones, whose corner loads already hit in
// L1/L2, so it is opt-in.
static int g_gather_staging = 0;

void set_gather_staging(int mode) { g_gather_staging = mode; }

// Poll limit of the first bounded wait of every staged or TMA-fed kernel
// (process-wide, pmb_set_wait_limit).
static uint32_t g_wait_polls = kWaitPolls;

void set_wait_polls(uint32_t polls) { g_wait_polls = polls; }
uint32_t wait_polls() { return g_wait_polls; }

constexpr int kStageMaxRX = 4;
constexpr int64_t kStageBudget = 110 * 1024;

// Shared bytes of the staged rows of an RX x RY tile with C channels.
inline int64_t stage_bytes(int RX, int RY, int C, int nz) { return (int64_t)(RX + 1) * (RY + 1) * C * nz * 4; }

// Tile of particle rows whose staged mesh rows fit the budget; false when the
// mesh rows cannot be bulk-copied (nz % 4 != 0 or a misaligned mesh).
bool stage_shape(Mesh3 m, int C, const float* mesh, int* RX, int* RY) {
  if (g_gather_staging == 0 || m.nz % 4 != 0 || ((uintptr_t)mesh & 15) != 0) return false;
  static const int shapes[5][2] = {{4, 4}, {2, 4}, {2, 2}, {1, 2}, {1, 1}};
  for (const auto& sh : shapes) {
    if (sh[0] <= m.nx && sh[1] <= m.ny && stage_bytes(sh[0], sh[1], C, m.nz) <= kStageBudget) {
      *RX = sh[0];
      *RY = sh[1];
      return true;
    }
  }
  return false;
}

// Tiles with fewer particles than this load their corners directly: staging
// costs the tile's rows, a direct gather about one 32-byte sector per corner
// and channel of every particle.
inline uint32_t stage_threshold(int64_t smem, int C) {
  return g_gather_staging == 2 ? 1u : (uint32_t)(smem / (8 * 32 * C));
}

// Copies the (RX+1) x (RY+1) mesh rows (periodic) of C channels starting at
// row (x0, y0) into stage[c][ix][iy][nz].  Returns false (after flagging the
// timeout) when the copies do not complete.
__device__ __forceinline__ bool stage_mesh_rows(float* stage, const float* __restrict__ mesh, Mesh3 m, int C, int x0,
                                                int y0, int RX, int RY, uint64_t* bar, uint32_t polls) {
  const int SX = RX + 1, SY = RY + 1;
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    const uint32_t row_bytes = (uint32_t)m.nz * 4u;
    mbar_expect_tx(bar, row_bytes * (uint32_t)(SX * SY * C));
    const int64_t cells = m.cells();
    for (int c = 0; c < C; ++c)
      for (int ix = 0; ix < SX; ++ix) {
        const int x = x0 + ix >= m.nx ? x0 + ix - m.nx : x0 + ix;
        for (int iy = 0; iy < SY; ++iy) {
          const int y = y0 + iy >= m.ny ? y0 + iy - m.ny : y0 + iy;
          bulk_copy_g2s(stage + ((c * SX + ix) * SY + iy) * m.nz, mesh + c * cells + ((int64_t)x * m.ny + y) * m.nz,
                        row_bytes, bar);
        }
      }
  }
  __syncthreads();
  return mbar_wait_or_flag(bar, 0, &g_wait_timeouts_cic, polls);
}

// Particle segments of the tile: rows (x0 + k, y0 .. y0+RY-1) are contiguous
// in the sorted records for each k.  Returns the particle count.
__device__ __forceinline__ uint32_t tile_segments(const uint32_t* __restrict__ offs, Mesh3 m, int x0, int y0, int RX,
                                                  int RY, uint32_t* seg_b, uint32_t* seg_n) {
  if (threadIdx.x < RX) {
    const int x = x0 + threadIdx.x;
    uint32_t b = 0, c = 0;
    if (x < m.nx) {
      const int y1 = y0 + RY < m.ny ? y0 + RY : m.ny;
      b = offs[(int64_t)x * m.ny + y0];
      c = offs[(int64_t)x * m.ny + y1] - b;
    }
    seg_b[threadIdx.x] = b;
    seg_n[threadIdx.x] = c;
  }
  __syncthreads();
  uint32_t total = 0;
  for (int k = 0; k < RX; ++k) total += seg_n[k];
  return total;
}

// Sorted index and tile-local row (k, iy) of the j-th particle of the tile.
__device__ __forceinline__ uint32_t tile_particle(uint32_t j, const uint32_t* seg_b, const uint32_t* seg_n, int* k) {
  int kk = 0;
  while (j >= seg_n[kk]) {
    j -= seg_n[kk];
    ++kk;
  }
  *k = kk;
  return seg_b[kk] + j;
}

// Same arithmetic as gather_one, reading the staged rows.
template <int C>
__global__ void __launch_bounds__(256) gather_staged_kernel(const Rec* __restrict__ rec, const uint32_t* __restrict__ perm,
                                                            const uint32_t* __restrict__ offs, Mesh3 m, int RX, int RY,
                                                            uint32_t min_stage, const float* __restrict__ mesh,
                                                            float* __restrict__ out, float* __restrict__ vel,
                                                            float kick, float kick2, uint32_t polls,
                                                            const uint32_t* __restrict__ status) {
  extern __shared__ __align__(16) float stage[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t seg_b[kStageMaxRX], seg_n[kStageMaxRX];
  if (flagged(status)) return;
  const int nby = (m.ny + RY - 1) / RY;
  const int x0 = (int)(blockIdx.x / nby) * RX, y0 = (int)(blockIdx.x % nby) * RY;
  const uint32_t total = tile_segments(offs, m, x0, y0, RX, RY, seg_b, seg_n);
  if (total == 0) return;
  if (total < min_stage) {
    // too few particles to pay for staging the rows: load corners directly
    for (uint32_t j = threadIdx.x; j < total; j += blockDim.x) {
      int k;
      const uint32_t i = tile_particle(j, seg_b, seg_n, &k);
      gather_one<C>(rec[i], perm[i], m, mesh, out, vel, kick, kick2);
    }
    return;
  }
  if (!stage_mesh_rows(stage, mesh, m, C, x0, y0, RX, RY, &bar, polls)) return;
  const int SX = RX + 1, SY = RY + 1, nz = m.nz;
  for (uint32_t j = threadIdx.x; j < total; j += blockDim.x) {
    int k;
    const uint32_t i = tile_particle(j, seg_b, seg_n, &k);
    const Rec r = rec[i];
    const uint32_t row = r.key / (uint32_t)nz;
    const int cz = (int)(r.key - row * (uint32_t)nz);
    const int iy = (int)(row - (uint32_t)(x0 + k) * (uint32_t)m.ny) - y0;
    const int z1 = cz + 1 == nz ? 0 : cz + 1;
    const float wx[2] = {axis_weight(r.fx, 0), axis_weight(r.fx, 1)};
    const float wy[2] = {axis_weight(r.fy, 0), axis_weight(r.fy, 1)};
    const float wz[2] = {axis_weight(r.fz, 0), axis_weight(r.fz, 1)};
    const uint32_t src = perm[i];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      float a = 0.f;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const int bx = b & 1, by = (b >> 1) & 1, bz = (b >> 2) & 1;
        const float v = stage[((c * SX + k + bx) * SY + iy + by) * nz + (bz ? z1 : cz)];
        a = __fadd_rn(a, __fmul_rn(v, __fmul_rn(__fmul_rn(wx[bx], wy[by]), wz[bz])));
      }
      if (out != nullptr) out[(int64_t)src * C + c] = a;
      if (vel != nullptr) vel[(int64_t)src * C + c] = kicked(vel[(int64_t)src * C + c], a, kick, kick2);
    }
  }
}

// Direct gather with two particles per thread: both particles' 8C corner
// loads are issued before either sum, doubling the loads in flight of this
// latency-bound kernel (10% faster on clustered particles at 512^3, same
// arithmetic per particle as gather_one).  The results go through shared
// memory, so that consecutive threads store consecutive components: the
// stores follow the particles' own order, and a store per component from the
// thread that computed it sends C partial sectors per particle to L2, which
// this kernel keeps busiest: 522 -> 433 us (256^3 clustered particles on 512^3), 4.85
// -> 4.11 ms (512^3 on 1024^3), 1.28 -> 0.90 ms (256^3 uniform).  A warp's
// results through its own part, without the block's barrier, measured 452 us
// and 4.46 ms.
constexpr int kGatherThreads = 256;
constexpr int kGatherTile = 2 * kGatherThreads;
constexpr int kGatherWarps = kGatherThreads / 32;

// An ordinary (coherent) load that the compiler may schedule among the kernel's
// stores as freely as a read-only one: for data that this kernel does not write,
// at addresses formed from what it read after wait_for_previous.  (By plain
// expressions the gather's 48 loads keep their order around its other accesses: 435 ->
// 479 us for 256^3 clustered particles on 512^3.)
__device__ __forceinline__ float load_global(const float* p) {
  float v;
  asm("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}

template <int C>
__global__ void __launch_bounds__(kGatherThreads)
    gather_kernel_x2(const Rec* rec, const uint32_t* perm, int64_t n, Mesh3 m,
                     const float* mesh, float* __restrict__ out, float* __restrict__ vel, float kick,
                     float kick2, const uint32_t* status) {
  __shared__ float s_val[kGatherTile * C];
  __shared__ uint32_t s_dst[kGatherTile];
  __shared__ bool s_masked[kGatherTile];
  wait_for_previous();
  let_next_start();
  if (flagged(status)) return;
  const int64_t base = (int64_t)blockIdx.x * kGatherTile;
  const int cnt = n - base < kGatherTile ? (int)(n - base) : kGatherTile;
  const int t0 = threadIdx.x, t1 = t0 + kGatherThreads;
  const int64_t cells = m.cells();
  if (t0 < cnt) {
    const int64_t i0 = base + t0, i1 = t1 < cnt ? base + t1 : i0;
    // masked particles (trailing records) interpolate from cell 0 and give zero
    bool mk0, mk1;
    const Rec r0 = unmasked_or_origin(rec[i0], &mk0);
    const Rec r1 = unmasked_or_origin(rec[i1], &mk1);
    Corners k0, k1;
    corners_of(r0, m, k0);
    corners_of(r1, m, k1);
    s_dst[t0] = perm[i0];
    s_dst[t1] = perm[i1];
    s_masked[t0] = mk0;
    s_masked[t1] = mk1;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const float* mc = mesh + (int64_t)c * cells;
      float v0[8], v1[8];
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        v0[b] = load_global(mc + k0.idx[b]);
        v1[b] = load_global(mc + k1.idx[b]);
      }
      float a0 = 0.f, a1 = 0.f;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        a0 = __fadd_rn(a0, __fmul_rn(v0[b], k0.w[b]));
        a1 = __fadd_rn(a1, __fmul_rn(v1[b], k1.w[b]));
      }
      s_val[t0 * C + c] = mk0 ? 0.f : a0;
      s_val[t1 * C + c] = mk1 ? 0.f : a1;
    }
  }
  __syncthreads();
  int64_t at[2 * C];
  float u[2 * C];
#pragma unroll
  for (int q = 0; q < 2 * C; ++q) {
    const int j = t0 + q * kGatherThreads, p = j / C;
    if (p < cnt) {
      at[q] = (int64_t)s_dst[p] * C + (j - p * C);
      if (vel != nullptr) u[q] = vel[at[q]];
    }
  }
#pragma unroll
  for (int q = 0; q < 2 * C; ++q) {
    const int j = t0 + q * kGatherThreads, p = j / C;
    if (p < cnt) {
      const float a = s_val[j];
      if (out != nullptr) out[at[q]] = a;
      if (vel != nullptr && !s_masked[p]) vel[at[q]] = kicked(u[q], a, kick, kick2);
    }
  }
}

// Records after the last row (masked particles) in the staged kernels, which
// only visit rows: zero gathered values; for the adjoint position terms zero
// (or keep, when accumulating) the cotangent, zero wsum and copy u to
// u_sorted.
__global__ void masked_tail_gather_kernel(const uint32_t* __restrict__ perm, const uint32_t* __restrict__ offs_end,
                                          int64_t n, int C, float* __restrict__ out,
                                          const uint32_t* __restrict__ status) {
  if (flagged(status)) return;
  for (int64_t i = (int64_t)*offs_end + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    for (int c = 0; c < C; ++c)
      if (out != nullptr) out[(int64_t)perm[i] * C + c] = 0.f;
}

__global__ void masked_tail_interp_kernel(const uint32_t* __restrict__ perm, const uint32_t* __restrict__ offs_end,
                                          int64_t n, int C, const float* __restrict__ u, float u_const,
                                          int accumulate, float* __restrict__ disp_cot, float* __restrict__ wsum,
                                          float* __restrict__ u_sorted, const uint32_t* __restrict__ status) {
  if (flagged(status)) return;
  for (int64_t i = (int64_t)*offs_end + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t src = perm[i];
    if (!accumulate) disp_cot[3 * src] = disp_cot[3 * src + 1] = disp_cot[3 * src + 2] = 0.f;
    for (int c = 0; c < C; ++c) {
      if (wsum != nullptr) wsum[src * C + c] = 0.f;
      if (u_sorted != nullptr) u_sorted[i * C + c] = u ? u[src * C + c] : u_const;
    }
  }
}

int gather_sorted(const Rec* rec, const uint32_t* perm, const uint32_t* offs, int64_t n, Mesh3 m, int C,
                  const float* mesh, float* out, float* vel, float kick, float kick2, cudaStream_t s,
                  const uint32_t* status) {
  if (n == 0) return kOk;
  int RX, RY;
  if (offs != nullptr && stage_shape(m, C, mesh, &RX, &RY)) {
    const int64_t smem = stage_bytes(RX, RY, C, m.nz);
    const uint32_t min_stage = stage_threshold(smem, C);
    const unsigned grid = (unsigned)((int64_t)((m.nx + RX - 1) / RX) * ((m.ny + RY - 1) / RY));
#define PMB_LAUNCH_GS(CC)                                                                                      \
  do {                                                                                                         \
    PMB_CUDA_CHECK(smem_optin((const void*)gather_staged_kernel<CC>, (int)kStageBudget));                     \
    gather_staged_kernel<CC><<<grid, 256, (size_t)smem, s>>>(rec, perm, offs, m, RX, RY, min_stage, mesh, out, vel, \
                                                              kick, kick2, g_wait_polls, status);               \
  } while (0)
    switch (C) {
      case 1: PMB_LAUNCH_GS(1); break;
      case 2: PMB_LAUNCH_GS(2); break;
      case 3: PMB_LAUNCH_GS(3); break;
      case 4: PMB_LAUNCH_GS(4); break;
      default: return kUnsupported;
    }
#undef PMB_LAUNCH_GS
    masked_tail_gather_kernel<<<148, 256, 0, s>>>(perm, offs + m.rows(), n, C, out, status);
    PMB_CUDA_CHECK(cudaGetLastError());
    return kOk;
  }
  const int th = 256;
  const unsigned g = (unsigned)((n + th - 1) / th);
  if (C == 3) {
    PMB_CUDA_CHECK(launch_dependent(small_mesh(m.nx, m.ny, m.nz), gather_kernel_x2<3>,
                                    (int)((n + kGatherTile - 1) / kGatherTile), kGatherThreads, 0, s, rec, perm, n, m, mesh, out, vel, kick, kick2, status));
    return kOk;
  }
  switch (C) {
    case 1: gather_kernel<1><<<g, th, 0, s>>>(rec, perm, n, m, mesh, out, vel, kick, kick2, status); break;
    case 2: gather_kernel<2><<<g, th, 0, s>>>(rec, perm, n, m, mesh, out, vel, kick, kick2, status); break;
    case 4: gather_kernel<4><<<g, th, 0, s>>>(rec, perm, n, m, mesh, out, vel, kick, kick2, status); break;
    default: return kUnsupported;
  }
  PMB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

// Reads and clears the device-wide flags (the staged gathers' wait counter
// becomes kFlagWaitTimeout).  Synchronous.
int device_flags_take(unsigned int* flags) {
  unsigned int f = 0, w = 0;
  PMB_CUDA_CHECK(cudaMemcpyFromSymbol(&f, g_device_flags, sizeof(unsigned int)));
  PMB_CUDA_CHECK(cudaMemcpyFromSymbol(&w, g_wait_timeouts_cic, sizeof(unsigned int)));
  const unsigned int zero = 0;
  PMB_CUDA_CHECK(cudaMemcpyToSymbol(g_device_flags, &zero, sizeof(unsigned int)));
  PMB_CUDA_CHECK(cudaMemcpyToSymbol(g_wait_timeouts_cic, &zero, sizeof(unsigned int)));
  *flags = f | (w ? (unsigned)kFlagWaitTimeout : 0u);
  return kOk;
}

int wait_timeouts(unsigned int* count) {
  PMB_CUDA_CHECK(cudaMemcpyFromSymbol(count, g_wait_timeouts_cic, sizeof(unsigned int)));
  return kOk;
}

// Position term of the CIC adjoints.  With per-particle weights u (N, C) or a
// constant u_const:
//   inner_b = sum_c u_c * mesh_c[i_b]
//   disp_cot[src] (+)= (sum_b inner_b * grad w_b) / cell
// This is gather.py:495-502 (u = val_cot) and scatter.py:366-370 (u = val).
// Optionally also emits wsum[src, c] = sum_b mesh_c[i_b] w_b (the scatter
// adjoint's val cotangent, scatter.py:372-373) and u_sorted[i, c] =
// u[src, c] (the weights in sorted order, so a following scatter of u reads
// them coalesced instead of through the permutation).
// Raveled index of a record's corner b in 32-bit arithmetic modulo 2^32 (a mesh
// has fewer cells than that): the lower cell and its steps to the upper one.
struct Steps {
  uint32_t key, dx, dy, dz;
  __device__ __forceinline__ uint32_t at(int b) const {
    return key + ((b & 1) ? dx : 0u) + ((b & 2) ? dy : 0u) + ((b & 4) ? dz : 0u);
  }
};

__device__ __forceinline__ Steps steps_of(uint32_t key, Mesh3 m) {
  const uint32_t nz = (uint32_t)m.nz, ny = (uint32_t)m.ny, plane = ny * nz;
  uint32_t cx, cy, cz;
  if (((nz & (nz - 1)) | (ny & (ny - 1))) == 0) {  // shifts instead of divisions
    const int lz = __ffs(nz) - 1, ly = __ffs(ny) - 1;
    cz = key & (nz - 1);
    cy = (key >> lz) & (ny - 1);
    cx = key >> (lz + ly);
  } else {
    const uint32_t row = key / nz;
    cz = key - row * nz;
    cx = row / ny;
    cy = row - cx * ny;
  }
  Steps k;
  k.key = key;
  k.dx = cx + 1 == (uint32_t)m.nx ? 0u - cx * plane : plane;
  k.dy = cy + 1 == ny ? 0u - cy * nz : nz;
  k.dz = cz + 1 == nz ? 0u - cz : 1u;
  return k;
}

// sum_b v_b w_b in the order of gather_one.
__device__ __forceinline__ float corner_sum(const Rec& r, const float (&v)[8]) {
  float a = 0.f;
#pragma unroll
  for (int b = 0; b < 8; ++b)
    a = __fadd_rn(a, __fmul_rn(v[b], __fmul_rn(__fmul_rn(axis_weight(r.fx, b & 1), axis_weight(r.fy, (b >> 1) & 1)),
                                               axis_weight(r.fz, (b >> 2) & 1))));
  return a;
}

// (sum_b inner_b * grad w_b) / cell of one particle, inner_b the weighted sum
// of the channels at corner b (bit a of b: +1 along axis a).
__device__ __forceinline__ void position_term(const Rec& r, const float (&inner)[8], float cell, float (&g)[3]) {
  const float f[3] = {r.fx, r.fy, r.fz};
  float wa[3][2], sg[3][2];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    wa[a][0] = axis_weight(f[a], 0);
    wa[a][1] = axis_weight(f[a], 1);
    sg[a][0] = axis_sign(f[a], 0);
    sg[a][1] = axis_sign(f[a], 1);
  }
  g[0] = g[1] = g[2] = 0.f;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const int bx = b & 1, by = (b >> 1) & 1, bz = (b >> 2) & 1;
    // grad_i = sign_i * w_{i+1} * w_{i+2} (enmesh.py:155-160)
    const float gx = __fmul_rn(__fmul_rn(sg[0][bx], wa[1][by]), wa[2][bz]);
    const float gy = __fmul_rn(__fmul_rn(sg[1][by], wa[2][bz]), wa[0][bx]);
    const float gz = __fmul_rn(__fmul_rn(sg[2][bz], wa[0][bx]), wa[1][by]);
    g[0] = __fadd_rn(g[0], __fmul_rn(inner[b], gx));
    g[1] = __fadd_rn(g[1], __fmul_rn(inner[b], gy));
    g[2] = __fadd_rn(g[2], __fmul_rn(inner[b], gz));
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) g[a] = __fdiv_rn(g[a], cell);
}

// Sums of one particle: g the position term, ws the interpolated values;
// fetch(c, b) returns channel c of corner b.
template <int C, class Fetch>
__device__ __forceinline__ void interp_grad_sums(const Rec& r, const Fetch& fetch, const float (&uu)[C], float cell,
                                                 float (&g)[3], float (&ws)[C]) {
  float inner[8];
#pragma unroll
  for (int c = 0; c < C; ++c) ws[c] = 0.f;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const float w = __fmul_rn(__fmul_rn(axis_weight(r.fx, b & 1), axis_weight(r.fy, (b >> 1) & 1)),
                              axis_weight(r.fz, (b >> 2) & 1));
    inner[b] = 0.f;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const float mv = fetch(c, b);
      inner[b] = __fadd_rn(inner[b], __fmul_rn(uu[c], mv));
      ws[c] = __fadd_rn(ws[c], __fmul_rn(mv, w));
    }
  }
  position_term(r, inner, cell, g);
}

// One particle's loads, sums and stores in the kernels that handle one at a time.
template <int C, class Fetch>
__device__ __forceinline__ void interp_grad_one(const Rec& r, uint32_t src, int64_t i, const Fetch& fetch,
                                                const float* __restrict__ u, float u_const, float cell, int accumulate,
                                                float* __restrict__ disp_cot, float* __restrict__ wsum,
                                                float* __restrict__ u_sorted, bool masked = false) {
  float uu[C], g[3], ws[C];
#pragma unroll
  for (int c = 0; c < C; ++c) uu[c] = u ? u[(int64_t)src * C + c] : u_const;
  if (u_sorted != nullptr) {
#pragma unroll
    for (int c = 0; c < C; ++c) u_sorted[i * C + c] = uu[c];
  }
  interp_grad_sums<C>(r, fetch, uu, cell, g, ws);
  float* dc = disp_cot + 3 * (int64_t)src;
  // a masked particle takes no adjoint: zero, or unchanged when accumulating
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (!accumulate)
      dc[a] = masked ? 0.f : g[a];
    else if (!masked)
      dc[a] = __fadd_rn(dc[a], g[a]);
  }
  if (wsum != nullptr) {
#pragma unroll
    for (int c = 0; c < C; ++c) wsum[(int64_t)src * C + c] = masked ? 0.f : ws[c];
  }
}

template <int C>
__global__ void interp_grad_kernel(const Rec* __restrict__ rec, const uint32_t* __restrict__ perm, int64_t n, Mesh3 m,
                                   const float* __restrict__ mesh, const float* __restrict__ u, float u_const,
                                   float cell, int accumulate, float* __restrict__ disp_cot,
                                   float* __restrict__ wsum, float* __restrict__ u_sorted,
                                   const uint32_t* __restrict__ status) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || flagged(status)) return;
  bool mk;
  const Rec r = unmasked_or_origin(rec[i], &mk);
  Corners k;
  corners_of(r, m, k);
  const int64_t cells = m.cells();
  auto fetch = [&](int c, int b) { return __ldg(mesh + (int64_t)c * cells + k.idx[b]); };
  interp_grad_one<C>(r, perm[i], i, fetch, u, u_const, cell, accumulate, disp_cot, wsum, u_sorted, mk);
}

// Two particles per thread, each result stored by the thread that computed it:
// three channels without accumulation, where there is nothing to read back and the
// staging below costs more than the partial sectors of the stores.  us, staged /
// direct: 256^3 particles in cell order on 256^3 cells 457 / 309, on 512^3 577 / 446, a
// smooth state there 547 / 424, a clustered one 570 / 569, independent positions 1345 /
// 1280.
template <int C>
__global__ void __launch_bounds__(kGatherThreads, 4)
    interp_grad_direct_kernel(const Rec* __restrict__ rec, const uint32_t* __restrict__ perm, int64_t n, Mesh3 m,
                              const float* __restrict__ mesh, const float* __restrict__ u, float u_const, float cell,
                              float* __restrict__ disp_cot, float* __restrict__ wsum, float* __restrict__ u_sorted,
                              const uint32_t* __restrict__ status) {
  const int64_t i0 = (int64_t)blockIdx.x * kGatherTile + threadIdx.x;
  const int64_t i1 = i0 + kGatherThreads;
  if (i0 >= n || flagged(status)) return;
  const bool two = i1 < n;
  bool mk0, mk1;
  const Rec r0 = unmasked_or_origin(rec[i0], &mk0);
  const Rec r1 = unmasked_or_origin(rec[two ? i1 : i0], &mk1);
  Corners k0, k1;
  corners_of(r0, m, k0);
  corners_of(r1, m, k1);
  const uint32_t s0 = perm[i0], s1 = perm[two ? i1 : i0];
  const int64_t cells = m.cells();
  float v0[C][8], v1[C][8];
#pragma unroll
  for (int c = 0; c < C; ++c)
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      v0[c][b] = __ldg(mesh + (int64_t)c * cells + k0.idx[b]);
      v1[c][b] = __ldg(mesh + (int64_t)c * cells + k1.idx[b]);
    }
  interp_grad_one<C>(r0, s0, i0, [&](int c, int b) { return v0[c][b]; }, u, u_const, cell, 0, disp_cot, wsum,
                     u_sorted, mk0);
  if (two)
    interp_grad_one<C>(r1, s1, i1, [&](int c, int b) { return v1[c][b]; }, u, u_const, cell, 0, disp_cot, wsum,
                       u_sorted, mk1);
}

// Two particles per thread with the weights and the cotangents carried by
// component through the warp's shared memory, as gather_kernel_x2; the channels
// are summed one after another at each corner, so that one channel's corner
// values are held at a time.  256^3 clustered particles on 512^3: three
// channels 949 -> 721 us (80 registers, three blocks; 64 registers spill: 782),
// one channel 805 -> 449 us accumulating and 360 -> 266 us not (64 registers).
template <int C>
__global__ void __launch_bounds__(kGatherThreads, C == 1 ? 4 : 3)
    interp_grad_kernel_x2(const Rec* __restrict__ rec, const uint32_t* __restrict__ perm, int64_t n, Mesh3 m,
                          const float* __restrict__ mesh, const float* __restrict__ u, float u_const, float cell,
                          int accumulate, float* __restrict__ disp_cot, float* __restrict__ wsum,
                          float* __restrict__ u_sorted, const uint32_t* __restrict__ status) {
  __shared__ float s_val_all[kGatherWarps][64 * 3];  // weights (C of 3) in, cotangents out
  __shared__ uint32_t s_dst_all[kGatherWarps][64];
  __shared__ bool s_masked_all[kGatherWarps][64];
  if (flagged(status)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* const s_val = s_val_all[warp];
  uint32_t* const s_dst = s_dst_all[warp];
  bool* const s_masked = s_masked_all[warp];
  const int64_t base = (int64_t)blockIdx.x * kGatherTile + warp * 64;
  if (base >= n) return;
  const int cnt = n - base < 64 ? (int)(n - base) : 64;
  const int t0 = lane, t1 = lane + 32;
  if (t0 < cnt) s_dst[t0] = perm[base + t0];
  if (t1 < cnt) s_dst[t1] = perm[base + t1];
  __syncwarp();
  // Loads in the order in which their results are needed: the accumulated
  // cotangents (by the lanes that will store them) and the weights, which
  // follow the permutation, then the first channel's corners; the weights are
  // passed on once those are on their way.
  float before[6], wgt[2 * C];
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const int j = lane + q * 32, p = j / 3;
    before[q] = accumulate && p < cnt ? disp_cot[(int64_t)s_dst[p] * 3 + (j - 3 * p)] : 0.f;
  }
#pragma unroll
  for (int q = 0; q < 2 * C; ++q) {
    const int j = lane + q * 32, p = j / C;
    wgt[q] = u != nullptr && p < cnt ? u[(int64_t)s_dst[p] * C + (j - C * p)] : u_const;
  }
  const bool on = t0 < cnt;
  const int e0 = on ? t0 : 0, e1 = t1 < cnt ? t1 : e0;
  bool mk0, mk1;
  const Rec r0 = unmasked_or_origin(rec[base + e0], &mk0);
  const Rec r1 = unmasked_or_origin(rec[base + e1], &mk1);
  const Steps k0 = steps_of(r0.key, m), k1 = steps_of(r1.key, m);
  const int64_t cells = m.cells();
  float in0[8], in1[8];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const float* mc = mesh + (int64_t)c * cells;
    float v0[8], v1[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      v0[b] = __ldg(mc + k0.at(b));
      v1[b] = __ldg(mc + k1.at(b));
    }
    if (c == 0) {
#pragma unroll
      for (int q = 0; q < 2 * C; ++q) {
        const int j = lane + q * 32, p = j / C;
        if (p < cnt) {
          s_val[j] = wgt[q];
          if (u_sorted != nullptr) u_sorted[base * C + j] = wgt[q];
        }
      }
      __syncwarp();
    }
    const float u0 = s_val[e0 * C + c], u1 = s_val[e1 * C + c];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      in0[b] = __fadd_rn(c == 0 ? 0.f : in0[b], __fmul_rn(u0, v0[b]));
      in1[b] = __fadd_rn(c == 0 ? 0.f : in1[b], __fmul_rn(u1, v1[b]));
    }
    if (wsum != nullptr && on) {
      wsum[(int64_t)s_dst[t0] * C + c] = mk0 ? 0.f : corner_sum(r0, v0);
      if (t1 < cnt) wsum[(int64_t)s_dst[t1] * C + c] = mk1 ? 0.f : corner_sum(r1, v1);
    }
  }
  float g0[3], g1[3];
  position_term(r0, in0, cell, g0);
  position_term(r1, in1, cell, g1);
  __syncwarp();  // the weights are read
  if (on) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      s_val[t0 * 3 + a] = mk0 ? 0.f : g0[a];
      s_val[t1 * 3 + a] = mk1 ? 0.f : g1[a];
    }
    s_masked[t0] = mk0;
    s_masked[t1] = mk1;
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const int j = lane + q * 32, p = j / 3;
    // a masked particle takes no adjoint: zero, or unchanged when accumulating
    if (p < cnt && !(accumulate && s_masked[p]))
      disp_cot[(int64_t)s_dst[p] * 3 + (j - 3 * p)] = accumulate ? __fadd_rn(before[q], s_val[j]) : s_val[j];
  }
}

template <int C>
__global__ void __launch_bounds__(256) interp_grad_staged_kernel(
    const Rec* __restrict__ rec, const uint32_t* __restrict__ perm, const uint32_t* __restrict__ offs, Mesh3 m, int RX,
    int RY, uint32_t min_stage, const float* __restrict__ mesh, const float* __restrict__ u, float u_const, float cell,
    int accumulate, float* __restrict__ disp_cot, float* __restrict__ wsum, float* __restrict__ u_sorted,
    uint32_t polls, const uint32_t* __restrict__ status) {
  extern __shared__ __align__(16) float stage[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t seg_b[kStageMaxRX], seg_n[kStageMaxRX];
  if (flagged(status)) return;
  const int nby = (m.ny + RY - 1) / RY;
  const int x0 = (int)(blockIdx.x / nby) * RX, y0 = (int)(blockIdx.x % nby) * RY;
  const uint32_t total = tile_segments(offs, m, x0, y0, RX, RY, seg_b, seg_n);
  if (total == 0) return;
  if (total < min_stage) {
    const int64_t cells = m.cells();
    for (uint32_t j = threadIdx.x; j < total; j += blockDim.x) {
      int k;
      const uint32_t i = tile_particle(j, seg_b, seg_n, &k);
      const Rec r = rec[i];
      Corners kc;
      corners_of(r, m, kc);
      auto fetch = [&](int c, int b) { return __ldg(mesh + (int64_t)c * cells + kc.idx[b]); };
      interp_grad_one<C>(r, perm[i], i, fetch, u, u_const, cell, accumulate, disp_cot, wsum, u_sorted);
    }
    return;
  }
  if (!stage_mesh_rows(stage, mesh, m, C, x0, y0, RX, RY, &bar, polls)) return;
  const int SX = RX + 1, SY = RY + 1, nz = m.nz;
  for (uint32_t j = threadIdx.x; j < total; j += blockDim.x) {
    int k;
    const uint32_t i = tile_particle(j, seg_b, seg_n, &k);
    const Rec r = rec[i];
    const uint32_t row = r.key / (uint32_t)nz;
    const int cz = (int)(r.key - row * (uint32_t)nz);
    const int iy = (int)(row - (uint32_t)(x0 + k) * (uint32_t)m.ny) - y0;
    const int z1 = cz + 1 == nz ? 0 : cz + 1;
    auto fetch = [&](int c, int b) {
      const int bx = b & 1, by = (b >> 1) & 1, bz = (b >> 2) & 1;
      return stage[((c * SX + k + bx) * SY + iy + by) * nz + (bz ? z1 : cz)];
    };
    interp_grad_one<C>(r, perm[i], i, fetch, u, u_const, cell, accumulate, disp_cot, wsum, u_sorted);
  }
}

int interp_grad_sorted(const Rec* rec, const uint32_t* perm, const uint32_t* offs, int64_t n, Mesh3 m, int C,
                       const float* mesh, const float* u, float u_const, float cell, int accumulate, float* disp_cot,
                       float* wsum, float* u_sorted, cudaStream_t s, const uint32_t* status) {
  if (n == 0) return kOk;
  int RX, RY;
  if (offs != nullptr && stage_shape(m, C, mesh, &RX, &RY)) {
    const int64_t smem = stage_bytes(RX, RY, C, m.nz);
    const uint32_t min_stage = stage_threshold(smem, C);
    const unsigned grid = (unsigned)((int64_t)((m.nx + RX - 1) / RX) * ((m.ny + RY - 1) / RY));
#define PMB_LAUNCH_IS(CC)                                                                                       \
  do {                                                                                                          \
    PMB_CUDA_CHECK(smem_optin((const void*)interp_grad_staged_kernel<CC>, (int)kStageBudget));                 \
    interp_grad_staged_kernel<CC><<<grid, 256, (size_t)smem, s>>>(rec, perm, offs, m, RX, RY, min_stage, mesh, u, \
                                                                   u_const, cell, accumulate, disp_cot, wsum,   \
                                                                   u_sorted, g_wait_polls, status);             \
  } while (0)
    switch (C) {
      case 1: PMB_LAUNCH_IS(1); break;
      case 2: PMB_LAUNCH_IS(2); break;
      case 3: PMB_LAUNCH_IS(3); break;
      case 4: PMB_LAUNCH_IS(4); break;
      default: return kUnsupported;
    }
#undef PMB_LAUNCH_IS
    masked_tail_interp_kernel<<<148, 256, 0, s>>>(perm, offs + m.rows(), n, C, u, u_const, accumulate, disp_cot, wsum,
                                                  u_sorted, status);
    PMB_CUDA_CHECK(cudaGetLastError());
    return kOk;
  }
  const int th = 256;
  const unsigned g = (unsigned)((n + th - 1) / th);
  const unsigned g2 = (unsigned)((n + kGatherTile - 1) / kGatherTile);
  if (C == 1) {
    interp_grad_kernel_x2<1><<<g2, kGatherThreads, 0, s>>>(rec, perm, n, m, mesh, u, u_const, cell, accumulate, disp_cot, wsum,
                                               u_sorted, status);
    PMB_CUDA_CHECK(cudaGetLastError());
    return kOk;
  }
  if (C == 3 && !accumulate) {
    interp_grad_direct_kernel<3><<<g2, kGatherThreads, 0, s>>>(rec, perm, n, m, mesh, u, u_const, cell, disp_cot, wsum,
                                                               u_sorted, status);
    PMB_CUDA_CHECK(cudaGetLastError());
    return kOk;
  }
  if (C == 3) {
    interp_grad_kernel_x2<3><<<g2, kGatherThreads, 0, s>>>(rec, perm, n, m, mesh, u, u_const, cell, accumulate, disp_cot, wsum,
                                               u_sorted, status);
    PMB_CUDA_CHECK(cudaGetLastError());
    return kOk;
  }
  switch (C) {
    case 2: interp_grad_kernel<2><<<g, th, 0, s>>>(rec, perm, n, m, mesh, u, u_const, cell, accumulate, disp_cot, wsum, u_sorted, status); break;
    case 4: interp_grad_kernel<4><<<g, th, 0, s>>>(rec, perm, n, m, mesh, u, u_const, cell, accumulate, disp_cot, wsum, u_sorted, status); break;
    default: return kUnsupported;
  }
  PMB_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

}  // namespace pmb
