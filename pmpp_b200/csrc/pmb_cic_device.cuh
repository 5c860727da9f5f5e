// Device-side CIC building blocks shared by the single-simulation kernels
// (cic.cu) and the persistent ensemble kernels (ensemble.cu).
//
// Reference semantics: cic/enmesh.py:34-165 (binning and weights),
// cic/scatter.py:315-338 and cic/gather.py:452-472 (deposit / interpolation).
#pragma once

#include "pmb_common.cuh"

namespace pmb {

struct Binned {
  int cx, cy, cz;
  float fx, fy, fz;
};

// Lower CIC corner and fractions of one particle: d = disp / cell in IEEE
// float, corner = pmid + floor(d) (periodic), fraction = d - floor(d).
// A non-finite displacement is binned as zero (the anchor cell) so that every
// index stays in the mesh; the sort flags it (kFlagNonFiniteDisp).
__device__ __forceinline__ float finite_or_zero(float x) { return isfinite(x) ? x : 0.f; }

__device__ __forceinline__ Binned bin_particle(const int16_t* __restrict__ pmid, const float d0, const float d1,
                                               const float d2, int64_t i, Mesh3 m, float cell) {
  Binned b;
  float q0 = finite_or_zero(__fdiv_rn(d0, cell)), q1 = finite_or_zero(__fdiv_rn(d1, cell)),
        q2 = finite_or_zero(__fdiv_rn(d2, cell));
  float l0 = floorf(q0), l1 = floorf(q1), l2 = floorf(q2);
  b.fx = __fsub_rn(q0, l0);
  b.fy = __fsub_rn(q1, l1);
  b.fz = __fsub_rn(q2, l2);
  b.cx = wrap((int)pmid[3 * i + 0] + (int)l0, m.nx);
  b.cy = wrap((int)pmid[3 * i + 1] + (int)l1, m.ny);
  b.cz = wrap((int)pmid[3 * i + 2] + (int)l2, m.nz);
  return b;
}

// Origin of the mesh in the particles' frame, split as whole cells q and a
// remainder r in [0, cell): the reference's common-grid offset path
// (cic/pallas.py:225-238, cic/enmesh.py:128-147) bins (disp - r) / cell from
// the anchor pmid - q.  A zero shift reproduces bin_particle bit for bit
// (d - 0 == d for every float).
struct BinShift {
  int qx, qy, qz;
  float rx, ry, rz;
};

__device__ __forceinline__ Binned bin_particle(const int16_t* __restrict__ pmid, float d0, float d1, float d2,
                                               int64_t i, Mesh3 m, float cell, const BinShift& sh) {
  Binned b;
  const float q0 = finite_or_zero(__fdiv_rn(__fsub_rn(d0, sh.rx), cell)),
              q1 = finite_or_zero(__fdiv_rn(__fsub_rn(d1, sh.ry), cell)),
              q2 = finite_or_zero(__fdiv_rn(__fsub_rn(d2, sh.rz), cell));
  const float l0 = floorf(q0), l1 = floorf(q1), l2 = floorf(q2);
  b.fx = __fsub_rn(q0, l0);
  b.fy = __fsub_rn(q1, l1);
  b.fz = __fsub_rn(q2, l2);
  b.cx = wrap((int)pmid[3 * i + 0] - sh.qx + (int)l0, m.nx);
  b.cy = wrap((int)pmid[3 * i + 1] - sh.qy + (int)l1, m.ny);
  b.cz = wrap((int)pmid[3 * i + 2] - sh.qz + (int)l2, m.nz);
  return b;
}

// Key of the records of particles left out by a validity mask (cic/pallas.py:
// 133-141): they follow the last mesh row, deposit nothing, gather zero and
// take no adjoint.  No cell has this key (meshes hold fewer than 2^32 - 1
// cells).
constexpr uint32_t kMaskedKey = 0xFFFFFFFFu;

// A record that is safe to interpolate from (cell 0) in place of a masked one.
__device__ __forceinline__ Rec unmasked_or_origin(const Rec& r, bool* masked) {
  *masked = r.key == kMaskedKey;
  if (!*masked) return r;
  Rec z;
  z.fx = z.fy = z.fz = 0.f;
  z.key = 0u;
  return z;
}

// Exact n / d for every 32-bit n: a multiplication by a rounded-up reciprocal of 33
// bits and shifts (Granlund and Montgomery, "Division by Invariant Integers using
// Multiplication", 1994, figure 4.1).
struct FastDiv {
  uint32_t mul;
  int sh1, sh2;
};

inline FastDiv fast_div(uint32_t d) {
  int l = 0;
  while (l < 32 && (1ull << l) < d) ++l;
  FastDiv f;
  f.mul = (uint32_t)((((1ull << l) - d) << 32) / d + 1);
  f.sh1 = l < 1 ? l : 1;
  f.sh2 = l > 1 ? l - 1 : 0;
  return f;
}

__device__ __forceinline__ uint32_t div_by(uint32_t n, FastDiv f) {
  const uint32_t q = __umulhi(f.mul, n);
  return (q + ((n - q) >> f.sh1)) >> f.sh2;
}

struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2_pack(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_bits(F2 x, int& a, int& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(x.v));
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_mul_rz(F2 a, F2 b) {
  F2 r;
  asm("mul.rz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

__device__ __forceinline__ float pow2f(int e) { return __int_as_float((127 + e) << 23); }  // -126 <= e <= 127

constexpr int kMaxSrcRows = 25;  // (RX + 1) (RY + 1) of a tile
constexpr int kMaxTile = 11;     // so RX, RY <= 11

// Shared-memory bookkeeping of one scatter tile: per pass and source x the
// records' range (as prefix sums of visits) and first row.
struct ScatterSmem {
  uint32_t pre[2][kMaxTile + 2], beg[2][kMaxTile + 1], row[2][kMaxTile + 1];
  // dynamic accumulator bytes of an RX x RY block
  static constexpr int64_t acc_bytes(int RX, int RY, int nz) { return (int64_t)8 * RX * RY * nz; }
};

// One RX x RY block of output rows at (x0, y0) of mesh m, shape known at run
// time (cic.cu's scatter_rows_kernel has the constant shapes and explains the
// arithmetic): pulls the particles of the (RX+1) x (RY+1) source rows that
// reach the block (offs[row] .. offs[row+1] in the sorted records; offs points
// at this mesh's first row), sums the constant val > 0 times the weights as
// integers in units of 1/scale on two 32-bit planes in shared memory, and
// writes every output cell once as the Poisson source (rho - 1) * src_mul
// (gravity.py:628-630).  The sums are exact, so the result is independent of
// the particle order and bit-identical to scatter_rows_kernel's.  Called by
// all threads of the block; leaves it synchronised.  by_nz: m.nz.
//
// Three 16-bit planes with 64-bit conversions per corner, in 2 x 2 rows, took
// 1.70 ms for five deposits of 24 members on 64^3 to 128^3 cells; this takes
// 1.07 ms in 4 x 4 rows.
__device__ __forceinline__ void scatter_tile(const Rec* __restrict__ rec, const uint32_t* __restrict__ offs, Mesh3 m,
                                             FastDiv by_nz, int RX, int RY, int x0, int y0, float val, double scale,
                                             int E, float src_mul, float* __restrict__ out, unsigned int* acc,
                                             ScatterSmem& sm) {
  const int nz = m.nz, cells = RX * RY * nz;
  const int rxe = min(RX, m.nx - x0), rye = min(RY, m.ny - y0);
  {
    uint4* a4 = reinterpret_cast<uint4*>(acc);
    const int n4 = (2 * cells) >> 2;
    for (int t = threadIdx.x; t < n4; t += blockDim.x) a4[t] = make_uint4(0u, 0u, 0u, 0u);
    for (int t = 4 * n4 + threadIdx.x; t < 2 * cells; t += blockDim.x) acc[t] = 0u;
  }
  if (threadIdx.x < 2 * (kMaxTile + 1)) {
    const int pass = threadIdx.x > kMaxTile, k = threadIdx.x - pass * (kMaxTile + 1);
    uint32_t b = 0, c = 0, row = 0;
    if (k <= rxe && (pass == 0 || y0 == 0)) {
      const int x = k == 0 ? (x0 == 0 ? m.nx - 1 : x0 - 1) : x0 + k - 1;
      row = (uint32_t)((int64_t)x * m.ny) + (uint32_t)(pass == 0 ? y0 : m.ny);
      const int64_t lo = pass == 0 ? (int64_t)row - (y0 > 0) : (int64_t)row - 1;
      const int64_t hi = pass == 0 ? (int64_t)row + rye : (int64_t)row;
      b = offs[lo];
      c = offs[hi] - b;
    }
    sm.beg[pass][k] = b;
    sm.pre[pass][k + 1] = c;
    sm.row[pass][k] = row;
  }
  __syncthreads();
  uint32_t kcell = 0;  // particles that may reach one cell: those of two neighbouring source x
  for (int k = 0; k < RX; ++k)
    kcell = max(kcell, sm.pre[0][k + 1] + sm.pre[1][k + 1] + sm.pre[0][k + 2] + sm.pre[1][k + 2]);
  __syncthreads();
  if (threadIdx.x < 2) {
    uint32_t run = 0;
    sm.pre[threadIdx.x][0] = 0;
    for (int k = 1; k <= kMaxTile + 1; ++k) {
      run += sm.pre[threadIdx.x][k];
      sm.pre[threadIdx.x][k] = run;
    }
  }
  const int dup = (m.nx == 1 ? 2 : 1) * (m.ny == 1 ? 2 : 1) * (m.nz == 1 ? 2 : 1);
  const uint64_t kmax = (uint64_t)kcell * (uint64_t)dup;
  const int L = kmax ? 64 - __clzll((long long)kmax) : 0;
  const int lo = max(max(E - 24, L + E - 32), 1), hi = min(24, 32 - L);
  const int s = max(lo, min(hi, (E + 1) / 2));
  const bool split = lo <= hi && scale >= 0x1p-50 && scale <= 0x1p100 && val >= 0.f;
  const float v = split ? __fmul_rn(val, __fmul_rn((float)scale, pow2f(-s - 49))) : val;
  const F2 v2 = f2_pack(v, v), to_h = f2_pack(pow2f(-100), pow2f(-100)), back = f2_pack(-pow2f(100), -pow2f(100));
  const F2 to_l = f2_pack(pow2f(s - 100), pow2f(s - 100));
  int* const planes = reinterpret_cast<int*>(acc);
  unsigned long long* const acc64 = reinterpret_cast<unsigned long long*>(acc);
  __syncthreads();
  for (int pass = 0; pass < 2; ++pass) {
    const uint32_t end = sm.pre[pass][kMaxTile + 1];
    for (uint32_t vi = threadIdx.x; vi < end; vi += blockDim.x) {
      int k = 0;
      while (vi >= sm.pre[pass][k + 1]) ++k;
      const Rec r = rec[sm.beg[pass][k] + (vi - sm.pre[pass][k])];
      const uint32_t rowk = div_by(r.key, by_nz);
      const int sx = k - 1, ly = (int)(rowk - sm.row[pass][k]), cz = (int)(r.key - rowk * (uint32_t)nz);
      const int dz = cz + 1 == nz ? 1 - nz : 1;
      const F2 wz = f2_pack(axis_weight(r.fz, 0), axis_weight(r.fz, 1));
#pragma unroll
      for (int bx = 0; bx < 2; ++bx) {
        const int lx = sx + bx;
        const float wx = axis_weight(r.fx, bx);
#pragma unroll
        for (int by = 0; by < 2; ++by) {
          if (lx < 0 || lx >= rxe || ly + by < 0 || ly + by >= rye) continue;
          const float wxy = __fmul_rn(wx, axis_weight(r.fy, by));
          const F2 q = f2_mul(v2, f2_mul(f2_pack(wxy, wxy), wz));
          const int a0 = (lx * RY + ly + by) * nz + cz, a1 = a0 + dz;
          int i0, i1, l0, l1;
          if (split) {
            const F2 t = f2_mul_rz(q, to_h);
            f2_bits(t, i0, i1);
            f2_bits(f2_mul(f2_fma(t, back, q), to_l), l0, l1);
            atomicAdd(planes + a0, i0);
            atomicAdd(planes + cells + a0, l0);
            atomicAdd(planes + a1, i1);
            atomicAdd(planes + cells + a1, l1);
          } else {
            f2_bits(q, i0, i1);
            atomicAdd(&acc64[a0], (unsigned long long)__double2ll_rn((double)__int_as_float(i0) * scale));
            atomicAdd(&acc64[a1], (unsigned long long)__double2ll_rn((double)__int_as_float(i1) * scale));
          }
        }
      }
    }
  }
  __syncthreads();
  // (float)(sum / scale): sums below 2^23 on both planes in single precision
  // with one rounding, the others exactly in double precision
  const double inv = __hiloint2double(0x7FE00000 - __double2hiint(scale), 0);
  const float invf = (float)inv, two_s = pow2f(split ? s : 0);
  const bool fconv = split && invf >= 0x1p-126f;
  for (int row = 0; row < RX * RY; ++row) {
    const int lx = row / RY, ly = row - lx * RY;
    if (lx >= rxe || ly >= rye) continue;
    float* o = out + ((int64_t)(x0 + lx) * m.ny + (y0 + ly)) * nz;
    for (int z = threadIdx.x; z < nz; z += blockDim.x) {
      const int a = row * nz + z;
      float rho;
      if (split) {
        const uint32_t h = acc[a], l = acc[cells + a];
        if (fconv && (h | l) < 0x800000u)
          rho = __fmul_rn(__fmaf_rn(__uint_as_float(0x4B000000u + h) - 0x1p23f, two_s,
                                    __uint_as_float(0x4B000000u + l) - 0x1p23f),
                          invf);
        else
          rho = (float)(fma(__hiloint2double(0x43300000, (int)h) - 0x1p52, (double)two_s,
                            __hiloint2double(0x43300000, (int)l) - 0x1p52) *
                        inv);
      } else {
        rho = (float)((double)(long long)acc64[a] * inv);
      }
      o[z] = __fmul_rn(__fsub_rn(rho, 1.0f), src_mul);
    }
  }
  __syncthreads();
}

struct Corners {
  int64_t idx[8];
  float w[8];
};

// Raveled indices and weights of the eight CIC corners of a sorted record;
// corner c moves +1 along axis a when bit a of c is set.
__device__ __forceinline__ void corners_of(const Rec& r, Mesh3 m, Corners& k) {
  const uint32_t key = r.key;
  int cx, cy, cz;
  if (((m.nz & (m.nz - 1)) | (m.ny & (m.ny - 1))) == 0) {
    // power-of-two rows and planes: shifts instead of divisions
    const int lz = __ffs(m.nz) - 1, ly = __ffs(m.ny) - 1;
    cz = (int)(key & (uint32_t)(m.nz - 1));
    cy = (int)((key >> lz) & (uint32_t)(m.ny - 1));
    cx = (int)(key >> (lz + ly));
  } else {
    cz = (int)(key % (uint32_t)m.nz);
    const uint32_t rowk = key / (uint32_t)m.nz;
    cy = (int)(rowk % (uint32_t)m.ny);
    cx = (int)(rowk / (uint32_t)m.ny);
  }
  // lower corner and the (periodic) steps to the upper one along each axis
  const int64_t plane = (int64_t)m.ny * m.nz;
  const int64_t base = (int64_t)key;  // raveled lower cell, (cx * ny + cy) * nz + cz
  const int64_t dx = cx + 1 == m.nx ? -(int64_t)cx * plane : plane;
  const int64_t dy = cy + 1 == m.ny ? -(int64_t)cy * m.nz : (int64_t)m.nz;
  const int64_t dz = cz + 1 == m.nz ? -(int64_t)cz : 1;
  const float wx[2] = {axis_weight(r.fx, 0), axis_weight(r.fx, 1)};
  const float wy[2] = {axis_weight(r.fy, 0), axis_weight(r.fy, 1)};
  const float wz[2] = {axis_weight(r.fz, 0), axis_weight(r.fz, 1)};
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int bx = c & 1, by = (c >> 1) & 1, bz = (c >> 2) & 1;
    k.idx[c] = base + (bx ? dx : 0) + (by ? dy : 0) + (bz ? dz : 0);
    k.w[c] = __fmul_rn(__fmul_rn(wx[bx], wy[by]), wz[bz]);
  }
}

// out[src, c] = sum_b mesh_c[i_b] w_b for one sorted record; with vel the
// half-kick vel += out * kick is applied in place (integrator.py:536).
// vel + a k1 (+ a k2): one or two half-kicks with the same acceleration, in
// order, each with two roundings as the separate update would (k2 == 0: none).
__device__ __forceinline__ float kicked(float v, float a, float k1, float k2) {
  v = __fadd_rn(v, __fmul_rn(a, k1));
  if (k2 != 0.f) v = __fadd_rn(v, __fmul_rn(a, k2));
  return v;
}

template <int C>
__device__ __forceinline__ void gather_one(const Rec& r, uint32_t src, Mesh3 m, const float* __restrict__ mesh,
                                           float* __restrict__ out, float* __restrict__ vel, float kick,
                                           float kick2 = 0.f) {
  if (r.key == kMaskedKey) {
    // masked particle: zero value, velocity untouched (a zero kick)
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (out != nullptr) out[(int64_t)src * C + c] = 0.f;
    return;
  }
  Corners k;
  corners_of(r, m, k);
  // velocities loaded ahead of the corner loads (latency overlapped)
  float u[C];
  if (vel != nullptr) {
#pragma unroll
    for (int c = 0; c < C; ++c) u[c] = vel[(int64_t)src * C + c];
  }
  const int64_t cells = m.cells();
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const float* mc = mesh + (int64_t)c * cells;
    float a = 0.f;
#pragma unroll
    for (int b = 0; b < 8; ++b) a = __fadd_rn(a, __fmul_rn(__ldg(mc + k.idx[b]), k.w[b]));
    if (out != nullptr) out[(int64_t)src * C + c] = a;
    if (vel != nullptr) vel[(int64_t)src * C + c] = kicked(u[c], a, kick, kick2);
  }
}

}  // namespace pmb
