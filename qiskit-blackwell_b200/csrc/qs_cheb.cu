// qs_cheb.cu — CSR SpMV and the Chebyshev recurrence for exp(-iHt)|psi>.
//
// Rows are processed by V-lane sub-warps (V = 1..32, picked from the mean row
// length and the number of rows; rows far above the mean by whole warps).  A 20-qubit Hamiltonian of 30 entries per row
// takes 104 us per degree with V = 4 (4.3 TB/s of its 12 nnz + 44 N bytes) and
// 322 us with a warp per row, whose gathers used 8 bytes of each 32-byte sector
// and whose merge cost 150 instructions per row.  Each lane
// accumulates its entries with error-free products and TwoSum (a compensated
// "Kahan" row sum); lanes are combined in a fixed shuffle order, also
// compensated, so results are deterministic.
//
// The fused recurrence kernel does, per degree k and row r, in one launch:
//     t      = 2 * scale * (A x_{k})_r - x_{k-1,r}      (x_{k+1}, in place of x_{k-1})
//     out_r += c_{k+1} * t
// which needs three vectors instead of the reference's five
// (blackwell_backend/chebyshev.py:117-123).
#include "qs_api.h"
#include "qs_common.cuh"
#include "qs_rows.h"
#include <algorithm>
#include <vector>

using namespace qs;

namespace {

constexpr int kThreads = 256;
constexpr int kPauliThreads = 256;

struct Acc { float s, c; };  // compensated sum: value = s + c

__device__ __forceinline__ void acc_add_prod(Acc& a, float x, float y) {
  float p, e, q;
  two_prod(x, y, p, e);
  two_sum(a.s, p, a.s, q);
  a.c = __fadd_rn(a.c, __fadd_rn(q, e));
}

template <int V>
__device__ __forceinline__ Acc acc_reduce(Acc a) {
#pragma unroll
  for (int o = V / 2; o > 0; o >>= 1) {
    float s2 = __shfl_down_sync(0xffffffffu, a.s, o, V);
    float c2 = __shfl_down_sync(0xffffffffu, a.c, o, V);
    float s, e;
    two_sum(a.s, s2, s, e);
    a.s = s;
    a.c = __fadd_rn(__fadd_rn(a.c, c2), e);
  }
  return a;
}

// Adds a lane's entries of a row, V entries apart, to the sums.  kAhead of them
// are in flight: their columns and values, then the gathers, then the sums (in
// the row's order).  More of them help the wide rows and only add predicated
// work to the short ones.
template <int V, int kAhead>
__device__ __forceinline__ float2 row_dot(RowWalk w, const int32_t* __restrict__ ci, const float2* __restrict__ val,
                                          const float2* __restrict__ x) {
  Acc re{0.f, 0.f}, im{0.f, 0.f};
  for (; w.more(); w.step(V * kAhead)) {
    const int32_t* cj = ci + w.at;
    const float2* vj = val + w.at;
    int32_t col[kAhead];
    float2 v[kAhead], xj[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const bool in = w.has(u * V);
      col[u] = in ? cj[u * V] : -1;
      v[u] = in ? vj[u * V] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (col[u] >= 0) xj[u] = x[col[u]];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (col[u] < 0) break;
      acc_add_prod(re, v[u].x, xj[u].x);
      acc_add_prod(re, -v[u].y, xj[u].y);
      acc_add_prod(im, v[u].x, xj[u].y);
      acc_add_prod(im, v[u].y, xj[u].x);
    }
  }
  re = acc_reduce<V>(re);
  im = acc_reduce<V>(im);
  return make_float2(__fadd_rn(re.s, re.c), __fadd_rn(im.s, im.c));
}

// store(r, (A x)_r) for every row.  Every warp handles 32/V consecutive rows per
// iteration, so all 32 lanes always execute the same shuffles.
//
// Rows of more than 64 V entries wait until the warp's others are done and are
// then walked by all its lanes, one after the other: V follows the mean row, and a
// star's centre or an arrowhead's first row in a few lanes would keep its warp
// long after the rest of the launch (one row of 2^17 entries among rows of 2: 0.96
// ms, 21 in the one lane of V = 1; among rows of 30: 0.98 / 7.0).  64 V leaves rows of
// twice the mean in their own lanes; Pareto rows (mean 5, exponent 1.3) take 204 /
// 218 / 243 us for 32 V / 64 V / 128 V, rows of one length the same.  Both walks in
// one loop cost every matrix registers (48 instead of 32): 11.8 instead of 9.6 ms
// for the 20-qubit evolution, which this form takes 9.0 against 9.1 without it;
// rows of 5 take 95 us against 92.
template <int V, class F>
__device__ __forceinline__ void for_rows(const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                         const float2* __restrict__ val, int64_t nrows, const float2* __restrict__ x,
                                         F store) {
  constexpr int kAhead = V <= 4 ? 2 : 4, rpw = 32 / V;
  const int lane = threadIdx.x & (V - 1);
  const int sub = (threadIdx.x & 31) / V;
  const int64_t first = (int64_t)(gtid() >> 5) * rpw, step = (int64_t)(gstride() >> 5) * rpw;
  bool late = false;
  for (int64_t base = first; base < nrows; base += step) {
    const int64_t r = base + sub;
    const bool live = r < nrows;
    int32_t b = 0, e = 0;
    if (live) { b = rp[r]; e = rp[r + 1]; }
    const bool whole = V < 32 && e - b > 64 * V;
    late |= whole;
    const float2 d = row_dot<V, kAhead>(RowWalk(b, whole ? b : e, lane), ci, val, x);
    if (live && lane == 0 && !whole) store(r, d);
  }
  if constexpr (V < 32) {
    if (!__any_sync(0xffffffffu, late)) return;
    for (int64_t base = first; base < nrows; base += step) {
      const int64_t r = base + sub;
      int32_t b = 0, e = 0;
      if (r < nrows) { b = rp[r]; e = rp[r + 1]; }
      for (uint32_t rows = __ballot_sync(0xffffffffu, lane == 0 && e - b > 64 * V); rows; rows &= rows - 1) {
        const int from = __ffs((int)rows) - 1;
        const RowWalk w(__shfl_sync(0xffffffffu, b, from), __shfl_sync(0xffffffffu, e, from), threadIdx.x & 31);
        const float2 d = row_dot<32, kAhead>(w, ci, val, x);
        if ((threadIdx.x & 31) == 0) store(base + from / V, d);
      }
    }
  }
}

template <int V>
__global__ void __launch_bounds__(kThreads, V <= 4 ? 8 : 6)
    k_spmv(const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, const float2* __restrict__ val,
           int64_t nrows, const float2* __restrict__ x, float2* __restrict__ y, float2 alpha, float2 beta) {
  pdl_begin();
  for_rows<V>(rp, ci, val, nrows, x, [&](int64_t r, float2 d) {
    const float2 yo = y[r];
    float2 o;
    o.x = alpha.x * d.x - alpha.y * d.y + (beta.x * yo.x - beta.y * yo.y);
    o.y = alpha.x * d.y + alpha.y * d.x + (beta.x * yo.y + beta.y * yo.x);
    y[r] = o;
  });
}

// Fused Chebyshev degree step.  xprev is overwritten with x_next.
template <int V>
__global__ void __launch_bounds__(kThreads, V <= 4 ? 8 : 6)
    k_cheb_fused(const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, const float2* __restrict__ val,
                 int64_t nrows, const float2* __restrict__ xk, float2* __restrict__ xprev, float2* __restrict__ out,
                 float two_scale, float2 c) {
  pdl_begin();
  for_rows<V>(rp, ci, val, nrows, xk, [&](int64_t r, float2 d) {
    const float2 p = xprev[r];
    const float2 t = make_float2(fmaf(two_scale, d.x, -p.x), fmaf(two_scale, d.y, -p.y));
    xprev[r] = t;
    float2 a = out[r];
    a.x = fmaf(c.x, t.x, fmaf(-c.y, t.y, a.x));
    a.y = fmaf(c.x, t.y, fmaf(c.y, t.x, a.y));
    out[r] = a;
  });
}

// x1 = scale * A x0 ; out = c0 * x0 + c1 * x1
template <int V>
__global__ void __launch_bounds__(kThreads, V <= 4 ? 8 : 6)
    k_cheb_first(const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, const float2* __restrict__ val,
                 int64_t nrows, const float2* __restrict__ x0, float2* __restrict__ x1, float2* __restrict__ out,
                 float scale, float2 c0, float2 c1) {
  pdl_begin();
  for_rows<V>(rp, ci, val, nrows, x0, [&](int64_t r, float2 d) {
    const float2 t = make_float2(scale * d.x, scale * d.y);
    x1[r] = t;
    const float2 a0 = x0[r];
    float2 a;
    a.x = c0.x * a0.x - c0.y * a0.y;
    a.y = c0.x * a0.y + c0.y * a0.x;
    a.x = fmaf(c1.x, t.x, fmaf(-c1.y, t.y, a.x));
    a.y = fmaf(c1.x, t.y, fmaf(c1.y, t.x, a.y));
    out[r] = a;
  });
}

// ---- reference mirrors (chebyshev_sm120.cu:24-91): float4 elementwise ----
__global__ void k_step(const float4* __restrict__ s, const float4* __restrict__ p, float4* __restrict__ nx, uint64_t nv) {
  pdl_begin();
  for (uint64_t i = gtid(); i < nv; i += gstride()) {
    float4 a = s[i], b = p[i];
    nx[i] = make_float4(2.f * a.x - b.x, 2.f * a.y - b.y, 2.f * a.z - b.z, 2.f * a.w - b.w);
  }
}
__global__ void k_accum(float4* __restrict__ acc, const float4* __restrict__ t, float2 c, uint64_t nv) {
  pdl_begin();
  for (uint64_t i = gtid(); i < nv; i += gstride()) {
    float4 a = acc[i], x = t[i];
    a.x += c.x * x.x - c.y * x.y;
    a.y += c.x * x.y + c.y * x.x;
    a.z += c.x * x.z - c.y * x.w;
    a.w += c.x * x.w + c.y * x.z;
    acc[i] = a;
  }
}
__global__ void k_step_accum(const float4* __restrict__ s, const float4* __restrict__ p, float4* __restrict__ nx,
                             float4* __restrict__ acc, float2 c, uint64_t nv) {
  pdl_begin();
  for (uint64_t i = gtid(); i < nv; i += gstride()) {
    float4 a = s[i], b = p[i], r = acc[i];
    float4 t = make_float4(2.f * a.x - b.x, 2.f * a.y - b.y, 2.f * a.z - b.z, 2.f * a.w - b.w);
    r.x += c.x * t.x - c.y * t.y;
    r.y += c.x * t.y + c.y * t.x;
    r.z += c.x * t.z - c.y * t.w;
    r.w += c.x * t.w + c.y * t.z;
    nx[i] = t;
    acc[i] = r;
  }
}

// ---- matrix-free Pauli-sum operator -------------------------------------
// (H x)_i = sum_t w_t (-1)^{popc((i^x_t) & z_t)} x[i ^ x_t],  w_t = c_t i^{|x_t&z_t|}.
// Terms live in shared memory; XOR with a constant maps aligned blocks onto
// aligned blocks, so the gathers of a warp stay coalesced.
struct __align__(16) PTerm { uint64_t x, z; float wr, wi, pad0, pad1; };

__device__ __forceinline__ float2 hx_row(const PTerm* __restrict__ st, int nterms, const float2* __restrict__ x,
                                         uint64_t i) {
  float re = 0.f, im = 0.f;
  for (int k = 0; k < nterms; ++k) {
    const PTerm T = st[k];
    const uint64_t j = i ^ T.x;
    const float2 v = x[j];
    const float sg = (__popcll(j & T.z) & 1) ? -1.f : 1.f;
    const float wr = sg * T.wr, wi = sg * T.wi;
    re = fmaf(wr, v.x, fmaf(-wi, v.y, re));
    im = fmaf(wr, v.y, fmaf(wi, v.x, im));
  }
  return make_float2(re, im);
}

__global__ void k_chebp_first(const PTerm* __restrict__ terms, int nterms, uint64_t n, const float2* __restrict__ x0,
                              float2* __restrict__ x1, float2* __restrict__ out, float scale, float2 c0, float2 c1) {
  pdl_begin();
  extern __shared__ PTerm st[];
  for (int k = threadIdx.x; k < nterms; k += blockDim.x) st[k] = terms[k];
  __syncthreads();
  for (uint64_t i = gtid(); i < n; i += gstride()) {
    const float2 d = hx_row(st, nterms, x0, i);
    const float2 t = make_float2(scale * d.x, scale * d.y);
    x1[i] = t;
    const float2 a0 = x0[i];
    float2 a;
    a.x = c0.x * a0.x - c0.y * a0.y;
    a.y = c0.x * a0.y + c0.y * a0.x;
    a.x = fmaf(c1.x, t.x, fmaf(-c1.y, t.y, a.x));
    a.y = fmaf(c1.x, t.y, fmaf(c1.y, t.x, a.y));
    out[i] = a;
  }
}

__global__ void k_chebp_fused(const PTerm* __restrict__ terms, int nterms, uint64_t n, const float2* __restrict__ xk,
                              float2* __restrict__ xprev, float2* __restrict__ out, float two_scale, float2 c) {
  pdl_begin();
  extern __shared__ PTerm st[];
  for (int k = threadIdx.x; k < nterms; k += blockDim.x) st[k] = terms[k];
  __syncthreads();
  for (uint64_t i = gtid(); i < n; i += gstride()) {
    const float2 d = hx_row(st, nterms, xk, i);
    const float2 p = xprev[i];
    const float2 t = make_float2(fmaf(two_scale, d.x, -p.x), fmaf(two_scale, d.y, -p.y));
    xprev[i] = t;
    float2 a = out[i];
    a.x = fmaf(c.x, t.x, fmaf(-c.y, t.y, a.x));
    a.y = fmaf(c.x, t.y, fmaf(c.y, t.x, a.y));
    out[i] = a;
  }
}

// Up to 32 qubits the matrix-free recurrence uses 32-bit indices and splits
// H into its diagonal and off-diagonal parts:
//   * terms with x_t = 0 sum to a real diagonal D_i = sum_t c_t (-1)^{popc(i & z_t)},
//     tabulated once per evolution (FP64 sums rounded to FP32, 4 B per
//     amplitude), so the degree loop reads D_i instead of evaluating them;
//   * every other weight w_t = c_t i^{|x_t & z_t|} is real or imaginary; terms
//     of equal X mask and kind are paired (e.g. X_a X_b and Y_a Y_b) so that a
//     pair shares its gather x[i ^ x], and a lone term has a zero partner.
// The pairs come in four runs, real / imaginary weights by even / odd X masks.
struct __align__(16) PMask {
  uint32_t x;        // X mask
  uint32_t z0, z1;   // Z masks without the bits a thread holds in registers
  uint32_t pat;      // signs of those bits: byte 0 for z0, byte 1 for z1
  float w0, w1;      // weights (real, or the factor of i)
  float pad0, pad1;
};
struct PRuns { int r0, r1, i0, end; };  // [0,r0) real even, [r0,r1) real odd, [r1,i0) imaginary even, [i0,end) odd
struct __align__(16) PDiag { uint64_t z; double c; };

__global__ void k_chebp_diag(const PDiag* __restrict__ terms, int nterms, uint64_t n, float* __restrict__ D) {
  pdl_begin();
  extern __shared__ PDiag sd[];
  for (int k = threadIdx.x; k < nterms; k += blockDim.x) sd[k] = terms[k];
  __syncthreads();
  for (uint64_t i = gtid(); i < n; i += gstride()) {
    double d = 0.0;
    for (int k = 0; k < nterms; ++k) d += (__popcll(i & sd[k].z) & 1) ? -sd[k].c : sd[k].c;
    D[i] = (float)d;
  }
}

__device__ __forceinline__ float flip_if(float w, uint32_t sbit) { return __int_as_float(__float_as_int(w) ^ sbit); }

// One run of pairs on a thread's 2*M amplitudes (qubit 0, and qubits 6 and 7
// for M = 4; v[m] is one 16-byte gather of two amplitudes, a warp's 32 lanes
// covering 512 consecutive bytes of it).  The parity of the
// index bits outside the registers is taken once for the 2*M amplitudes (POPC
// runs at an eighth of the FP32 rate); inside them the sign is a bit of `pat`.
// SWAP: the X mask has bit 0, so the two amplitudes of a gather trade places.
template <int M, bool IMAG, bool SWAP>
__device__ __forceinline__ void pauli_run(const PMask* __restrict__ sp, int b, int e, const float4* __restrict__ x4,
                                          uint32_t t4, float2 (&acc)[2 * M]) {
  auto add = [&](int r, float w, float vx, float vy) {
    float2& a = acc[SWAP ? r ^ 1 : r];
    if (IMAG) {
      a.x = fmaf(-w, vy, a.x);
      a.y = fmaf(w, vx, a.y);
    } else {
      a.x = fmaf(w, vx, a.x);
      a.y = fmaf(w, vy, a.y);
    }
  };
#pragma unroll 2
  for (int k = b; k < e; ++k) {
    const PMask P = sp[k];
    const uint32_t j4 = t4 ^ (P.x >> 1);
    float4 v[M];
#pragma unroll
    for (int m = 0; m < M; ++m) v[m] = x4[j4 ^ (uint32_t)(m << 5)];
    const uint32_t j = j4 << 1;
    const float w0 = flip_if(P.w0, (uint32_t)__popc(j & P.z0) << 31);
    const float w1 = flip_if(P.w1, (uint32_t)__popc(j & P.z1) << 31);
    if (P.pat == 0) {
      const float w = w0 + w1;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        add(2 * m, w, v[m].x, v[m].y);
        add(2 * m + 1, w, v[m].z, v[m].w);
      }
    } else {
#pragma unroll
      for (int r = 0; r < 2 * M; ++r) {
        const float w = flip_if(w0, (P.pat << (31 - r)) & 0x80000000u) + flip_if(w1, (P.pat << (23 - r)) & 0x80000000u);
        const float4 u = v[r >> 1];
        add(r, w, (r & 1) ? u.z : u.x, (r & 1) ? u.w : u.y);
      }
    }
  }
}

// One degree of the recurrence, x_{k+1} in place of x_{k-1} and accumulated
// into out (FIRST: x_1 = scale H x_0 and out = c0 x_0 + c1 x_1).  S groups of a
// CTA's threads share its amplitudes, each taking a part of every run; their
// sums meet in shared memory in a fixed order.
//
// Bound by the gathers' L2 traffic and their issue slots.  22 qubits, 42 masks:
// 73 us per degree; 176 us with one amplitude per thread, of which the two
// POPCs of a pair (16 lanes per clock and SM: 149 thousand cycles) alone are 78.
template <int M, int S, bool FIRST>
__global__ void __launch_bounds__(kPauliThreads)
    k_chebp_masks(const PMask* __restrict__ masks, PRuns R, uint32_t nthr, const float2* __restrict__ D,
                  const float4* __restrict__ xk, float4* __restrict__ xprev, float4* __restrict__ out, float scale,
                  float2 c0, float2 c) {
  extern __shared__ __align__(16) PMask sm[];
  constexpr int G = kPauliThreads / S;   // threads of a group, a multiple of 32
  __shared__ float2 part[S > 1 ? S - 1 : 1][S > 1 ? 2 * M : 1][S > 1 ? G : 1];
  // the table was copied before the first kernel of the evolution began, so
  // it may be read before the kernel in front of this one has finished
  for (int k = threadIdx.x; k < R.end; k += blockDim.x) sm[k] = masks[k];
  pdl_begin();
  __syncthreads();
  const int s = threadIdx.x / G;
  auto cut = [&](int b, int e, int k) { return b + (e - b) * k / S; };
  const uint32_t g = blockIdx.x * (uint32_t)G + threadIdx.x % G;
  const bool live = g < nthr;
  const uint32_t t4 = (g >> 5) * (32u * M) + (g & 31u);
  float2 acc[2 * M];
#pragma unroll
  for (int r = 0; r < 2 * M; ++r) acc[r] = make_float2(0.f, 0.f);
  if (live) {
    if (D && s == 0) {
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const float2 d = D[t4 + 32 * m];
        const float4 v = xk[t4 + 32 * m];
        acc[2 * m] = make_float2(d.x * v.x, d.x * v.y);
        acc[2 * m + 1] = make_float2(d.y * v.z, d.y * v.w);
      }
    }
    pauli_run<M, false, false>(sm, cut(0, R.r0, s), cut(0, R.r0, s + 1), xk, t4, acc);
    pauli_run<M, false, true>(sm, cut(R.r0, R.r1, s), cut(R.r0, R.r1, s + 1), xk, t4, acc);
    pauli_run<M, true, false>(sm, cut(R.r1, R.i0, s), cut(R.r1, R.i0, s + 1), xk, t4, acc);
    pauli_run<M, true, true>(sm, cut(R.i0, R.end, s), cut(R.i0, R.end, s + 1), xk, t4, acc);
  }
  if (S > 1) {
    if (s > 0) {
#pragma unroll
      for (int r = 0; r < 2 * M; ++r) part[s - 1][r][threadIdx.x % G] = acc[r];
    }
    __syncthreads();
    if (s > 0) return;
    for (int q = 0; q < S - 1; ++q) {
#pragma unroll
      for (int r = 0; r < 2 * M; ++r) {
        const float2 v = part[q][r][threadIdx.x];
        acc[r].x += v.x;
        acc[r].y += v.y;
      }
    }
  }
  if (!live) return;
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const uint32_t i = t4 + 32 * m;
    const float2 d0 = acc[2 * m], d1 = acc[2 * m + 1];
    float4 t, a;
    if (FIRST) {
      t = make_float4(scale * d0.x, scale * d0.y, scale * d1.x, scale * d1.y);
      const float4 v = xk[i];
      a = make_float4(c0.x * v.x - c0.y * v.y, c0.x * v.y + c0.y * v.x, c0.x * v.z - c0.y * v.w,
                      c0.x * v.w + c0.y * v.z);
    } else {
      const float4 p = xprev[i];
      t = make_float4(fmaf(scale, d0.x, -p.x), fmaf(scale, d0.y, -p.y), fmaf(scale, d1.x, -p.z),
                      fmaf(scale, d1.y, -p.w));
      a = out[i];
    }
    xprev[i] = t;
    a.x = fmaf(c.x, t.x, fmaf(-c.y, t.y, a.x));
    a.y = fmaf(c.x, t.y, fmaf(c.y, t.x, a.y));
    a.z = fmaf(c.x, t.z, fmaf(-c.y, t.w, a.z));
    a.w = fmaf(c.x, t.w, fmaf(c.y, t.z, a.w));
    out[i] = a;
  }
}

int pick_V(int64_t nrows, const int32_t* rp_dev, qs_context* h) {
  // mean row length from the first and last row pointers
  int32_t ends[2] = {0, 0};
  QS_CUDA(cudaMemcpyAsync(&ends[0], rp_dev, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
  QS_CUDA(cudaMemcpyAsync(&ends[1], rp_dev + nrows, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
  QS_CUDA(cudaStreamSynchronize(h->stream));
  const double mean = nrows > 0 ? double(ends[1] - ends[0]) / double(nrows) : 1.0;
  // Few lanes per row: a warp then covers rows whose columns lie together, so
  // a gather's 32-byte sectors are used whole, and fewer lanes are merged by
  // shuffles.  Measured (64 M entries, us for V = 1 / 2 / 4 / 8 / 16 / 32):
  // 5 per row 120 / 136 / 181 / 292 / 576 / 1149, 20 per row 126 / 107 / 106 /
  // 132 / 194 / 318, 200 per row 178 / 118 / 118 / 97 / 105 / 124, 2000 per row
  // 1189 / 623 / 338 / 128 / 120 / 107.
  int V = mean <= 10 ? 1 : mean <= 16 ? 2 : mean <= 80 ? 4 : mean <= 250 ? 8 : mean <= 1000 ? 16 : 32;
  // A matrix with few rows is bound by the latency of a lane's entries: more
  // lanes until there are threads for every SM (13 qubits, 29 per row: V = 4
  // 549 us an evolution, V = 8 500).
  while (nrows * V < (1 << 16) && V < 32 && 2 * V <= mean) V *= 2;
  return V;
}

#define DISPATCH_V(V, KERN, GRID, ...)                                            \
  switch (V) {                                                                   \
    case 1: qs_launch_pdl(h, KERN<1>, dim3(GRID), dim3(kThreads), 0, __VA_ARGS__); break;       \
    case 2: qs_launch_pdl(h, KERN<2>, dim3(GRID), dim3(kThreads), 0, __VA_ARGS__); break;       \
    case 4: qs_launch_pdl(h, KERN<4>, dim3(GRID), dim3(kThreads), 0, __VA_ARGS__); break;       \
    case 8: qs_launch_pdl(h, KERN<8>, dim3(GRID), dim3(kThreads), 0, __VA_ARGS__); break;       \
    case 16: qs_launch_pdl(h, KERN<16>, dim3(GRID), dim3(kThreads), 0, __VA_ARGS__); break;     \
    default: qs_launch_pdl(h, KERN<32>, dim3(GRID), dim3(kThreads), 0, __VA_ARGS__); break;     \
  }

inline void check_vec(const void* p, const char* what) {
  if (!p || ((uintptr_t)p & 15u)) throw qs_error(QS_ERR_INVALID, std::string(what) + " must be a 16-byte aligned device pointer");
}

}  // namespace

extern "C" {

int qs_spmv_csr(qs_handle_t h, const int32_t* rp, const int32_t* ci, const void* val, int64_t nrows, const void* x,
                void* y, double ar, double ai, double br, double bi) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  QS_CHECK_ARG(rp && ci && val && x && y, "null CSR or vector pointer");
  QS_CHECK_ARG(nrows >= 0, "n_rows must be >= 0");
  QS_CHECK_ARG(x != y, "x and y must not alias");
  if (nrows == 0) return QS_OK;
  const int V = pick_V(nrows, rp, h);
  const unsigned grid = (unsigned)qs_blocks_for(h, (uint64_t)nrows * V, kThreads, 16);
  DISPATCH_V(V, k_spmv, grid, rp, ci, (const float2*)val, nrows, (const float2*)x, (float2*)y,
             make_float2((float)ar, (float)ai), make_float2((float)br, (float)bi));
  qs_after_launch(h, "k_spmv");
  QS_API_END(h)
}

int qs_cheb_step(qs_handle_t h, const void* s, const void* p, void* nx, int64_t n) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  check_vec(s, "spmv_result"); check_vec(p, "t_prev"); check_vec(nx, "t_next");
  QS_CHECK_ARG(n >= 0 && (n & 1) == 0, "n must be even and >= 0");
  const uint64_t nv = (uint64_t)n / 2;
  if (nv) {
    qs_launch_pdl(h, k_step, dim3(qs_blocks_for(h, nv, kThreads)), dim3(kThreads), 0, (const float4*)s, (const float4*)p, (float4*)nx, nv);
    qs_after_launch(h, "k_step");
  }
  QS_API_END(h)
}

int qs_cheb_accum(qs_handle_t h, void* acc, const void* t, double cr, double ci_, int64_t n) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  check_vec(acc, "accum"); check_vec(t, "t_k");
  QS_CHECK_ARG(n >= 0 && (n & 1) == 0, "n must be even and >= 0");
  const uint64_t nv = (uint64_t)n / 2;
  if (nv) {
    qs_launch_pdl(h, k_accum, dim3(qs_blocks_for(h, nv, kThreads)), dim3(kThreads), 0, (float4*)acc, (const float4*)t,
                                                                        make_float2((float)cr, (float)ci_), nv);
    qs_after_launch(h, "k_accum");
  }
  QS_API_END(h)
}

int qs_cheb_step_accum(qs_handle_t h, const void* s, const void* p, void* nx, void* acc, double cr, double ci_,
                       int64_t n) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  check_vec(s, "spmv_result"); check_vec(p, "t_prev"); check_vec(nx, "t_next"); check_vec(acc, "accum");
  QS_CHECK_ARG(n >= 0 && (n & 1) == 0, "n must be even and >= 0");
  const uint64_t nv = (uint64_t)n / 2;
  if (nv) {
    qs_launch_pdl(h, k_step_accum, dim3(qs_blocks_for(h, nv, kThreads)), dim3(kThreads), 0, 
        (const float4*)s, (const float4*)p, (float4*)nx, (float4*)acc, make_float2((float)cr, (float)ci_), nv);
    qs_after_launch(h, "k_step_accum");
  }
  QS_API_END(h)
}

int qs_cheb_evolve(qs_handle_t h, const int32_t* rp, const int32_t* ci, const void* val, int n, const void* psi,
                   void* out, const double* coeffs, int K, double scale, void* work) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(psi, n);
  qs_check_state(out, n);
  qs_check_state(work, n);
  QS_CHECK_ARG(rp && ci && val && coeffs, "null CSR or coefficient pointer");
  QS_CHECK_ARG(K >= 1, "K must be >= 1");
  const int64_t N = (int64_t)1 << n;
  float2* x0 = (float2*)work;        // x_{k-1}
  float2* x1 = x0 + N;               // x_k
  QS_CUDA(cudaMemcpyAsync(x0, psi, sizeof(float2) * N, cudaMemcpyDeviceToDevice, h->stream));
  const int V = pick_V(N, rp, h);
  const unsigned grid = (unsigned)qs_blocks_for(h, (uint64_t)N * V, kThreads, 16);
  auto C = [&](int k) { return make_float2((float)coeffs[2 * k], (float)coeffs[2 * k + 1]); };
  DISPATCH_V(V, k_cheb_first, grid, rp, ci, (const float2*)val, N, x0, x1, (float2*)out, (float)scale, C(0), C(1));
  qs_after_launch(h, "k_cheb_first");
  const float two_scale = (float)(2.0 * scale);
  for (int k = 2; k <= K; ++k) {
    // x0 holds x_{k-2}, x1 holds x_{k-1}; x0 becomes x_k
    DISPATCH_V(V, k_cheb_fused, grid, rp, ci, (const float2*)val, N, x1, x0, (float2*)out, two_scale, C(k));
    qs_after_launch(h, "k_cheb_fused");
    std::swap(x0, x1);
  }
  QS_API_END(h)
}

int qs_cheb_evolve_pauli(qs_handle_t h, int n, const void* psi, void* out, const uint64_t* xm, const uint64_t* zm,
                         const double* coefs, int nterms, const double* coeffs, int K, double scale, void* work) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(psi, n);
  qs_check_state(out, n);
  qs_check_state(work, n);
  QS_CHECK_ARG(xm && zm && coefs && coeffs, "null term or coefficient pointer");
  QS_CHECK_ARG(nterms >= 1 && nterms <= 1024, "n_terms must be in [1, 1024]");
  QS_CHECK_ARG(K >= 1, "K must be >= 1");
  const uint64_t lim = (1ull << n) - 1ull;
  std::vector<PTerm> T(nterms);
  static const float pr[4] = {1.f, 0.f, -1.f, 0.f}, pim[4] = {0.f, 1.f, 0.f, -1.f};
  for (int k = 0; k < nterms; ++k) {
    QS_CHECK_ARG((xm[k] & ~lim) == 0 && (zm[k] & ~lim) == 0, "Pauli mask has bits beyond n_qubits");
    const int ny = __builtin_popcountll(xm[k] & zm[k]) & 3;
    T[k] = PTerm{xm[k], zm[k], (float)(coefs[k] * pr[ny]), (float)(coefs[k] * pim[ny]), 0.f, 0.f};
  }
  const uint64_t N = 1ull << n;
  float2* x0 = (float2*)work;
  float2* x1 = x0 + N;
  auto C = [&](int k) { return make_float2((float)coeffs[2 * k], (float)coeffs[2 * k + 1]); };
  const float two_scale = (float)(2.0 * scale);
  if (n <= 32) {
    // Amplitudes per thread and groups per CTA.  Below 2^16 amplitudes a degree
    // is the latency of the mask loop, so two amplitudes per thread and the
    // masks over 8 groups (13 qubits, 84 terms, t = 2: 450 us; 594 in one
    // group); to 2^18 eight amplitudes and 4 groups keep the SMs filled (18
    // qubits 918 us; 1024 in one group); above, one group (22 qubits 73 us per
    // degree; 110 in 4 groups, 94 with two amplitudes per thread).
    const int M = n < 16 ? 1 : 4, S = n < 16 ? 8 : n < 19 ? 4 : 1;
    const uint32_t regs = M == 4 ? 0xC1u : 0x01u;   // the index bits inside a thread
    std::vector<PDiag> dg;
    std::vector<int> off;
    for (int k = 0; k < nterms; ++k) {
      if (xm[k] == 0) dg.push_back(PDiag{zm[k], coefs[k]});
      else off.push_back(k);
    }
    auto run_of = [&](int k) { return 2 * (__builtin_popcountll(xm[k] & zm[k]) & 1) + (int)(xm[k] & 1); };
    std::stable_sort(off.begin(), off.end(), [&](int a, int b) {
      return run_of(a) != run_of(b) ? run_of(a) < run_of(b) : xm[a] < xm[b];
    });
    // signs over a thread's 2*M source amplitudes: bit 2m + e for the gather
    // that output m reads, whose own register bits are m ^ (those of x)
    auto pattern = [&](uint64_t x, uint64_t z) {
      uint32_t pat = 0;
      for (int r = 0; r < 2 * M; ++r) {
        const uint64_t j = (uint64_t)(r & 1) | (((uint64_t)(r >> 1) << 6) ^ (x & regs & ~1ull));
        pat |= (uint32_t)(__builtin_popcountll(j & z & regs) & 1) << r;
      }
      return pat;
    };
    std::vector<PMask> pm;
    int ends[4] = {0, 0, 0, 0};
    for (size_t u = 0; u < off.size();) {
      const int a = off[u], run = run_of(a);
      auto weight = [&](int k) { return run < 2 ? T[k].wr : T[k].wi; };
      PMask P{(uint32_t)xm[a], (uint32_t)zm[a] & ~regs, 0u, pattern(xm[a], zm[a]), weight(a), 0.f, 0.f, 0.f};
      ++u;
      if (u < off.size() && xm[off[u]] == xm[a] && run_of(off[u]) == run) {
        const int b = off[u++];
        P.z1 = (uint32_t)zm[b] & ~regs;
        P.pat |= pattern(xm[b], zm[b]) << 8;
        P.w1 = weight(b);
      }
      pm.push_back(P);
      for (int r = run; r < 4; ++r) ends[r] = (int)pm.size();
    }
    const size_t pbytes = sizeof(PMask) * pm.size(), dbytes = sizeof(PDiag) * dg.size();
    char* dmem = (char*)h->scratch_get(std::max<size_t>(16, pbytes + dbytes));
    const PMask* dP = (const PMask*)dmem;
    const PDiag* dD = (const PDiag*)(dmem + pbytes);
    if (pbytes) QS_CUDA(cudaMemcpyAsync(dmem, pm.data(), pbytes, cudaMemcpyHostToDevice, h->stream));
    if (dbytes) QS_CUDA(cudaMemcpyAsync(dmem + pbytes, dg.data(), dbytes, cudaMemcpyHostToDevice, h->stream));
    float* D = nullptr;
    if (!dg.empty()) {
      QS_CUDA(cudaMallocAsync((void**)&D, sizeof(float) * N, h->stream));
      qs_launch_pdl(h, k_chebp_diag, dim3(qs_blocks_for(h, N, kThreads)), dim3(kThreads), dbytes, dD, (int)dg.size(), N, D);
      qs_after_launch(h, "k_chebp_diag");
    }
    try {
      QS_CUDA(cudaMemcpyAsync(x0, psi, sizeof(float2) * N, cudaMemcpyDeviceToDevice, h->stream));
      const uint32_t nthr = (uint32_t)(N / (2 * M));
      const uint32_t per = (uint32_t)(kPauliThreads / S);
      const dim3 grid((unsigned)((nthr + per - 1) / per));
      const PRuns R{ends[0], ends[1], ends[2], ends[3]};
      auto step = [&](auto kern, const float2* xk, float2* xp, float s, float2 c0, float2 c) {
        qs_launch_pdl(h, kern, grid, dim3(kPauliThreads), pbytes, dP, R, nthr, (const float2*)D, (const float4*)xk,
                      (float4*)xp, (float4*)out, s, c0, c);
        qs_after_launch(h, "k_chebp_masks");
      };
      auto first = M == 1 ? k_chebp_masks<1, 8, true> : S == 4 ? k_chebp_masks<4, 4, true> : k_chebp_masks<4, 1, true>;
      auto next = M == 1 ? k_chebp_masks<1, 8, false> : S == 4 ? k_chebp_masks<4, 4, false> : k_chebp_masks<4, 1, false>;
      step(first, x0, x1, (float)scale, C(0), C(1));
      for (int k = 2; k <= K; ++k) {
        step(next, x1, x0, two_scale, C(0), C(k));
        std::swap(x0, x1);
      }
    } catch (...) {
      if (D) cudaFreeAsync(D, h->stream);
      throw;
    }
    if (D) QS_CUDA(cudaFreeAsync(D, h->stream));
    return QS_OK;
  }
  PTerm* dT = (PTerm*)h->scratch_get(sizeof(PTerm) * nterms);
  QS_CUDA(cudaMemcpyAsync(dT, T.data(), sizeof(PTerm) * nterms, cudaMemcpyHostToDevice, h->stream));
  QS_CUDA(cudaMemcpyAsync(x0, psi, sizeof(float2) * N, cudaMemcpyDeviceToDevice, h->stream));
  const unsigned grid = (unsigned)qs_blocks_for(h, N, kThreads, 8);
  const size_t smem = sizeof(PTerm) * nterms;
  qs_launch_pdl(h, k_chebp_first, dim3(grid), dim3(kThreads), smem, dT, nterms, N, x0, x1, (float2*)out, (float)scale, C(0), C(1));
  qs_after_launch(h, "k_chebp_first");
  for (int k = 2; k <= K; ++k) {
    qs_launch_pdl(h, k_chebp_fused, dim3(grid), dim3(kThreads), smem, dT, nterms, N, x1, x0, (float2*)out, two_scale, C(k));
    qs_after_launch(h, "k_chebp_fused");
    std::swap(x0, x1);
  }
  QS_API_END(h)
}

}  // extern "C"
