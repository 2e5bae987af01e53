// qs_adjoint.cu — adjoint-method gradient of E(theta) = <psi|H|psi>.
//
// Method (Jones & Gacon, "Efficient calculation of gradients in classical
// simulations of variational quantum algorithms", arXiv:2009.02823):
//   psi = U_L..U_1|0>,  lam = H psi,  E = Re<psi|lam>;
//   for l = L..1:  if U_l = exp(-i theta G/2):  dE/dtheta += Im<lam|G|psi>
//                  psi <- U_l^dag psi,  lam <- U_l^dag lam.
// (2 Re<lam| dU/dtheta |psi_{l-1}> = 2 Re(-i/2 <lam|G U psi_{l-1}>) = Im<lam|G|psi_l>.)
//
// Both sweeps are cut into tile passes (below): psi, in the reverse sweep psi
// and lambda, cross HBM once per pass instead of once per gate, and CTAs apply
// the gates of a pass to a tile in shared memory.  The FP64 partial sums of
// <lambda|P|psi> are reduced in a fixed order (deterministic).
// QSIM_ADJ_PASSES=0 selects the older sweep (a batch-planned forward, then one
// launch per gate; kept for comparison).
// There is no reference counterpart (ROADMAP.md:173-175 lists adjoint
// differentiation as future work).
#include "qs_api.h"
#include "qs_common.cuh"
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>

using namespace qs;

void qs_pauli_apply(qs_context* h, const float2* in, float2* out, uint64_t vstride, int nb, int n, const uint64_t* x,
                    const uint64_t* z, const double* c, int nterms);

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double ws[32];
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) ws[w] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  v = 0.0;
  if (w == 0) { v = lane < nw ? ws[lane] : 0.0; v = warp_sum(v); }
  return v;
}

// Per-vector slicing along grid.x.
struct Slice { int nbx; uint64_t per; };
Slice slice(uint64_t items) {
  uint64_t nb = (items + 8191) / 8192;
  if (nb > 256) nb = 256;
  if (nb < 1) nb = 1;
  return Slice{(int)nb, (items + nb - 1) / nb};
}

struct Mat2 { float2 g[4]; };

// One 2x2 gate U^dag on both psi and lam of every vector b; if gkind != 0,
// partial[b][bx] = sum Im(<lam|G|psi>) over this block's pairs (before U^dag).
__global__ void k_adj_1q(float2* __restrict__ base, uint64_t vstride, uint64_t npairs, int t,
                         const Mat2* __restrict__ udag, int gkind, uint64_t per, double* __restrict__ partial) {
  const int b = blockIdx.y;
  float2* psi = base + (uint64_t)b * vstride;
  float2* lam = psi + (vstride / 3);
  const Mat2 U = udag[b];
  const uint64_t st = 1ull << t;
  const uint64_t p0 = (uint64_t)blockIdx.x * per, pe = min(p0 + per, npairs);
  double acc = 0.0;
  for (uint64_t p = p0 + threadIdx.x; p < pe; p += blockDim.x) {
    const uint64_t i0 = insert_zero(p, t), i1 = i0 | st;
    float2 a0 = psi[i0], a1 = psi[i1], l0 = lam[i0], l1 = lam[i1];
    if (gkind) {
      // (G psi) on the pair
      float2 g0, g1;
      if (gkind == 1) { g0 = a1; g1 = a0; }                                          // X
      else if (gkind == 2) { g0 = make_float2(a1.y, -a1.x); g1 = make_float2(-a0.y, a0.x); }  // Y
      else { g0 = a0; g1 = make_float2(-a1.x, -a1.y); }                             // Z
      // Im(conj(l) * g) = l.x*g.y - l.y*g.x
      acc += (double)l0.x * g0.y - (double)l0.y * g0.x + (double)l1.x * g1.y - (double)l1.y * g1.x;
    }
    psi[i0] = cfma2(U.g[0], a0, U.g[1], a1);
    psi[i1] = cfma2(U.g[2], a0, U.g[3], a1);
    lam[i0] = cfma2(U.g[0], l0, U.g[1], l1);
    lam[i1] = cfma2(U.g[2], l0, U.g[3], l1);
  }
  if (gkind) {
    acc = block_sum(acc);
    if (threadIdx.x == 0) partial[(uint64_t)b * gridDim.x + blockIdx.x] = acc;
  }
}

struct Mat4 { float2 g[16]; };
__global__ void k_adj_2q(float2* __restrict__ base, uint64_t vstride, uint64_t nquads, int q0, int q1, Mat4 U) {
  const int b = blockIdx.y;
  float2* psi = base + (uint64_t)b * vstride;
  float2* lam = psi + (vstride / 3);
  const int lo = min(q0, q1), hi = max(q0, q1);
  const uint64_t s0 = 1ull << q0, s1 = 1ull << q1;
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nquads; p += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = insert_zero(insert_zero(p, lo), hi);
    float2* vs[2] = {psi, lam};
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      float2* s = vs[v];
      float2 a0 = s[i], a1 = s[i | s0], a2 = s[i | s1], a3 = s[i | s0 | s1];
      s[i] = cfma4(U.g + 0, a0, a1, a2, a3);
      s[i | s0] = cfma4(U.g + 4, a0, a1, a2, a3);
      s[i | s1] = cfma4(U.g + 8, a0, a1, a2, a3);
      s[i | s0 | s1] = cfma4(U.g + 12, a0, a1, a2, a3);
    }
  }
}

struct SortedQ { int pos[10]; int k; };
__global__ void k_adj_mcx(float2* __restrict__ base, uint64_t vstride, uint64_t items, SortedQ P, uint64_t cmask,
                          int t) {
  const int b = blockIdx.y;
  float2* psi = base + (uint64_t)b * vstride;
  float2* lam = psi + (vstride / 3);
  const uint64_t st = 1ull << t;
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < items; p += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i0 = insert_zeros(p, P.pos, P.k) | cmask;
    float2 a = psi[i0], c = psi[i0 | st];
    psi[i0] = c; psi[i0 | st] = a;
    a = lam[i0]; c = lam[i0 | st];
    lam[i0] = c; lam[i0 | st] = a;
  }
}

__global__ void k_adj_phase(float2* __restrict__ base, uint64_t vstride, uint64_t items, SortedQ P, uint64_t mask,
                            float2 ph, int neg) {
  const int b = blockIdx.y;
  float2* psi = base + (uint64_t)b * vstride;
  float2* lam = psi + (vstride / 3);
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < items; p += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = insert_zeros(p, P.pos, P.k) | mask;
    float2 a = psi[i], l = lam[i];
    if (neg) { psi[i] = make_float2(-a.x, -a.y); lam[i] = make_float2(-l.x, -l.y); }
    else { psi[i] = cmul_comp(a, ph); lam[i] = cmul_comp(l, ph); }
  }
}

// E_b partials: Re<psi|lam>
__global__ void k_adj_dot(const float2* __restrict__ base, uint64_t vstride, uint64_t n, uint64_t per,
                          double* __restrict__ partial) {
  const int b = blockIdx.y;
  const float2* psi = base + (uint64_t)b * vstride;
  const float2* lam = psi + (vstride / 3);
  const uint64_t i0 = (uint64_t)blockIdx.x * per, e = min(i0 + per, n);
  double acc = 0.0;
  for (uint64_t i = i0 + threadIdx.x; i < e; i += blockDim.x) {
    const float2 a = psi[i], l = lam[i];
    acc += (double)a.x * l.x + (double)a.y * l.y;
  }
  acc = block_sum(acc);
  if (threadIdx.x == 0) partial[(uint64_t)b * gridDim.x + blockIdx.x] = acc;
}

// out[b*ostride + idx] (+)= sum_x partial[b][x], fixed order
__global__ void k_adj_final(const double* __restrict__ partial, int nbx, double* __restrict__ out, int ostride,
                            int idx, int add) {
  const int b = blockIdx.x;
  double acc = 0.0;
  for (int i = threadIdx.x; i < nbx; i += blockDim.x) acc += partial[(uint64_t)b * nbx + i];
  acc = block_sum(acc);
  if (threadIdx.x == 0) {
    double* o = out + (uint64_t)b * ostride + idx;
    *o = add ? (*o + acc) : acc;
  }
}

// ------------------------------------------------------ tile passes ----
// A pass is a list of steps on a tile of 2^T amplitudes staged in shared
// memory.  A tile bit k (position) has an address column: amplitude i lies at
// the XOR of the columns of its set bits and a constant.  So X and CNOT move
// nothing: they change the constant or add one column to another (a control
// outside the tile adds a constant in the tiles where it is 1).  The first
// columns also spread the tile over the banks.
//
// Kinds of step:
//   block  three positions (forward: four) whose pending 1Q gates are fused into
//          one 2x2 matrix each (k_adj_prepare).  A thread
//          holds the amplitudes over those bits in registers; in the reverse
//          sweep psi and lambda share a matrix, packed for two-lane FMAs.
//          All parameter gates of a position's run are rotations about axes
//          that the rest of the run turns, so their gradients are combinations
//          of three sums, Im<lambda|P|psi> for P = X, Y, Z, taken before the run
//          is undone.
//   MCX (two or more controls), phase, U2: one sweep of the tile, over a table of
//          addresses that is rebuilt (with a barrier of its own) only where the
//          columns changed since the pass's last sweep: 4 layers of Toffolis, phases
//          and RXX on 8 / 12 / 20 qubits 164 / 508 / 3996 us of GPU time, 206 / 595 /
//          4484 rebuilt for every sweep.
//   store  the last: the tile goes back in the order of its columns.
enum AdjKind : int32_t { AG_BLOCK = 0, AG_MCX, AG_PHASE, AG_U2, AG_STORE };

constexpr int kAdjTileBits = 12;
constexpr int kAdjLowQubits = 4;
constexpr int kAdjOut = 8;

struct alignas(16) AdjStep {
  int32_t kind;
  int32_t mat;               // U2: Mat4 index
  uint16_t col[kAdjTileBits];  // block: columns of the thread index; others: of the tile bits (all in bytes)
  uint16_t v[4];             // block: columns of the register bits
  uint16_t c, nout;
  int32_t slot[3];           // first of a run's three sums, or -1
  uint32_t out[kAdjOut];     // controls outside the tile: qubit << 16 | constant
  uint64_t cmask;            // MCX controls / phase qubits, as a global index mask
  float2 ph;                 // phase factor (already conjugated)
  uint8_t p0, p1;            // tile positions of the targets; U2: p0 = matrix bit 0
  uint8_t neg;               // phase: negate instead of multiplying
  uint8_t gates;             // block: bit j set where position j has a matrix
  int32_t mapped;            // sweep: the addresses are those of the pass's last sweep
  uint32_t pad[4];
};
static_assert(sizeof(AdjStep) == 128, "eight 16-byte loads");

struct PassArg {
  int32_t S[kAdjTileBits];  // tile positions (global qubits), ascending
  int32_t T, bits;    // tile bits, and those of them that exist (n < T)
  int32_t gb, ge;     // steps of the pass
  int32_t nslots;     // sums of the pass's part of the sweep
  int32_t from_zero;  // forward: the tile starts as |0..0> instead of being loaded
};

__device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }

// Sums v[0..N) over the warp; returns the index of the total that this lane's
// v[0] then holds, -1 if none.  Each round passes half of the values on, so
// nine cost 12 exchanges instead of 45.
template <int N, int O>
__device__ __forceinline__ void warp_totals_round(double* v, int lane, int& base, int& end) {
  constexpr int H = (N + 1) / 2;
  const bool up = lane & O;
  if (N == 1) {
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
  } else {
#pragma unroll
    for (int k = 0; k < H; ++k) {
      const double hi = k + H < N ? v[k + H] : 0.0;
      const double keep = up ? hi : v[k], send = up ? v[k] : hi;
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, O);
    }
    if (up) base += H; else end = min(end, base + H);
  }
  if constexpr (O > 1) warp_totals_round<H, O / 2>(v, lane, base, end);
}
template <int N>
__device__ __forceinline__ int warp_totals(double (&v)[N], int lane) {
  int base = 0, end = N;
  warp_totals_round<N, 16>(v, lane, base, end);
  return base < end ? base : -1;
}

// U on the pairs of register bit J of eight packed amplitudes.
template <int J>
__device__ __forceinline__ void adj_gate(float2 (&re)[8], float2 (&im)[8], const float4* __restrict__ U) {
  // row by row, each entry twice for the two lanes: (x0, y0), (-y0, x1), (y1, -y1)
  auto lo = [](float4 q) { return make_float2(q.x, q.y); };
  auto hi = [](float4 q) { return make_float2(q.z, q.w); };
  const float4 a0 = U[0], a1 = U[1], a2 = U[2], b0 = U[3], b1 = U[4], b2 = U[5];
  const float2 g0x = lo(a0), g0y = hi(a0), m0y = lo(a1), g1x = hi(a1), g1y = lo(a2), m1y = hi(a2);
  const float2 g2x = lo(b0), g2y = hi(b0), m2y = lo(b1), g3x = hi(b1), g3y = lo(b2), m3y = hi(b2);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = ((q >> J) << (J + 1)) | (q & ((1 << J) - 1)), k = i | (1 << J);
    const float2 r0 = re[i], i0 = im[i], r1 = re[k], i1 = im[k];
    re[i] = __ffma2_rn(m1y, i1, __ffma2_rn(g1x, r1, __ffma2_rn(m0y, i0, __fmul2_rn(g0x, r0))));
    im[i] = __ffma2_rn(g1y, r1, __ffma2_rn(g1x, i1, __ffma2_rn(g0y, r0, __fmul2_rn(g0x, i0))));
    re[k] = __ffma2_rn(m3y, i1, __ffma2_rn(g3x, r1, __ffma2_rn(m2y, i0, __fmul2_rn(g2x, r0))));
    im[k] = __ffma2_rn(g3y, r1, __ffma2_rn(g3x, i1, __ffma2_rn(g2y, r0, __fmul2_rn(g2x, i0))));
  }
}

// Im<lambda|P|psi> for P = X, Y, Z on register bit J, in FP64.
template <int J>
__device__ __forceinline__ void adj_sums(const double2 (&a)[8], const double2 (&l)[8], double* s) {
  double t[2][3] = {{s[0], s[1], s[2]}, {0.0, 0.0, 0.0}};   // two chains per sum
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = ((q >> J) << (J + 1)) | (q & ((1 << J) - 1)), k = i | (1 << J);
    const double2 a0 = a[i], a1 = a[k], l0 = l[i], l1 = l[k];
    double* u = t[q & 1];
    u[0] = fma(l0.x, a1.y, fma(-l0.y, a1.x, fma(l1.x, a0.y, fma(-l1.y, a0.x, u[0]))));
    u[1] = fma(-l0.x, a1.x, fma(-l0.y, a1.y, fma(l1.x, a0.x, fma(l1.y, a0.y, u[1]))));
    u[2] = fma(l0.x, a0.y, fma(-l0.y, a0.x, fma(-l1.x, a1.y, fma(l1.y, a1.x, u[2]))));
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) s[k] = t[0][k] + t[1][k];
}

// One pass: CTA (tile, vector b).  Reverse (FWD false): psi and lambda, each
// element of the tile (psi.re, lambda.re, psi.im, lambda.im).  Forward: psi
// only, from |0..0> when P.from_zero.
//
// Bound by issue and FP64/conversion latency (16 warps per SM): a reverse block
// of three runs is 16 shared loads and stores, 32 conversions, 144 FP64 and 192
// packed FMAs per eight amplitudes; a forward block of four, 512 FMAs per 16.
// 8 vectors of 20 qubits, 200 parameters: 8 reverse passes of 226 us and 7
// forward ones of 102 us on average; one sweep of the tile per gate, with eight
// conversions per pair and parameter gate, took 9 x 493 and 8 x 237 us.
template <bool FWD>
__global__ void __launch_bounds__(kThreads, FWD ? 3 : 2)
    k_adj_pass(float2* __restrict__ base, uint64_t vstride, PassArg P, const AdjStep* __restrict__ steps,
               const float4* __restrict__ mats, int nb, const Mat4* __restrict__ u2, double* __restrict__ partial) {
  using Elem = typename std::conditional<FWD, float2, float4>::type;
  extern __shared__ __align__(16) unsigned char adj_smem[];
  constexpr uint32_t kElem = sizeof(Elem);
  constexpr int kRegs = FWD ? 4 : 3, kMat = FWD ? 2 : 6;   // a staged matrix in 16-byte words
  auto el = [&](uint32_t byte) -> Elem& { return *reinterpret_cast<Elem*>(adj_smem + byte); };
  __shared__ uint64_t dep_lo[64], dep_hi[32];   // global index of a pair of amplitudes (tile bits 1-6, 7-11)
  __shared__ uint16_t map_lo[64], map_hi[64];
  __shared__ __align__(16) uint4 next[2][8 + kRegs * kMat];   // a step and its matrices (see adj_gate)
  __shared__ double red[2][kThreads / 32][9];
  const int T = P.T, tid = threadIdx.x, lane = tid & 31;
  const uint32_t NT = 1u << T;
  const int b = blockIdx.y;
  const uint64_t tile = blockIdx.x, ntiles = gridDim.x;
  float4* psi = reinterpret_cast<float4*>(base + (uint64_t)b * vstride);
  float4* lam = reinterpret_cast<float4*>(base + (uint64_t)b * vstride + vstride / 3);
  if (tid < 96) {
    const int first = tid < 64 ? 1 : 7, x = tid < 64 ? tid : tid - 64;
    uint64_t d = 0;
    for (int k = 0; first + k < P.bits && k < 6; ++k)
      if ((x >> k) & 1) d |= 1ull << P.S[first + k];
    if (tid < 64) dep_lo[x] = d; else dep_hi[x] = d;
  }
  constexpr int kChunks = 8 + 2 * kRegs;   // by one thread each, all of warp 0
  auto step_chunk = [&](int s) -> uint4 {
    if (tid < 8) return reinterpret_cast<const uint4*>(steps + s)[tid];
    const int j = (tid - 8) >> 1;
    return reinterpret_cast<const uint4*>(mats)[(((uint64_t)s * 4 + j) * nb + b) * 2 + (tid & 1)];
  };
  auto step_put = [&](int buf, uint4 d) {
    if (FWD || tid < 8) { next[buf][tid] = d; return; }
    uint4* m = next[buf] + 8 + 3 * (tid - 8);
    const uint32_t neg = 0x80000000u;
    m[0] = make_uint4(d.x, d.x, d.y, d.y);
    m[1] = make_uint4(d.y ^ neg, d.y ^ neg, d.z, d.z);
    m[2] = make_uint4(d.w, d.w, d.w ^ neg, d.w ^ neg);
  };
  // the byte address of tile index i from `first` up, by six bits each
  auto map_build = [&](uint32_t c, int first, auto column) {
    if (tid < 128) {
      const int at = first + (tid < 64 ? 0 : 6), x = tid & 63;
      uint32_t m = tid < 64 ? c : 0;
      for (int k = 0; k < 6 && at + k < T; ++k)
        if ((x >> k) & 1) m ^= column(at + k);
      (tid < 64 ? map_lo : map_hi)[x] = (uint16_t)m;
    }
  };
  auto addr = [&](uint32_t i) -> uint32_t { return map_lo[i & 63] ^ map_hi[i >> 6]; };
  if (tid < kChunks) step_put(0, step_chunk(P.gb));
  map_build(0, 1, [&](int k) { return tile_col(k) * kElem; });
  uint64_t gbase = tile;
  for (int k = 0; k < P.bits; ++k) gbase = insert_zero(gbase, P.S[k]);
  __syncthreads();
  // amplitudes 2e and 2e + 1 of the tile are neighbours (qubit 0 is in every tile)
  auto pair_at = [&](uint32_t e) { return (gbase | dep_lo[e & 63] | dep_hi[e >> 6]) >> 1; };
  const uint32_t npairs = 1u << (P.bits - 1);
  constexpr int kLoads = 4;   // 16-byte loads in flight per thread (of each vector)
  for (uint32_t e0 = tid; e0 < NT / 2; e0 += kThreads * kLoads) {
    float4 a[kLoads], l[kLoads];
#pragma unroll
    for (int k = 0; k < kLoads; ++k) {
      const uint32_t e = e0 + kThreads * k;
      a[k] = l[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (FWD && P.from_zero) {
        if (e == 0 && gbase == 0) a[k].x = 1.f;
      } else if (e < npairs) {
        const uint64_t g = pair_at(e);
        a[k] = psi[g];
        if (!FWD) l[k] = lam[g];
      }
    }
#pragma unroll
    for (int k = 0; k < kLoads; ++k) {
      const uint32_t e = e0 + kThreads * k;
      if (e >= NT / 2) break;
      const uint32_t A = addr(e);
      if constexpr (FWD) {
        el(A) = make_float2(a[k].x, a[k].y);
        el(A ^ kElem) = make_float2(a[k].z, a[k].w);
      } else {
        el(A) = make_float4(a[k].x, l[k].x, a[k].y, l[k].y);
        el(A ^ kElem) = make_float4(a[k].z, l[k].z, a[k].w, l[k].w);
      }
    }
  }
  __syncthreads();
  for (int s = P.gb; s < P.ge; ++s) {
    const int cur = (s - P.gb) & 1;
    uint4 pre = make_uint4(0, 0, 0, 0);
    if (tid < kChunks && s + 1 < P.ge) pre = step_chunk(s + 1);
    const AdjStep& G = *reinterpret_cast<const AdjStep*>(next[cur]);
    uint32_t c = G.c;
    for (int k = 0; k < G.nout; ++k)
      if ((gbase >> (G.out[k] >> 16)) & 1) c ^= G.out[k] & 0xffffu;
    double sum[9];
    bool summed = false;
    if (G.kind == AG_BLOCK) {
      const float4* U = reinterpret_cast<const float4*>(next[cur] + 8);
      uint32_t A0 = c;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if ((tid >> j) & 1) A0 ^= G.col[j];
      uint32_t off[1 << kRegs];
      off[0] = 0;
#pragma unroll
      for (int r = 1; r < (1 << kRegs); ++r) off[r] = off[r & (r - 1)] ^ G.v[31 - __clz(r & -r)];
      const bool sums = !FWD && (G.slot[0] >= 0 || G.slot[1] >= 0 || G.slot[2] >= 0);
      if (sums) {
#pragma unroll
        for (int k = 0; k < 9; ++k) sum[k] = 0.0;
      }
      for (uint32_t g = tid; g < (NT >> kRegs); g += kThreads) {
        const uint32_t A = g & 256u ? A0 ^ G.col[8] : A0;
        if constexpr (FWD) {
          float2 w[16];
#pragma unroll
          for (int r = 0; r < 16; ++r) w[r] = el(A ^ off[r]);
          if (G.gates & 1) gate_on_bit<0>(w, U);
          if (G.gates & 2) gate_on_bit<1>(w, U + 2);
          if (G.gates & 4) gate_on_bit<2>(w, U + 4);
          if (G.gates & 8) gate_on_bit<3>(w, U + 6);
#pragma unroll
          for (int r = 0; r < 16; ++r) el(A ^ off[r]) = w[r];
        } else {
          float2 re[8], im[8];
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const float4 p = el(A ^ off[r]);
            re[r] = make_float2(p.x, p.y);
            im[r] = make_float2(p.z, p.w);
          }
          if (sums) {
            double2 a[8], l[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              a[r] = make_double2(re[r].x, im[r].x);
              l[r] = make_double2(re[r].y, im[r].y);
            }
            if (G.slot[0] >= 0) adj_sums<0>(a, l, sum);
            if (G.slot[1] >= 0) adj_sums<1>(a, l, sum + 3);
            if (G.slot[2] >= 0) adj_sums<2>(a, l, sum + 6);
          }
          if (G.gates & 1) adj_gate<0>(re, im, U);
          if (G.gates & 2) adj_gate<1>(re, im, U + 6);
          if (G.gates & 4) adj_gate<2>(re, im, U + 12);
#pragma unroll
          for (int r = 0; r < 8; ++r) el(A ^ off[r]) = make_float4(re[r].x, re[r].y, im[r].x, im[r].y);
        }
      }
      if (sums) {
        const int k = warp_totals<9>(sum, lane);
        if (k >= 0 && !(lane & 1)) red[cur][tid >> 5][k] = sum[0];
        summed = true;
      }
    } else {
      // addresses of the tile's indices (of its pairs for a store)
      if (!G.mapped) {
        map_build(c, G.kind == AG_STORE ? 1 : 0, [&](int k) { return (uint32_t)G.col[k]; });
        __syncthreads();
      }
      auto gidx = [&](uint32_t i) { return 2 * pair_at(i >> 1) | (i & 1); };
      // psi (and lambda) of an element
      auto get = [&](uint32_t x, float2 (&w)[2]) {
        if constexpr (FWD) {
          w[0] = el(x);
        } else {
          const float4 p = el(x);
          w[0] = make_float2(p.x, p.z);
          w[1] = make_float2(p.y, p.w);
        }
      };
      auto put = [&](uint32_t x, const float2 (&w)[2]) {
        if constexpr (FWD) el(x) = w[0];
        else el(x) = make_float4(w[0].x, w[1].x, w[0].y, w[1].y);
      };
      constexpr int NV = FWD ? 1 : 2;
      if (G.kind == AG_STORE) {
        for (uint32_t e = tid; e < npairs; e += kThreads) {
          const uint32_t x = addr(e);
          float2 p[2], q[2];
          get(x, p);
          get(x ^ G.col[0], q);
          const uint64_t g = pair_at(e);
          psi[g] = make_float4(p[0].x, p[0].y, q[0].x, q[0].y);
          if (!FWD) lam[g] = make_float4(p[1].x, p[1].y, q[1].x, q[1].y);
        }
      } else if (G.kind == AG_MCX) {
        const int p = G.p0;
        for (uint32_t k = tid; k < NT / 2; k += kThreads) {
          const uint32_t i = (uint32_t)insert_zero(k, p);
          if ((gidx(i) & G.cmask) != G.cmask) continue;
          const uint32_t x0 = addr(i), x1 = x0 ^ G.col[p];
          const Elem t = el(x0);
          el(x0) = el(x1);
          el(x1) = t;
        }
      } else if (G.kind == AG_PHASE) {
        const float2 ph = FWD ? conjf2(G.ph) : G.ph;
        for (uint32_t i = tid; i < NT; i += kThreads) {
          if ((gidx(i) & G.cmask) != G.cmask) continue;
          float2 w[2];
          const uint32_t x = addr(i);
          get(x, w);
#pragma unroll
          for (int k = 0; k < NV; ++k) w[k] = G.neg ? make_float2(-w[k].x, -w[k].y) : cmul_comp(w[k], ph);
          put(x, w);
        }
      } else {  // AG_U2
        Mat4 U = u2[G.mat];
        if (FWD) {
          const Mat4 D = U;
#pragma unroll
          for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int k = 0; k < 4; ++k) U.g[4 * r + k] = conjf2(D.g[4 * k + r]);
        }
        const int lo2 = min(G.p0, G.p1), hi2 = max(G.p0, G.p1);
        for (uint32_t k = tid; k < NT / 4; k += kThreads) {
          const uint32_t x0 = addr((uint32_t)insert_zero(insert_zero(k, lo2), hi2));
          const uint32_t x[4] = {x0, x0 ^ G.col[G.p0], x0 ^ G.col[G.p1], x0 ^ G.col[G.p0] ^ G.col[G.p1]};
          float2 w[4][2], o[4][2];
#pragma unroll
          for (int r = 0; r < 4; ++r) get(x[r], w[r]);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
#pragma unroll
            for (int m = 0; m < NV; ++m) o[r][m] = cfma4(U.g + 4 * r, w[0][m], w[1][m], w[2][m], w[3][m]);
            put(x[r], o[r]);
          }
        }
      }
    }
    if (tid < kChunks && s + 1 < P.ge) step_put(cur ^ 1, pre);
    __syncthreads();
    if (!FWD && summed && tid < 9 && G.slot[tid / 3] >= 0) {
      double t = 0.0;
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) t += red[cur][w][tid];
      partial[((uint64_t)b * P.nslots + G.slot[tid / 3] + tid % 3) * ntiles + tile] = t;
    }
    __syncwarp();   // the step is read above and its buffer refilled by this warp
  }
}

// A gate of a run: RX, RY or RZ by its angle, or a constant matrix.
struct AdjOp { int32_t kind, param, mat, pad; double angle; };
// A run: its place in the matrix table, its gates in the order they are applied
// (reverse: undone), the first of its gates' weights.
struct AdjRun { int32_t row, op0, op1, ref, reverse; };

struct C2 { double re[4], im[4]; };
__device__ __forceinline__ C2 c2_mul(const C2& a, const C2& b) {
  C2 c;
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const int p = 2 * x, q = p + 1;
      c.re[p + y] = a.re[p] * b.re[y] - a.im[p] * b.im[y] + a.re[q] * b.re[2 + y] - a.im[q] * b.im[2 + y];
      c.im[p + y] = a.re[p] * b.im[y] + a.im[p] * b.re[y] + a.re[q] * b.im[2 + y] + a.im[q] * b.re[2 + y];
    }
  return c;
}
__device__ __forceinline__ C2 c2_dagger(const C2& a) {
  return {{a.re[0], a.re[2], a.re[1], a.re[3]}, {-a.im[0], -a.im[2], -a.im[1], -a.im[3]}};
}

// One thread per (run, vector): the run's matrix (FP64 products, rounded once)
// and, in the reverse sweep, the axis of each parameter gate as the run's last
// state sees it.
__global__ void k_adj_prepare(const AdjRun* __restrict__ runs, int nruns, const AdjOp* __restrict__ ops,
                              const double* __restrict__ consts, const double* __restrict__ params, int nparams, int nb,
                              Mat2* __restrict__ mats, double* __restrict__ weights) {
  const uint64_t id = gtid();
  if (id >= (uint64_t)nruns * nb) return;
  const int b = (int)(id % nb);
  const AdjRun R = runs[id / nb];
  C2 V{{1, 0, 0, 1}, {0, 0, 0, 0}};   // the gates so far
  int ref = R.ref;
  for (int o = R.op0; o < R.op1; ++o) {
    const AdjOp O = ops[o];
    C2 U{{0, 0, 0, 0}, {0, 0, 0, 0}};
    if (O.mat >= 0) {
      for (int k = 0; k < 4; ++k) { U.re[k] = consts[8 * O.mat + 2 * k]; U.im[k] = consts[8 * O.mat + 2 * k + 1]; }
    } else {
      double sn, cs;
      sincos(0.5 * (O.param >= 0 ? params[(uint64_t)b * nparams + O.param] : O.angle), &sn, &cs);
      U.re[0] = U.re[3] = cs;
      if (O.kind == 1) U.im[1] = U.im[2] = -sn;
      else if (O.kind == 2) { U.re[1] = -sn; U.re[2] = sn; }
      else { U.im[0] = -sn; U.im[3] = sn; }
    }
    if (R.reverse && O.param >= 0) {
      C2 G{{0, 0, 0, 0}, {0, 0, 0, 0}};
      if (O.kind == 1) G.re[1] = G.re[2] = 1;
      else if (O.kind == 2) { G.im[1] = -1; G.im[2] = 1; }
      else { G.re[0] = 1; G.re[3] = -1; }
      const C2 A = c2_mul(c2_mul(V, G), c2_dagger(V));   // n . sigma
      double* w = weights + ((uint64_t)ref * nb + b) * 3;
      w[0] = A.re[2];
      w[1] = A.im[2];
      w[2] = A.re[0];
      ++ref;
    }
    V = R.reverse ? c2_mul(V, U) : c2_mul(U, V);
  }
  if (R.reverse) V = c2_dagger(V);
  Mat2 D;
  for (int k = 0; k < 4; ++k) D.g[k] = make_float2((float)V.re[k], (float)V.im[k]);
  mats[(uint64_t)R.row * nb + b] = D;
}

// A parameter gate: the first of its run's sums, and which weights it has.
struct AdjRef { int32_t slot, w; };

// grads[b][p] += sum over a part's gates with parameter p of its axis . (sums
// over the tiles), one warp per (p, b), in a fixed order.
__global__ void k_adj_grads(const double* __restrict__ partial, int nslots, uint64_t ntiles,
                            const int32_t* __restrict__ first, const AdjRef* __restrict__ refs,
                            const double* __restrict__ weights, int nb, double* __restrict__ grads, int nparams) {
  const int p = (int)(gtid() >> 5), lane = threadIdx.x & 31, b = blockIdx.y;
  if (p >= nparams || first[p] == first[p + 1]) return;
  double total = 0.0;
  for (int k = first[p]; k < first[p + 1]; ++k) {
    const AdjRef R = refs[k];
    const double* s = partial + ((uint64_t)b * nslots + R.slot) * ntiles;
    double x = 0.0, y = 0.0, z = 0.0;
    for (uint64_t t = lane; t < ntiles; t += 32) {
      x += s[t];
      y += s[ntiles + t];
      z += s[2 * ntiles + t];
    }
    const double* w = weights + ((uint64_t)R.w * nb + b) * 3;
    total += w[0] * warp_sum(x) + w[1] * warp_sum(y) + w[2] * warp_sum(z);
  }
  if (lane == 0) grads[(uint64_t)b * nparams + p] += total;
}

SortedQ sortedq(std::vector<int> q) {
  std::sort(q.begin(), q.end());
  SortedQ P;
  std::memset(&P, 0, sizeof(P));
  P.k = (int)q.size();
  for (int i = 0; i < P.k; ++i) P.pos[i] = q[i];
  return P;
}

using cd = std::complex<double>;

// 2x2 matrix of a rotation / U1 / DIAG1 op with parameter theta
void mat_1q(const qs_op& o, double theta, cd* m) {
  const double c = std::cos(theta / 2), s = std::sin(theta / 2);
  switch (o.kind) {
    case QS_OP_RX: m[0] = c; m[1] = cd(0, -s); m[2] = cd(0, -s); m[3] = c; break;
    case QS_OP_RY: m[0] = c; m[1] = -s; m[2] = s; m[3] = c; break;
    case QS_OP_RZ: m[0] = std::polar(1.0, -theta / 2); m[1] = 0; m[2] = 0; m[3] = std::polar(1.0, theta / 2); break;
    case QS_OP_U1: for (int i = 0; i < 4; ++i) m[i] = cd(o.m[2 * i], o.m[2 * i + 1]); break;
    case QS_OP_DIAG1: m[0] = cd(o.m[0], o.m[1]); m[1] = 0; m[2] = 0; m[3] = cd(o.m[2], o.m[3]); break;
    case QS_OP_Y: m[0] = 0; m[1] = cd(0, -1); m[2] = cd(0, 1); m[3] = 0; break;
    default: throw qs_error(QS_ERR_INVALID, "internal: not a 1Q op");
  }
}

bool adj_passes_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("QSIM_ADJ_PASSES");
    return !(e && e[0] == '0');
  }();
  return on;
}

// Bytes of partial sums held at a time.  28 qubits, 40 layers of RY and CX chains
// (1120 runs of three sums): 801 ms in two parts, 5336 in one launch per gate.
constexpr size_t kAdjPartials = 3ull << 29;

// Reverse passes [pass0, pass1) and their sums.
struct AdjPart { size_t pass0, pass1; int32_t slot0, nslots; };

bool is_1q_kind(int k) {
  return k == QS_OP_RX || k == QS_OP_RY || k == QS_OP_RZ || k == QS_OP_U1 || k == QS_OP_DIAG1 || k == QS_OP_Y;
}

// The passes of a sweep over `order` (op indices): tile qubits by list
// scheduling, steps by collecting 1Q gates per qubit until a gate needs them done.
struct AdjPlan {
  int n, T, L;
  const qs_op* ops;
  std::vector<AdjStep> steps;      // each with four rows of the matrix table
  std::vector<AdjRun> runs;
  std::vector<AdjOp> run_ops;
  std::vector<double> consts;      // constant 2x2 matrices
  std::vector<Mat4> u2s;           // U^dag (the forward kernel transposes it back)
  std::vector<AdjRef> refs;
  std::vector<int32_t> ref_param;
  int nslots = 0;
  size_t max_params = ~size_t(0);  // parameter gates of a reverse pass

  // state of the pass that is being cut into steps
  int pos[64];
  uint32_t col[kAdjTileBits], cst;
  std::vector<std::pair<int, uint32_t>> out;
  std::vector<int> pending[kAdjTileBits];
  bool reverse;
  int regs;                        // positions of a block
  uint32_t elem;                   // bytes of a tile element

  AdjStep step(int kind) {
    AdjStep G;
    std::memset(&G, 0, sizeof(G));
    G.kind = kind;
    G.c = (uint16_t)(cst * elem);
    G.slot[0] = G.slot[1] = G.slot[2] = -1;
    for (const auto& o : out)
      if (o.second) G.out[G.nout++] = (uint32_t)o.first << 16 | o.second * elem;
    for (int k = 0; k < T; ++k) G.col[k] = (uint16_t)(col[k] * elem);
    return G;
  }

  // The pending gates of up to `regs` positions as one block.
  void block(const int* which, int count) {
    int bits[4];
    bool used[kAdjTileBits] = {};
    for (int j = 0; j < count; ++j) { bits[j] = which[j]; used[which[j]] = true; }
    for (int j = count, k = T - 1; j < regs; --k)
      if (!used[k]) { bits[j++] = k; used[k] = true; }
    AdjStep G = step(AG_BLOCK);
    for (int j = 0; j < regs; ++j) G.v[j] = (uint16_t)(col[bits[j]] * elem);
    // thread bits: first those whose columns spread the lanes of one access
    // over the banks (8 elements of 16 bytes or 16 of 8)
    const uint32_t low = reverse ? 7u : 15u;
    std::vector<uint32_t> basis, lead, rest;
    for (int k = 0; k < T; ++k) {
      if (used[k]) continue;
      uint32_t x = col[k] & low;
      for (uint32_t e : basis) x = std::min(x, x ^ e);
      if (x) { basis.push_back(x); lead.push_back(col[k]); } else rest.push_back(col[k]);
    }
    std::memset(G.col, 0, sizeof(G.col));
    int j = 0;
    for (uint32_t x : lead) G.col[j++] = (uint16_t)(x * elem);
    for (uint32_t x : rest) G.col[j++] = (uint16_t)(x * elem);
    steps.push_back(G);
    AdjStep& S = steps.back();
    for (int q = 0; q < count; ++q) {
      std::vector<int>& run = pending[which[q]];
      S.gates |= 1u << q;
      AdjRun R{(int32_t)(4 * (steps.size() - 1)) + q, (int32_t)run_ops.size(), 0, (int32_t)refs.size(), reverse};
      for (int o : run) {
        run_ops.push_back(run_op(ops[o]));
        if (!reverse || ops[o].param < 0) continue;
        refs.push_back(AdjRef{nslots, (int32_t)refs.size()});
        ref_param.push_back(ops[o].param);
      }
      if ((int32_t)refs.size() > R.ref) {
        S.slot[q] = nslots;
        nslots += 3;
      }
      R.op1 = (int32_t)run_ops.size();
      runs.push_back(R);
      run.clear();
    }
  }

  AdjOp run_op(const qs_op& o) {
    AdjOp O{o.kind == QS_OP_RX ? 1 : o.kind == QS_OP_RY ? 2 : 3, o.param, -1, 0, o.m[0]};
    if (o.kind == QS_OP_RX || o.kind == QS_OP_RY || o.kind == QS_OP_RZ) return O;
    cd m[4];
    mat_1q(o, 0.0, m);
    O.param = -1;
    O.mat = (int32_t)(consts.size() / 8);
    for (const cd& x : m) { consts.push_back(x.real()); consts.push_back(x.imag()); }
    return O;
  }

  // Runs the pending gates of the tile positions in `need`; free places of a
  // block go to the positions that a later op of the pass needs first.
  void flush(uint32_t need, const std::vector<int>& cur, size_t at) {
    int which[4], count = 0;
    uint32_t taken = 0;
    auto take = [&](int p) {
      which[count++] = p;
      taken |= 1u << p;
      if (count == regs) { block(which, regs); count = 0; }
    };
    bool any = false;
    for (int p = 0; p < T; ++p)
      if (((need >> p) & 1) && !pending[p].empty()) { take(p); any = true; }
    if (!any || count == 0) return;
    uint32_t open = 0;   // positions that get more gates before they are needed
    for (size_t k = at; k < cur.size() && count > 0; ++k) {
      const qs_op& o = ops[cur[k]];
      for (int q = 0; q < o.nq && count > 0; ++q) {
        const int p = pos[o.q[q]];
        if (p < 0) continue;
        if (is_1q_kind(o.kind)) open |= 1u << p;
        else if (!((open | taken) >> p & 1) && !pending[p].empty()) take(p);
      }
    }
    for (int p = 0; p < T && count > 0; ++p)
      if (!((open | taken) >> p & 1) && !pending[p].empty()) take(p);
    if (count) block(which, count);
  }

  void pass(uint64_t S, const std::vector<int>& cur, std::vector<PassArg>& passes) {
    PassArg P;
    std::memset(&P, 0, sizeof(P));
    P.T = T;
    P.bits = std::min(n, T);
    std::fill(pos, pos + 64, -1);
    int k = 0;
    for (int q = 0; q < n; ++q)
      if ((S >> q) & 1) { P.S[k] = q; pos[q] = k++; }
    for (int j = 0; j < T; ++j) col[j] = tile_col(j);
    cst = 0;
    out.clear();
    const int slot0 = nslots;
    P.gb = (int)steps.size();
    int swept = -1;   // the pass's last sweep
    for (size_t at = 0; at < cur.size(); ++at) {
      const int i = cur[at];
      const qs_op& o = ops[i];
      if (is_1q_kind(o.kind)) {
        pending[pos[o.q[0]]].push_back(i);
        continue;
      }
      // an X controlled by its own target never acts
      if (o.kind == QS_OP_MCX && std::find(o.q, o.q + o.nq - 1, o.q[o.nq - 1]) != o.q + o.nq - 1) continue;
      uint32_t need = 0;
      for (int q = 0; q < o.nq; ++q)
        if (pos[o.q[q]] >= 0) need |= 1u << pos[o.q[q]];
      flush(need, cur, at + 1);
      if (o.kind == QS_OP_MCX && o.nq <= 2) {
        const int t = pos[o.q[o.nq - 1]], c = o.nq == 2 ? pos[o.q[0]] : -1;
        if (o.nq == 1) { cst ^= col[t]; continue; }
        if (c >= 0) { col[c] ^= col[t]; continue; }
        size_t e = 0;
        while (e < out.size() && out[e].first != o.q[0]) ++e;
        if (e == out.size() && e < (size_t)kAdjOut) out.push_back({o.q[0], 0u});
        if (e < out.size()) { out[e].second ^= col[t]; continue; }
        // more controls outside the tile than a step holds: a sweep
      }
      AdjStep G = step(o.kind == QS_OP_MCX ? AG_MCX : o.kind == QS_OP_MCPHASE ? AG_PHASE : AG_U2);
      if (o.kind == QS_OP_MCX) {
        G.p0 = (uint8_t)pos[o.q[o.nq - 1]];
        for (int q = 0; q + 1 < o.nq; ++q) G.cmask |= 1ull << o.q[q];
      } else if (o.kind == QS_OP_MCPHASE) {
        for (int q = 0; q < o.nq; ++q) G.cmask |= 1ull << o.q[q];
        G.neg = (o.m[0] == -1.0 && o.m[1] == 0.0) ? 1 : 0;
        G.ph = make_float2((float)o.m[0], (float)-o.m[1]);
      } else {
        G.p0 = (uint8_t)pos[o.q[0]];
        G.p1 = (uint8_t)pos[o.q[1]];
        G.mat = (int)u2s.size();
        Mat4 U;
        for (int r = 0; r < 4; ++r)
          for (int q = 0; q < 4; ++q)
            U.g[4 * r + q] = make_float2((float)o.m[2 * (4 * q + r)], (float)-o.m[2 * (4 * q + r) + 1]);
        u2s.push_back(U);
      }
      if (swept >= 0) {
        const AdjStep& W = steps[swept];
        G.mapped = G.c == W.c && G.nout == W.nout && !std::memcmp(G.col, W.col, sizeof(G.col)) &&
                   !std::memcmp(G.out, W.out, sizeof(G.out));
      }
      swept = (int)steps.size();
      steps.push_back(G);
    }
    int which[4], count = 0;
    for (int p = 0; p < T; ++p) {
      if (pending[p].empty()) continue;
      which[count++] = p;
      if (count == regs) { block(which, regs); count = 0; }
    }
    if (count) block(which, count);
    steps.push_back(step(AG_STORE));
    P.ge = (int)steps.size();
    P.nslots = nslots - slot0;
    passes.push_back(P);
  }

  // List scheduling: an op is ready when it is the next op of the order on
  // every qubit it touches (ops on disjoint qubits commute, and so do their
  // contributions to the gradient); a pass keeps taking ready ops whose targets
  // are in its tile, and adds the targets of the earliest ready op to the tile
  // while room is left.
  void sweep(const std::vector<int>& order, bool rev, std::vector<PassArg>& passes) {
    reverse = rev;
    regs = rev ? 3 : 4;
    elem = rev ? sizeof(float4) : sizeof(float2);
    const int m = (int)order.size(), bits = std::min(n, T);
    std::vector<uint64_t> touch(m), targ(m);
    std::vector<std::vector<int>> per_q(n);   // positions in `order` touching each qubit
    for (int k = 0; k < m; ++k) {
      const qs_op& o = ops[order[k]];
      for (int q = 0; q < o.nq; ++q) {
        touch[k] |= 1ull << o.q[q];
        per_q[o.q[q]].push_back(k);
      }
      if (is_1q_kind(o.kind)) targ[k] = 1ull << o.q[0];
      else if (o.kind == QS_OP_MCX) targ[k] = 1ull << o.q[o.nq - 1];
      else if (o.kind == QS_OP_U2) targ[k] = 1ull << o.q[0] | 1ull << o.q[1];
    }
    std::vector<size_t> head(n, 0);   // next unscheduled position per qubit
    std::vector<char> done(m, 0);
    auto ready = [&](int k) {
      for (uint64_t t = touch[k]; t; t &= t - 1) {
        const int q = __builtin_ctzll(t);
        if (per_q[q][head[q]] != k) return false;
      }
      return true;
    };
    const uint64_t lows = (1ull << (bits == n ? n : L)) - 1;
    uint64_t S = lows;
    std::vector<int> cur;
    size_t params = 0;   // parameter gates in cur
    auto close = [&]() {
      params = 0;
      for (int q = 0; __builtin_popcountll(S) < bits && q < n; ++q) S |= 1ull << q;  // fill the tile
      // back in the order of the sweep (it respects every dependency): taken as
      // the tile grew, a layer's gates would be scattered over many blocks
      std::sort(cur.begin(), cur.end());
      for (int& k : cur) k = order[k];
      if (!cur.empty()) pass(S, cur, passes);
      cur.clear();
      S = lows;
    };
    int remaining = m, first = 0;
    while (remaining > 0) {
      bool progress = true;
      while (progress) {
        progress = false;
        for (int k = first; k < m; ++k) {
          if (done[k] || (targ[k] & ~S) || !ready(k)) continue;
          done[k] = 1;
          --remaining;
          const qs_op& o = ops[order[k]];   // a qubit may be listed twice
          for (int q = 0; q < o.nq; ++q) ++head[o.q[q]];
          cur.push_back(k);
          progress = true;
          if (rev && o.param >= 0 && ++params >= max_params) close();
        }
        while (first < m && done[first]) ++first;
      }
      if (remaining == 0) break;
      // widen the tile with the earliest ready op's targets, or close the pass
      int pick = first;
      while (done[pick] || !ready(pick)) ++pick;
      if (__builtin_popcountll(S | targ[pick]) <= bits) S |= targ[pick];
      else close();
    }
    close();
  }
};

}  // namespace

extern "C" int qs_adjoint_gradient(qs_handle_t h, int n, const qs_op* ops, int nops, int nparams,
                                   const double* params, int nb, const uint64_t* xm, const uint64_t* zm,
                                   const double* coefs, int nterms, void* work, double* energies, double* grads) {
  QS_REQUIRE_HANDLE(h);
  qs_batch_plan_t fwd = nullptr;
  void* dbuf = nullptr;
  void* pbuf = nullptr;
  QS_API_BEGIN
  qs_check_state(work, n);
  QS_CHECK_ARG(nb >= 1 && nb <= 65535, "n_batch must be in [1, 65535]");
  QS_CHECK_ARG(nparams >= 0 && (nparams == 0 || params), "bad params");
  QS_CHECK_ARG(nops >= 1 && ops, "need at least one op");
  QS_CHECK_ARG(nterms >= 1 && nterms <= 1024, "n_terms must be in [1, 1024]");
  QS_CHECK_ARG(energies && grads, "null output pointers");
  const uint64_t N = 1ull << n;
  const uint64_t vstride = 3 * N;
  for (int i = 0; i < nops; ++i)
    if (ops[i].param >= nparams) throw qs_error(QS_ERR_INVALID, "op param index out of range");

  for (int i = 0; i < nops; ++i) {
    const qs_op& o = ops[i];
    if (o.param >= 0 && is_1q_kind(o.kind))
      QS_CHECK_ARG(o.kind == QS_OP_RX || o.kind == QS_OP_RY || o.kind == QS_OP_RZ,
                   "only RX/RY/RZ ops may carry a parameter");
    QS_CHECK_ARG(is_1q_kind(o.kind) || o.kind == QS_OP_MCX || o.kind == QS_OP_MCPHASE || o.kind == QS_OP_U2,
                 "op kind not supported by the adjoint sweep");
    QS_CHECK_ARG(o.nq >= 1 && o.nq <= 8, "bad qubit count");
    for (int q = 0; q < o.nq; ++q) qs_check_qubit(o.q[q], n, "op");
  }
  // Tiles of at least the register bits of a block; the low qubits in every
  // tile make its runs of global memory whole 128-byte lines.
  const int T = std::max(4, std::min(n, kAdjTileBits));
  const uint64_t ntiles = 1ull << std::max(0, n - T);
  AdjPlan plan{n, T, std::min(n, kAdjLowQubits), ops};
  std::vector<PassArg> fpasses, rpasses;
  std::vector<AdjPart> parts;
  size_t part_slots = 1;
  const bool use_passes = adj_passes_enabled();
  if (use_passes) {
    std::vector<int> order(nops);
    for (int i = 0; i < nops; ++i) order[i] = i;
    plan.sweep(order, false, fpasses);
    std::reverse(order.begin(), order.end());
    // At most three sums per parameter gate, each an FP64 partial per vector and
    // tile.  The reverse passes are run in parts of at most kAdjPartials of them,
    // whose gradients are added up before the next part writes its own.
    plan.max_params = std::max<size_t>(1, kAdjPartials / (3 * sizeof(double) * nb * ntiles));
    plan.sweep(order, true, rpasses);
    fpasses[0].from_zero = 1;
    const size_t most = std::max<size_t>(3, kAdjPartials / (sizeof(double) * nb * ntiles));
    int32_t slot0 = 0;
    for (size_t k = 0; k < rpasses.size(); ++k) {
      const PassArg& P = rpasses[k];
      if (parts.empty()) parts.push_back({0, 0, 0, 0});
      else if ((size_t)(parts.back().nslots + P.nslots) > most) parts.push_back({k, k, slot0, 0});
      parts.back().pass1 = k + 1;
      parts.back().nslots += P.nslots;
      slot0 += P.nslots;
    }
    for (const AdjPart& A : parts) {
      part_slots = std::max(part_slots, (size_t)A.nslots);
      for (size_t k = A.pass0; k < A.pass1; ++k) rpasses[k].nslots = A.nslots;
    }
  }

  // device buffer: grads [nb][nparams] | energies [nb] | partial [nb][256] | U^dag table of the per-gate sweep
  const size_t ng = (size_t)nb * std::max(nparams, 1);
  const Slice sl = slice(N / 2);
  const Slice sd = slice(N);
  const int nbx = std::max(sl.nbx, sd.nbx);
  std::vector<Mat2> udag(use_passes ? 0 : (size_t)nb * nops);
  const size_t bytes = sizeof(double) * (ng + nb + (size_t)nb * nbx) + sizeof(Mat2) * udag.size() + 64;
  QS_CUDA(cudaMallocAsync(&dbuf, bytes, h->stream));
  double* d_grads = (double*)dbuf;
  double* d_energy = d_grads + ng;
  double* d_part = d_energy + nb;
  Mat2* d_udag = (Mat2*)(((uintptr_t)(d_part + (size_t)nb * nbx) + 15) & ~uintptr_t(15));
  QS_CUDA(cudaMemsetAsync(d_grads, 0, sizeof(double) * ng, h->stream));
  for (int i = 0; i < nops && !use_passes; ++i) {
    if (!is_1q_kind(ops[i].kind)) continue;
    for (int b = 0; b < nb; ++b) {
      cd m[4];
      mat_1q(ops[i], ops[i].param >= 0 ? params[(size_t)b * nparams + ops[i].param] : ops[i].m[0], m);
      for (int k = 0; k < 4; ++k) {   // conjugate transpose
        const cd x = m[2 * (k & 1) + (k >> 1)];
        udag[(size_t)i * nb + b].g[k] = make_float2((float)x.real(), (float)-x.imag());
      }
    }
  }
  if (!udag.empty())
    QS_CUDA(cudaMemcpyAsync(d_udag, udag.data(), sizeof(Mat2) * udag.size(), cudaMemcpyHostToDevice, h->stream));

  AdjStep* d_steps = nullptr;
  float4* d_mats = nullptr;
  Mat4* d_u2 = nullptr;
  AdjRef* d_refs = nullptr;
  int32_t* d_first = nullptr;
  double *d_weights = nullptr, *d_parts = nullptr;
  const size_t pass_smem[2] = {sizeof(float2) << T, sizeof(float4) << T};
  if (use_passes) {
    // the gates of each parameter, part by part, in the order of the sweep
    const size_t row = (size_t)nparams + 1;
    std::vector<int32_t> pfirst(parts.size() * row, 0);
    std::vector<AdjRef> refs(plan.refs.size());
    size_t r = 0;
    for (size_t k = 0; k < parts.size(); ++k) {
      int32_t* f = pfirst.data() + k * row;
      const size_t r0 = r;
      for (; r < refs.size() && plan.refs[r].slot < parts[k].slot0 + parts[k].nslots; ++r) ++f[plan.ref_param[r] + 1];
      f[0] = (int32_t)r0;
      for (int p = 0; p < nparams; ++p) f[p + 1] += f[p];
      std::vector<int32_t> fill(f, f + nparams);
      for (size_t q = r0; q < r; ++q) {
        AdjRef R = plan.refs[q];
        R.slot -= parts[k].slot0;
        refs[fill[plan.ref_param[q]]++] = R;
      }
    }
    std::vector<char> host;
    size_t off[8];
    auto put = [&](int k, const void* d, size_t size) {
      off[k] = host.size();
      host.resize((host.size() + size + 255) & ~size_t(255));
      if (size) std::memcpy(host.data() + off[k], d, size);
    };
    put(0, plan.steps.data(), plan.steps.size() * sizeof(AdjStep));
    put(1, plan.runs.data(), plan.runs.size() * sizeof(AdjRun));
    put(2, plan.u2s.data(), plan.u2s.size() * sizeof(Mat4));
    put(3, refs.data(), refs.size() * sizeof(AdjRef));
    put(4, pfirst.data(), pfirst.size() * sizeof(int32_t));
    put(5, plan.run_ops.data(), plan.run_ops.size() * sizeof(AdjOp));
    put(6, plan.consts.data(), plan.consts.size() * sizeof(double));
    put(7, params, sizeof(double) * (size_t)nb * nparams);
    const size_t npartials = (size_t)nb * part_slots * ntiles, nmats = plan.steps.size() * 4 * nb;
    QS_CUDA(cudaMallocAsync(&pbuf, host.size() + sizeof(Mat2) * nmats +
                            sizeof(double) * (npartials + 3 * (size_t)nb * refs.size()), h->stream));
    char* pc = static_cast<char*>(pbuf);
    d_steps = reinterpret_cast<AdjStep*>(pc + off[0]);
    d_mats = reinterpret_cast<float4*>(pc + host.size());
    d_u2 = reinterpret_cast<Mat4*>(pc + off[2]);
    d_refs = reinterpret_cast<AdjRef*>(pc + off[3]);
    d_first = reinterpret_cast<int32_t*>(pc + off[4]);
    d_parts = reinterpret_cast<double*>(pc + host.size() + sizeof(Mat2) * nmats);
    d_weights = d_parts + npartials;
    QS_CUDA(cudaMemcpyAsync(pc, host.data(), host.size(), cudaMemcpyHostToDevice, h->stream));
    const int nruns = (int)plan.runs.size();
    if (nruns) {
      k_adj_prepare<<<(unsigned)(((uint64_t)nruns * nb + 127) / 128), 128, 0, h->stream>>>(
          reinterpret_cast<AdjRun*>(pc + off[1]), nruns, reinterpret_cast<AdjOp*>(pc + off[5]),
          reinterpret_cast<double*>(pc + off[6]), reinterpret_cast<double*>(pc + off[7]), nparams, nb, (Mat2*)d_mats,
          d_weights);
      qs_after_launch(h, "k_adj_prepare");
    }
    qs_smem_limit(h, (const void*)k_adj_pass<true>, sizeof(float2) << kAdjTileBits);
    qs_smem_limit(h, (const void*)k_adj_pass<false>, sizeof(float4) << kAdjTileBits);
  }

  // ---- forward
  if (use_passes) {
    for (const PassArg& P : fpasses) {
      k_adj_pass<true><<<dim3((unsigned)ntiles, nb), kThreads, pass_smem[0], h->stream>>>(
          (float2*)work, vstride, P, d_steps, d_mats, nb, d_u2, nullptr);
      qs_after_launch(h, "k_adj_pass");
    }
  } else {
    // one circuit per vector, params substituted, through the batch planner
    std::vector<qs_op> all((size_t)nops * nb);
    std::vector<int64_t> ooff(nb + 1), soff(nb);
    std::vector<int32_t> widths(nb, n);
    for (int b = 0; b < nb; ++b) {
      ooff[b] = (int64_t)b * nops;
      soff[b] = (int64_t)(b * vstride);
      for (int i = 0; i < nops; ++i) {
        qs_op o = ops[i];
        if (o.param >= 0) o.m[0] = params[(size_t)b * nparams + o.param];
        all[(size_t)b * nops + i] = o;
      }
    }
    ooff[nb] = (int64_t)nops * nb;
    int rc = qs_batch_plan_create(h, nb, widths.data(), ooff.data(), all.data(), soff.data(), &fwd);
    if (rc != QS_OK) throw qs_error(rc, h->err);
    rc = qs_batch_plan_execute(h, fwd, work);
    if (rc != QS_OK) throw qs_error(rc, h->err);
  }

  // ---- lam = H psi, E = Re<psi|lam>
  {
    qs_pauli_apply(h, (const float2*)work, (float2*)work + N, vstride, nb, n, xm, zm, coefs, nterms);
    k_adj_dot<<<dim3(sd.nbx, nb), kThreads, 0, h->stream>>>((const float2*)work, vstride, N, sd.per, d_part);
    qs_after_launch(h, "k_adj_dot");
    k_adj_final<<<nb, kThreads, 0, h->stream>>>(d_part, sd.nbx, d_energy, 1, 0, 0);
    qs_after_launch(h, "k_adj_final");
  }

  // ---- reverse sweep
  if (use_passes) {
    for (size_t k = 0; k < parts.size(); ++k) {
      // the steps number the sums over all parts: the part's first is at the buffer's start
      double* part0 = reinterpret_cast<double*>((uintptr_t)d_parts - sizeof(double) * ntiles * parts[k].slot0);
      for (size_t q = parts[k].pass0; q < parts[k].pass1; ++q) {
        k_adj_pass<false><<<dim3((unsigned)ntiles, nb), kThreads, pass_smem[1], h->stream>>>(
            (float2*)work, vstride, rpasses[q], d_steps, d_mats, nb, d_u2, part0);
        qs_after_launch(h, "k_adj_pass");
      }
      if (parts[k].nslots > 0) {
        k_adj_grads<<<dim3((unsigned)((nparams + 3) / 4), nb), 128, 0, h->stream>>>(
            d_parts, parts[k].nslots, ntiles, d_first + k * (nparams + 1), d_refs, d_weights, nb, d_grads, nparams);
        qs_after_launch(h, "k_adj_grads");
      }
    }
  } else
  for (int i = nops - 1; i >= 0; --i) {
    const qs_op& o = ops[i];
    if (is_1q_kind(o.kind)) {
      const int t = o.q[0];
      int gk = 0;
      if (o.param >= 0) gk = o.kind == QS_OP_RX ? 1 : o.kind == QS_OP_RY ? 2 : o.kind == QS_OP_RZ ? 3 : 0;
      QS_CHECK_ARG(o.param < 0 || gk != 0, "only RX/RY/RZ ops may carry a parameter");
      k_adj_1q<<<dim3(sl.nbx, nb), kThreads, 0, h->stream>>>((float2*)work, vstride, N / 2, t,
                                                              d_udag + (size_t)i * nb, gk, sl.per, d_part);
      qs_after_launch(h, "k_adj_1q");
      if (gk) {
        k_adj_final<<<nb, kThreads, 0, h->stream>>>(d_part, sl.nbx, d_grads, nparams, o.param, 1);
        qs_after_launch(h, "k_adj_final");
      }
    } else if (o.kind == QS_OP_MCX) {
      std::vector<int> all_q(o.q, o.q + o.nq);
      uint64_t cmask = 0;
      for (int k = 0; k + 1 < o.nq; ++k) cmask |= 1ull << o.q[k];
      const uint64_t items = N >> o.nq;
      dim3 grid((unsigned)std::max<uint64_t>(1, std::min<uint64_t>((items + kThreads - 1) / kThreads, 64)), nb);
      k_adj_mcx<<<grid, kThreads, 0, h->stream>>>((float2*)work, vstride, items, sortedq(all_q), cmask, o.q[o.nq - 1]);
      qs_after_launch(h, "k_adj_mcx");
    } else if (o.kind == QS_OP_MCPHASE) {
      std::vector<int> all_q(o.q, o.q + o.nq);
      uint64_t mask = 0;
      for (int k = 0; k < o.nq; ++k) mask |= 1ull << o.q[k];
      const uint64_t items = N >> o.nq;
      const bool neg = (o.m[0] == -1.0 && o.m[1] == 0.0);
      dim3 grid((unsigned)std::max<uint64_t>(1, std::min<uint64_t>((items + kThreads - 1) / kThreads, 64)), nb);
      k_adj_phase<<<grid, kThreads, 0, h->stream>>>((float2*)work, vstride, items, sortedq(all_q), mask,
                                                     make_float2((float)o.m[0], (float)-o.m[1]), neg ? 1 : 0);
      qs_after_launch(h, "k_adj_phase");
    } else if (o.kind == QS_OP_U2) {
      Mat4 U;
      for (int r = 0; r < 4; ++r)
        for (int c = 0; c < 4; ++c)
          U.g[4 * r + c] = make_float2((float)o.m[2 * (4 * c + r)], (float)-o.m[2 * (4 * c + r) + 1]);
      const uint64_t items = N >> 2;
      dim3 grid((unsigned)std::max<uint64_t>(1, std::min<uint64_t>((items + kThreads - 1) / kThreads, 64)), nb);
      k_adj_2q<<<grid, kThreads, 0, h->stream>>>((float2*)work, vstride, items, o.q[0], o.q[1], U);
      qs_after_launch(h, "k_adj_2q");
    } else {
      throw qs_error(QS_ERR_INVALID, "op kind not supported by the adjoint sweep");
    }
  }
  QS_CUDA(cudaMemcpyAsync(grads, d_grads, sizeof(double) * (size_t)nb * nparams, cudaMemcpyDeviceToHost, h->stream));
  QS_CUDA(cudaMemcpyAsync(energies, d_energy, sizeof(double) * nb, cudaMemcpyDeviceToHost, h->stream));
  QS_CUDA(cudaFreeAsync(dbuf, h->stream));
  dbuf = nullptr;
  if (pbuf) QS_CUDA(cudaFreeAsync(pbuf, h->stream));
  pbuf = nullptr;
  QS_CUDA(cudaStreamSynchronize(h->stream));
  qs_batch_plan_destroy(fwd);
  fwd = nullptr;
  return QS_OK;
  }
  catch (const qs_error& e) {
    h->err = e.what();
    cudaStreamSynchronize(h->stream);
    if (dbuf) cudaFreeAsync(dbuf, h->stream);
    if (pbuf) cudaFreeAsync(pbuf, h->stream);
    if (fwd) qs_batch_plan_destroy(fwd);
    return e.code;
  }
  catch (const std::exception& e) {
    h->err = e.what();
    cudaStreamSynchronize(h->stream);
    if (dbuf) cudaFreeAsync(dbuf, h->stream);
    if (pbuf) cudaFreeAsync(pbuf, h->stream);
    if (fwd) qs_batch_plan_destroy(fwd);
    return QS_ERR_INVALID;
  }
}
