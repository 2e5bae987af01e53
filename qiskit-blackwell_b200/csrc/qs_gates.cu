// qs_gates.cu — one-gate-per-launch kernels (the reference's per-op API).
//
// Every kernel streams the state in place with 64-bit indices and grid-stride
// loops sized to the SM count.  Wherever the touched amplitudes come in
// adjacent pairs the kernels use 128-bit accesses (two complex64 per float4).
// Dense gates use the compensated Dot2 evaluation (qs_common.cuh); diagonal
// gates the compensated Kahan complex product; X/CNOT/Toffoli/SWAP/Z/CZ are
// exact moves or negations.
#include "qs_api.h"
#include "qs_common.cuh"
#include <algorithm>
#include <cstdlib>

using namespace qs;

namespace {

struct G2 { float2 g[4]; };
struct G4 { float2 g[16]; };
struct Sorted { int pos[12]; int k; };

constexpr int kThreads = 256;

// Every kernel here is launched with programmatic dependent launch
// (qs_launch_pdl) and begins with pdl_begin().

// ------------------------------------------------------------ init --------
__global__ void k_state_init(float4* __restrict__ s4, uint64_t nvec, uint64_t index) {
  pdl_begin();
  for (uint64_t i = gtid(); i < nvec; i += gstride()) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if ((index >> 1) == i) { if (index & 1) v.z = 1.f; else v.x = 1.f; }
    s4[i] = v;
  }
}

// states back to back, each of 2^n amplitudes: amplitude 0 of each is 1.
__global__ void k_state_init_batched(float4* __restrict__ s4, uint64_t nvec, int n) {
  pdl_begin();
  uint64_t mask = (1ull << n) - 1ull;
  for (uint64_t i = gtid(); i < nvec; i += gstride()) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (((2 * i) & mask) == 0) v.x = 1.f;
    s4[i] = v;
  }
}

// ------------------------------------------------------------- 1Q ---------
__device__ __forceinline__ void apply2(const G2& G, float2& a0, float2& a1) {
  float2 r0[2] = {G.g[0], G.g[1]}, r1[2] = {G.g[2], G.g[3]}, v[2] = {a0, a1};
  float2 n0 = cdot_comp<2>(r0, v);
  float2 n1 = cdot_comp<2>(r1, v);
  a0 = n0; a1 = n1;
}

// A gate given by value, or read by every thread from device memory when gd
// is not null (callers whose matrix lives in a device tensor, so that no
// host copy and no stream synchronisation is needed).
__device__ __forceinline__ G2 gate2(const G2& G, const float2* __restrict__ gd) {
  if (!gd) return G;
  G2 R;
#pragma unroll
  for (int i = 0; i < 4; ++i) R.g[i] = gd[i];
  return R;
}

// target 0: the pair is one float4.
__global__ void k_1q_t0(float2* __restrict__ s, uint64_t npairs, G2 G0, const float2* __restrict__ gd) {
  pdl_begin();
  const G2 G = gate2(G0, gd);
  for (uint64_t p = gtid(); p < npairs; p += gstride()) {
    float4 v = ld4(s + 2 * p);
    float2 a0 = lo2(v), a1 = hi2(v);
    apply2(G, a0, a1);
    st4(s + 2 * p, a0, a1);
  }
}

// target t >= 1: two neighbouring pairs per thread, two float4 accesses.
__global__ void k_1q_tn(float2* __restrict__ s, uint64_t nitems, int t, G2 G0, const float2* __restrict__ gd) {
  pdl_begin();
  const G2 G = gate2(G0, gd);
  const uint64_t st = 1ull << t;
  for (uint64_t it = gtid(); it < nitems; it += gstride()) {
    uint64_t i0 = insert_zero(2 * it, t);
    float4 v0 = ld4(s + i0), v1 = ld4(s + i0 + st);
    float2 a0 = lo2(v0), b0 = hi2(v0), a1 = lo2(v1), b1 = hi2(v1);
    apply2(G, a0, a1);
    apply2(G, b0, b1);
    st4(s + i0, a0, b0);
    st4(s + i0 + st, a1, b1);
  }
}

// K <= 12 single-qubit gates whose matrices and targets are device arrays,
// applied in one launch (the device-tensor form of apply_gates_fused: no host
// copy of the gates, no stream synchronisation).  A CTA stages a tile of
// 2^T amplitudes (T = min(n, 12)) whose qubits are the gates' distinct
// targets and the lowest other qubits, applies the gates to the tile in
// shared memory as an FMA chain per output (each FMA rounds once; the
// single-gate kernels' compensated Dot2 costs four times the arithmetic),
// and writes the tile back.  Gates on different qubits commute, so the gates
// are applied in groups on distinct tile positions, each gate after every
// earlier gate on its own qubit: a thread holds the amplitudes that a group
// mixes in registers, one shared-memory sweep and barrier per group instead of
// per gate.  A target outside [0, n) makes every CTA return before it writes
// (bit 16 of the status word).
//
// This kernel: states below 12 qubits, one CTA whose tile is the state, groups of
// two.  A group takes at most one position below 5 from 10 qubits on, which keeps a
// warp's shared-memory accesses within two-way bank conflicts.  Bound by latency (one
// round trip, thread 0's grouping, a sweep and a barrier per group): ten gates on 10
// qubits 5.3 us of GPU time, 7.0 with the tables of a kernel for wider states.
constexpr int kFusedMax = 12;
constexpr int kFusedGroup = 2;
constexpr int kFusedThreads = 512;

// One sweep of a group of G gates over the tile: gate b of the group (matrix
// M[b], tile position pos[b]) acts on register bit b of each thread's 2^G
// amplitudes; srt = the group's positions ascending.
template <int G>
__device__ __forceinline__ void fused_group_sweep(float2* __restrict__ tile, uint32_t tsize, const int* gidx,
                                                  const int* srt_s, const G2* sg, const int* targets) {
  int pos[G], srt[G];
  G2 M[G];
#pragma unroll
  for (int b = 0; b < G; ++b) {
    pos[b] = targets[gidx[b]];
    M[b] = sg[gidx[b]];
    srt[b] = srt_s[b];
  }
  uint32_t off[1 << G];
#pragma unroll
  for (int c = 0; c < (1 << G); ++c) {
    uint32_t o = 0;
#pragma unroll
    for (int b = 0; b < G; ++b)
      if ((c >> b) & 1) o |= 1u << pos[b];
    off[c] = o;
  }
  const uint32_t nitems = tsize >> G;
  for (uint32_t j = threadIdx.x; j < nitems; j += blockDim.x) {
    uint32_t base = j;
#pragma unroll
    for (int b = 0; b < G; ++b) base = (uint32_t)insert_zero(base, srt[b]);
    float2 a[1 << G];
#pragma unroll
    for (int c = 0; c < (1 << G); ++c) a[c] = tile[base | off[c]];
#pragma unroll
    for (int b = 0; b < G; ++b) {
#pragma unroll
      for (int c = 0; c < (1 << G); ++c) {
        if ((c >> b) & 1) continue;
        const int c1 = c | (1 << b);
        const float2 x0 = a[c], x1 = a[c1];
        a[c] = cfma2(M[b].g[0], x0, M[b].g[1], x1);
        a[c1] = cfma2(M[b].g[2], x0, M[b].g[3], x1);
      }
    }
#pragma unroll
    for (int c = 0; c < (1 << G); ++c) tile[base | off[c]] = a[c];
  }
}
__global__ void __launch_bounds__(kFusedThreads, 2) k_fused1q_dev(float2* __restrict__ s, int n, const float2* __restrict__ gates,
                                                          const int32_t* __restrict__ targets, int K,
                                                          uint32_t* status) {
  pdl_begin();
  extern __shared__ float2 tile[];
  __shared__ G2 sg[kFusedMax];
  __shared__ int st[kFusedMax];                 // targets, which are the tile positions
  __shared__ int gidx[kFusedMax][kFusedGroup];  // groups: gate indices, application order
  __shared__ int gsrt[kFusedMax][kFusedGroup];  // groups: tile positions ascending
  __shared__ int gsize[kFusedMax];
  __shared__ int s_ngroups;                     // -1: a target is out of range
  // one round trip for the gates' matrices, the targets and the state; then
  // thread 0 groups the gates from shared memory
  if ((int)threadIdx.x < K) st[threadIdx.x] = targets[threadIdx.x];
  if ((int)threadIdx.x < 4 * K) sg[threadIdx.x >> 2].g[threadIdx.x & 3] = gates[threadIdx.x];
  const uint32_t tsize = 1u << n;
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < tsize; i += kFusedThreads) tile[i] = s[i];
  __syncthreads();
  if (threadIdx.x == 0) {
    // thread 0 alone, while the CTA waits at the barrier: the targets live in
    // registers (loops unrolled over kFusedMax), so the setup costs no
    // shared-memory round trips
    int tg[kFusedMax];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < kFusedMax; ++k) {
      tg[k] = k < K ? st[k] : 0;
      if (tg[k] < 0 || tg[k] >= n) ok = false;
    }
    int ng = ok ? 0 : -1;
    if (ok) {
      uint32_t same[kFusedMax];  // earlier gates on the same position
#pragma unroll
      for (int k = 0; k < kFusedMax; ++k) {
        same[k] = 0;
#pragma unroll
        for (int k2 = 0; k2 < k; ++k2)
          if (tg[k2] == tg[k]) same[k] |= 1u << k2;
      }
      // groups: scan the unscheduled gates in order and take gate k unless
      // an earlier unscheduled gate (in this group or later) has its
      // position, the group is full, or it would be a second low position
      const int lowlim = n >= 10 ? 5 : 0;
      const uint32_t all = (1u << K) - 1u;
      for (uint32_t done = 0; done != all; ++ng) {
        int cnt = 0;
        uint32_t used = 0, pick = 0;
        bool low = false;
#pragma unroll
        for (int k = 0; k < kFusedMax; ++k) {
          const int p = tg[k];
          if (k < K && cnt < kFusedGroup && !((done >> k) & 1u) && !(same[k] & ~done) && !(p < lowlim && low)) {
            gidx[ng][cnt++] = k;
            used |= 1u << p;
            pick |= 1u << k;
            if (p < lowlim) low = true;
          }
        }
        done |= pick;
        uint32_t r = used;
        for (int j = 0; r != 0; ++j, r &= r - 1) gsrt[ng][j] = __ffs((int)r) - 1;
        gsize[ng] = cnt;
      }
    } else {
      atomicOr(status, 16u);
    }
    s_ngroups = ng;
  }
  __syncthreads();
  if (s_ngroups < 0) return;
  for (int g = 0; g < s_ngroups; ++g) {
    switch (gsize[g]) {
      case 1: fused_group_sweep<1>(tile, tsize, gidx[g], gsrt[g], sg, st); break;
      default: fused_group_sweep<2>(tile, tsize, gidx[g], gsrt[g], sg, st); break;
    }
    __syncthreads();
  }
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < tsize; i += kFusedThreads) s[i] = tile[i];
}

// The same for states of 12 qubits and more: groups of four tile positions, a thread
// holding the 16 amplitudes that a group mixes and applying all gates of each
// position in their order; byte addresses built from the columns of the tile's bits;
// the next tile's 16-byte copies (qubit 0 is in the tile unless twelve other qubits
// are targets) in flight while one is worked on.
//
// Bound by issue: ten gates are 80 FMAs per amplitude, 37 us of FP32 time at 24
// qubits, as many shared-memory and address instructions, and 41 us of HBM
// beside them: 115-133 us; 187-202 in sweeps of two gates, which move the tile
// five times through shared memory.  Three CTAs per SM spill (120 us, and 18.5
// instead of 14.2 at 20 qubits); registers instead of cp.async cost the same.
// Twelve gates on one qubit of 16: 10.7 us a call; 26 with a group for each.  The loop
// over a position's gates only where a target repeats: run always, it costs eight
// gates on 22 qubits 33.7 us instead of 29.8.
constexpr int kTileThreads = 256;

// The tile's columns: as tile_col, but bit 0 stays with position 0, so that a
// pair of amplitudes is one 16-byte word (powers of an element of GF(8)).
__host__ __device__ constexpr uint32_t pair_col(int k) {
  return k < 4 ? 1u << k : (1u << k) | 2u * (uint32_t)((0x5763421ull >> (4 * ((k - 1) % 7))) & 7);
}
__device__ __forceinline__ void copy_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

struct FusedGroup {
  uint16_t v[4], rem[8];   // byte columns of the register bits and of the thread index
  int32_t gate[4];         // first gate on each register bit, -1 for none
};

__global__ void __launch_bounds__(kTileThreads, 2)
    k_fused1q_tiles(float2* __restrict__ s, int n, const float2* __restrict__ gates, const int32_t* __restrict__ targets,
                    int K, uint32_t* status) {
  pdl_begin();
  constexpr int T = kFusedMax;
  extern __shared__ __align__(16) unsigned char tile_smem[];
  __shared__ __align__(16) G2 sg[kFusedMax];
  __shared__ FusedGroup grp[kFusedMax / 4];
  __shared__ int nxt[kFusedMax];            // the next gate on the same target, -1 for none
  __shared__ int last[T];                   // setup: the last gate so far on a position
  __shared__ int st[kFusedMax], sq[T];
  __shared__ uint64_t dep_lo[64], dep_hi[32];   // state index of a pair of amplitudes (tile bits 1-6, 7-11)
  __shared__ uint16_t map_lo[64], map_hi[32];   // its byte address in the tile
  __shared__ int s_groups;
  __shared__ bool s_more;                   // some target has several gates
  const int tid = threadIdx.x;
  if (tid < K) st[tid] = targets[tid];
  if (tid < 4 * K) sg[tid >> 2].g[tid & 3] = gates[tid];
  if (tid < 96) {
    const int first = tid < 64 ? 1 : 7, x = tid < 64 ? tid : tid - 64;
    uint32_t a = 0;
    for (int k = 0; k < (tid < 64 ? 6 : 5); ++k)
      if ((x >> k) & 1) a ^= pair_col(first + k) * 8;
    if (tid < 64) map_lo[x] = (uint16_t)a; else map_hi[x] = (uint16_t)a;
  }
  __syncthreads();
  if (tid == 0) {
    uint64_t m = 0;
    bool ok = true;
    for (int k = 0; k < K; ++k) {
      if (st[k] < 0 || st[k] >= n) ok = false;
      else m |= 1ull << st[k];
    }
    int ng = ok ? 0 : -1;
    const bool more = __popcll(m) < K;
    if (ok) {
      for (int q = 0; __popcll(m) < T; ++q) m |= 1ull << q;
      uint64_t r = m;
      for (int j = 0; j < T; ++j, r &= r - 1) sq[j] = __ffsll((long long)r) - 1;
      // positions in the order of their first gates, four to a group; a
      // position's further gates follow by nxt
      uint32_t seen = 0;
      for (int k = 0; k < K; ++ng) {
        FusedGroup& G = grp[ng];
        uint32_t bits = 0;
        int cnt = 0;
        for (; k < K; ++k) {
          const int p = __popcll(m & ((1ull << st[k]) - 1ull));
          const bool first = !((seen >> p) & 1);
          if (first && cnt == 4) break;
          if (first) {
            G.gate[cnt] = k;
            G.v[cnt++] = (uint16_t)(pair_col(p) * 8);
            bits |= 1u << p;
            seen |= 1u << p;
          } else {
            nxt[last[p]] = k;
          }
          if (more) {
            nxt[k] = -1;
            last[p] = k;
          }
        }
        for (int p = T - 1; cnt < 4; --p)
          if (!((bits >> p) & 1)) {
            G.gate[cnt] = -1;
            G.v[cnt++] = (uint16_t)(pair_col(p) * 8);
            bits |= 1u << p;
          }
        for (int p = 0, j = 0; p < T; ++p)
          if (!((bits >> p) & 1)) G.rem[j++] = (uint16_t)(pair_col(p) * 8);
      }
    } else if (blockIdx.x == 0) {
      atomicOr(status, 16u);
    }
    s_groups = ng;
    s_more = more;
  }
  __syncthreads();
  const int ngroups = s_groups;
  const bool more = s_more;
  if (ngroups < 0) return;
  const bool pairs = sq[0] == 0;
  if (tid < 96) {
    const int first = tid < 64 ? 1 : 7, x = tid < 64 ? tid : tid - 64;
    uint64_t d = 0;
    for (int k = 0; k < (tid < 64 ? 6 : 5); ++k)
      if ((x >> k) & 1) d |= 1ull << sq[first + k];
    if (tid < 64) dep_lo[x] = d; else dep_hi[x] = d;
  }
  __syncthreads();
  constexpr int kPer = (1 << (T - 1)) / kTileThreads;   // pairs per thread
  constexpr uint32_t kTile = 8u << T;
  const uint64_t ntiles = 1ull << (n - T), second = 1ull << sq[0];
  const uint32_t smem = (uint32_t)__cvta_generic_to_shared(tile_smem);
  auto first_of = [&](uint64_t tl) {
    for (int q = 0; q < T; ++q) tl = insert_zero(tl, sq[q]);
    return tl;
  };
  auto fetch = [&](uint64_t tl, uint32_t buf) {
    const uint64_t gbase = first_of(tl);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const uint32_t e = tid + kTileThreads * j, A = buf + (map_lo[e & 63] ^ map_hi[e >> 6]);
      const uint64_t g = gbase | dep_lo[e & 63] | dep_hi[e >> 6];
      if (pairs) {
        copy_async16(smem + A, s + g);
      } else {
        copy_async8(smem + A, s + g);
        copy_async8(smem + A + 8, s + (g | second));
      }
    }
  };
  if (blockIdx.x < ntiles) fetch(blockIdx.x, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  uint32_t buf = 0;
  for (uint64_t tl = blockIdx.x; tl < ntiles; tl += gridDim.x, buf ^= kTile) {
    if (tl + gridDim.x < ntiles) fetch(tl + gridDim.x, buf ^ kTile);
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    auto el = [&](uint32_t byte) -> float2& { return *reinterpret_cast<float2*>(tile_smem + byte); };
    for (int q = 0; q < ngroups; ++q) {
      const FusedGroup& G = grp[q];
      uint32_t A = buf;   // a bit above the tile's
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if ((tid >> j) & 1) A ^= G.rem[j];
      uint32_t at[16];
      at[0] = A;
#pragma unroll
      for (int r = 1; r < 16; ++r) at[r] = at[r & (r - 1)] ^ G.v[31 - __clz(r & -r)];
      float2 w[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) w[r] = el(at[r]);
      const float4* U = reinterpret_cast<const float4*>(sg);
      if (!more) {
        if (G.gate[0] >= 0) gate_on_bit<0>(w, U + 2 * G.gate[0]);
        if (G.gate[1] >= 0) gate_on_bit<1>(w, U + 2 * G.gate[1]);
        if (G.gate[2] >= 0) gate_on_bit<2>(w, U + 2 * G.gate[2]);
        if (G.gate[3] >= 0) gate_on_bit<3>(w, U + 2 * G.gate[3]);
      } else {
        for (int k = G.gate[0]; k >= 0; k = nxt[k]) gate_on_bit<0>(w, U + 2 * k);
        for (int k = G.gate[1]; k >= 0; k = nxt[k]) gate_on_bit<1>(w, U + 2 * k);
        for (int k = G.gate[2]; k >= 0; k = nxt[k]) gate_on_bit<2>(w, U + 2 * k);
        for (int k = G.gate[3]; k >= 0; k = nxt[k]) gate_on_bit<3>(w, U + 2 * k);
      }
#pragma unroll
      for (int r = 0; r < 16; ++r) el(at[r]) = w[r];
      __syncthreads();
    }
    const uint64_t gbase = first_of(tl);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const uint32_t e = tid + kTileThreads * j, A = map_lo[e & 63] ^ map_hi[e >> 6];
      const uint64_t g = gbase | dep_lo[e & 63] | dep_hi[e >> 6];
      const float4 v = *reinterpret_cast<const float4*>(tile_smem + (buf ^ A));
      if (pairs) {
        *reinterpret_cast<float4*>(s + g) = v;
      } else {
        s[g] = lo2(v);
        s[g | second] = hi2(v);
      }
    }
    __syncthreads();   // before the buffer is filled again
  }
}

// ------------------------------------------------------------- 2Q ---------
__device__ __forceinline__ void apply4(const G4& G, float2& a0, float2& a1, float2& a2, float2& a3) {
  float2 v[4] = {a0, a1, a2, a3};
  float2 o[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    float2 row[4] = {G.g[4 * r], G.g[4 * r + 1], G.g[4 * r + 2], G.g[4 * r + 3]};
    o[r] = cdot_comp<4>(row, v);
  }
  a0 = o[0]; a1 = o[1]; a2 = o[2]; a3 = o[3];
}

// As gate2 for 4x4; swap: exchange the roles of matrix index bits 0 and 1.
__device__ __forceinline__ G4 gate4(const G4& G, const float2* __restrict__ gd, int swap) {
  if (!gd) return G;
  G4 R;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int pr = swap ? ((r & 1) << 1 | r >> 1) : r, pc = swap ? ((c & 1) << 1 | c >> 1) : c;
      R.g[4 * r + c] = gd[4 * pr + pc];
    }
  return R;
}

// lo == 0: a00,a01 adjacent and a10,a11 adjacent.
__global__ void k_2q_lo0(float2* __restrict__ s, uint64_t nquads, int hi, G4 G0, const float2* __restrict__ gd,
                         int swap) {
  pdl_begin();
  const G4 G = gate4(G0, gd, swap);
  const uint64_t sh = 1ull << hi;
  for (uint64_t it = gtid(); it < nquads; it += gstride()) {
    uint64_t i00 = insert_zero(insert_zero(it, 0), hi);
    float4 v0 = ld4(s + i00), v1 = ld4(s + i00 + sh);
    float2 a0 = lo2(v0), a1 = hi2(v0), a2 = lo2(v1), a3 = hi2(v1);
    apply4(G, a0, a1, a2, a3);
    st4(s + i00, a0, a1);
    st4(s + i00 + sh, a2, a3);
  }
}

// lo >= 1: two neighbouring quads per thread.
__global__ void k_2q_gen(float2* __restrict__ s, uint64_t nitems, int lo, int hi, G4 G0,
                         const float2* __restrict__ gd, int swap) {
  pdl_begin();
  const G4 G = gate4(G0, gd, swap);
  const uint64_t sl = 1ull << lo, sh = 1ull << hi;
  for (uint64_t it = gtid(); it < nitems; it += gstride()) {
    uint64_t i00 = insert_zero(insert_zero(2 * it, lo), hi);
    float4 v00 = ld4(s + i00), v01 = ld4(s + i00 + sl), v10 = ld4(s + i00 + sh), v11 = ld4(s + i00 + sl + sh);
    float2 a0 = lo2(v00), a1 = lo2(v01), a2 = lo2(v10), a3 = lo2(v11);
    float2 b0 = hi2(v00), b1 = hi2(v01), b2 = hi2(v10), b3 = hi2(v11);
    apply4(G, a0, a1, a2, a3);
    apply4(G, b0, b1, b2, b3);
    st4(s + i00, a0, b0);
    st4(s + i00 + sl, a1, b1);
    st4(s + i00 + sh, a2, b2);
    st4(s + i00 + sl + sh, a3, b3);
  }
}

// ----------------------------------------------------------- diagonal -----
__global__ void k_diag1(float2* __restrict__ s, uint64_t nvec, int t, float2 d0v, float2 d1v,
                        const float2* __restrict__ gd) {
  pdl_begin();
  const float2 d0 = gd ? gd[0] : d0v, d1 = gd ? gd[1] : d1v;
  for (uint64_t i = gtid(); i < nvec; i += gstride()) {
    uint64_t idx = 2 * i;
    float4 v = ld4(s + idx);
    float2 e0, e1;
    if (t == 0) { e0 = d0; e1 = d1; }
    else { e0 = e1 = ((idx >> t) & 1) ? d1 : d0; }
    st4(s + idx, cmul_comp(lo2(v), e0), cmul_comp(hi2(v), e1));
  }
}

// Only amplitudes with bit t = 1 (half the traffic).
__global__ void k_phase_t0(float2* __restrict__ s, uint64_t npairs, float2 ph) {
  pdl_begin();
  for (uint64_t p = gtid(); p < npairs; p += gstride()) {
    uint64_t idx = 2 * p + 1;
    s[idx] = cmul_comp(s[idx], ph);
  }
}
__global__ void k_phase_tn(float2* __restrict__ s, uint64_t nitems, int t, float2 ph) {
  pdl_begin();
  for (uint64_t it = gtid(); it < nitems; it += gstride()) {
    uint64_t idx = insert_zero(2 * it, t) | (1ull << t);
    float4 v = ld4(s + idx);
    st4(s + idx, cmul_comp(lo2(v), ph), cmul_comp(hi2(v), ph));
  }
}

__global__ void k_diag2(float2* __restrict__ s, uint64_t nvec, int q0, int q1, G2 D0, const float2* __restrict__ gd) {
  pdl_begin();
  const G2 D = gate2(D0, gd);
  for (uint64_t i = gtid(); i < nvec; i += gstride()) {
    uint64_t idx = 2 * i;
    float4 v = ld4(s + idx);
    uint64_t j = idx + 1;
    int s0 = (int)(((idx >> q1) & 1) << 1 | ((idx >> q0) & 1));
    int s1 = (int)(((j >> q1) & 1) << 1 | ((j >> q0) & 1));
    st4(s + idx, cmul_comp(lo2(v), D.g[s0]), cmul_comp(hi2(v), D.g[s1]));
  }
}

// ------------------------------------------------- multi-controlled -------
__global__ void k_mc1q(float2* __restrict__ s, uint64_t nitems, Sorted P, uint64_t cmask, int t, G2 G0,
                       const float2* __restrict__ gd) {
  pdl_begin();
  const G2 G = gate2(G0, gd);
  const uint64_t st = 1ull << t;
  for (uint64_t it = gtid(); it < nitems; it += gstride()) {
    uint64_t i0 = insert_zeros(it, P.pos, P.k) | cmask;
    float2 a0 = s[i0], a1 = s[i0 | st];
    apply2(G, a0, a1);
    s[i0] = a0;
    s[i0 | st] = a1;
  }
}

__global__ void k_mc2q(float2* __restrict__ s, uint64_t nitems, Sorted P, uint64_t cmask, int lo, int hi, G4 G0,
                       const float2* __restrict__ gd) {
  pdl_begin();
  const G4 G = gate4(G0, gd, 0);
  const uint64_t sl = 1ull << lo, sh = 1ull << hi;
  for (uint64_t it = gtid(); it < nitems; it += gstride()) {
    uint64_t i = insert_zeros(it, P.pos, P.k) | cmask;
    float2 a0 = s[i], a1 = s[i | sl], a2 = s[i | sh], a3 = s[i | sl | sh];
    apply4(G, a0, a1, a2, a3);
    s[i] = a0; s[i | sl] = a1; s[i | sh] = a2; s[i | sl | sh] = a3;
  }
}

// ---------------------------------------------------------- exact ---------
__global__ void k_x_t0(float2* __restrict__ s, uint64_t npairs) {
  pdl_begin();
  for (uint64_t p = gtid(); p < npairs; p += gstride()) {
    float4 v = ld4(s + 2 * p);
    st4(s + 2 * p, hi2(v), lo2(v));
  }
}
__global__ void k_x_tn(float2* __restrict__ s, uint64_t nitems, int t) {
  pdl_begin();
  const uint64_t st = 1ull << t;
  for (uint64_t it = gtid(); it < nitems; it += gstride()) {
    uint64_t i0 = insert_zero(2 * it, t);
    float4 v0 = ld4(s + i0), v1 = ld4(s + i0 + st);
    *reinterpret_cast<float4*>(s + i0) = v1;
    *reinterpret_cast<float4*>(s + i0 + st) = v0;
  }
}
__global__ void k_mcx(float2* __restrict__ s, uint64_t nitems, Sorted P, uint64_t cmask, int t) {
  pdl_begin();
  const uint64_t st = 1ull << t;
  for (uint64_t it = gtid(); it < nitems; it += gstride()) {
    uint64_t i0 = insert_zeros(it, P.pos, P.k) | cmask;
    float2 a0 = s[i0], a1 = s[i0 | st];
    s[i0] = a1;
    s[i0 | st] = a0;
  }
}
__global__ void k_mcswap(float2* __restrict__ s, uint64_t nitems, Sorted P, uint64_t cmask, int t0, int t1) {
  pdl_begin();
  const uint64_t s0 = 1ull << t0, s1 = 1ull << t1;
  for (uint64_t it = gtid(); it < nitems; it += gstride()) {
    uint64_t i = insert_zeros(it, P.pos, P.k) | cmask;
    float2 a = s[i | s0], b = s[i | s1];
    s[i | s0] = b;
    s[i | s1] = a;
  }
}
__global__ void k_mcz(float2* __restrict__ s, uint64_t nitems, Sorted P, uint64_t mask) {
  pdl_begin();
  for (uint64_t it = gtid(); it < nitems; it += gstride()) {
    uint64_t i = insert_zeros(it, P.pos, P.k) | mask;
    float2 a = s[i];
    s[i] = make_float2(-a.x, -a.y);
  }
}

// --------------------------------------------------------- host side ------
inline float2 f2(const float* p) { return make_float2(p[0], p[1]); }

G2 load_g2(const float* g) {
  QS_CHECK_ARG(g != nullptr, "gate pointer is null");
  G2 G;
  for (int i = 0; i < 4; ++i) G.g[i] = f2(g + 2 * i);
  return G;
}

G4 load_g4(const float* g) {
  QS_CHECK_ARG(g != nullptr, "gate pointer is null");
  G4 G;
  for (int i = 0; i < 16; ++i) G.g[i] = f2(g + 2 * i);
  return G;
}

// Swap the roles of matrix index bits 0 and 1 (basis order 00,01,10,11).
G4 swap_bits(const G4& G) {
  static const int perm[4] = {0, 2, 1, 3};
  G4 R;
  for (int r = 0; r < 4; ++r)
    for (int c = 0; c < 4; ++c) R.g[4 * r + c] = G.g[4 * perm[r] + perm[c]];
  return R;
}

Sorted make_sorted(const int* qs, int k) {
  QS_CHECK_ARG(k <= 12, "too many qubits in a controlled gate");
  Sorted P;
  for (int i = 0; i < k; ++i) P.pos[i] = qs[i];
  std::sort(P.pos, P.pos + k);
  for (int i = 1; i < k; ++i) QS_CHECK_ARG(P.pos[i] != P.pos[i - 1], "duplicate qubit in gate");
  for (int i = k; i < 12; ++i) P.pos[i] = 0;
  P.k = k;
  return P;
}

void check_controls(const int* controls, int nc, int n) {
  QS_CHECK_ARG(nc >= 0 && nc <= QS_MAX_CONTROLS, "controls must have 0-7 elements");
  QS_CHECK_ARG(nc == 0 || controls != nullptr, "controls pointer is null");
  for (int i = 0; i < nc; ++i) qs_check_qubit(controls[i], n, "control");
}

#define LAUNCH(h, kern, items, ...)                                              \
  do {                                                                          \
    uint64_t _items = (items);                                                  \
    if (_items) {                                                               \
      qs_launch_pdl(h, kern, dim3((unsigned)qs_blocks_for(h, _items, kThreads)), dim3(kThreads), 0, __VA_ARGS__); \
      qs_after_launch(h, #kern);                                                \
    }                                                                           \
  } while (0)

}  // namespace

// Exposed to other units (apply_gates_fused fallback and tests).
void qs_launch_1q(qs_context* h, float2* s, uint64_t npairs_total, int t, const G2& G,
                  const float2* gd = nullptr);

void qs_launch_1q(qs_context* h, float2* s, uint64_t npairs, int t, const G2& G, const float2* gd) {
  if (t == 0) LAUNCH(h, k_1q_t0, npairs, s, npairs, G, gd);
  else LAUNCH(h, k_1q_tn, npairs / 2, s, npairs / 2, t, G, gd);
}

extern "C" {

int qs_state_init(qs_handle_t h, void* state, int n) {
  return qs_state_init_basis(h, state, n, 0);
}

int qs_state_init_basis(qs_handle_t h, void* state, int n, uint64_t index) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(index < (1ull << n), "basis index out of range");
  uint64_t nvec = (1ull << n) / 2;
  LAUNCH(h, k_state_init, nvec, (float4*)state, nvec, index);
  QS_API_END(h)
}

int qs_state_alloc(qs_handle_t h, int n, void** out) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  QS_CHECK_ARG(out != nullptr, "out is null");
  *out = nullptr;
  QS_CHECK_ARG(n >= 1 && n <= QS_MAX_QUBITS, "n_qubits out of range [1, 34]");
  void* p = nullptr;
  const cudaError_t e = cudaMallocAsync(&p, (size_t)8 << n, h->stream);
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw qs_error(QS_ERR_NOMEM, std::string("state allocation: ") + cudaGetErrorString(e));
  }
  *out = p;
  QS_API_END(h)
}

int qs_state_free(qs_handle_t h, void* state) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  if (state) QS_CUDA(cudaFreeAsync(state, h->stream));
  QS_API_END(h)
}

int qs_state_copy_to_host(qs_handle_t h, const void* state, int n, void* host) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(host != nullptr, "host buffer is null");
  QS_CUDA(cudaMemcpyAsync(host, state, (size_t)8 << n, cudaMemcpyDeviceToHost, h->stream));
  QS_CUDA(cudaStreamSynchronize(h->stream));
  QS_API_END(h)
}

int qs_state_copy_from_host(qs_handle_t h, void* state, int n, const void* host) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(host != nullptr, "host buffer is null");
  QS_CUDA(cudaMemcpyAsync(state, host, (size_t)8 << n, cudaMemcpyHostToDevice, h->stream));
  QS_CUDA(cudaStreamSynchronize(h->stream));
  QS_API_END(h)
}

int qs_state_init_batched(qs_handle_t h, void* states, int n_states, int n) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(states, n);
  QS_CHECK_ARG(n_states >= 0, "n_states must be >= 0");
  uint64_t nvec = (uint64_t)n_states * ((1ull << n) / 2);
  LAUNCH(h, k_state_init_batched, nvec, (float4*)states, nvec, n);
  QS_API_END(h)
}

int qs_apply_1q(qs_handle_t h, void* state, int n, const float* gate, int t) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  qs_check_qubit(t, n, "target");
  G2 G = load_g2(gate);
  qs_launch_1q(h, (float2*)state, 1ull << (n - 1), t, G);
  QS_API_END(h)
}

int qs_apply_1q_batched(qs_handle_t h, void* states, int n_states, int n, const float* gate, int t) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(states, n);
  qs_check_qubit(t, n, "target");
  QS_CHECK_ARG(n_states >= 0, "n_states must be >= 0");
  G2 G = load_g2(gate);
  // Pair index p ranges over n_states * 2^(n-1); inserting a zero at t < n
  // leaves the state index in the bits above n.
  qs_launch_1q(h, (float2*)states, (uint64_t)n_states << (n - 1), t, G);
  QS_API_END(h)
}

// Gates whose matrix is a device array (complex64, row-major): the kernel
// reads it, so the call neither copies it to the host nor waits for the
// stream.  The pointer must be device memory of the handle's own GPU (or
// managed memory): a gate on another GPU would be read across the link, or
// fault when peer access is off.
// The last four pointers that passed are remembered per handle together with
// the device each was checked for (gate tensors are usually reused call after
// call).  An address that was freed and handed out again by another
// allocation of the same GPU is still device memory of that GPU, so the
// remembered answer stays true for it.
static void check_dev_ptr(qs_context* h, const void* p, const char* what) {
  QS_CHECK_ARG(p != nullptr && ((uintptr_t)p & 7u) == 0, std::string(what) + " must be 8-byte aligned");
  for (int k = 0; k < 4; ++k)
    if (p == h->dev_ptr_ok[k] && h->dev_ptr_ok_device[k] == h->device) return;
  cudaPointerAttributes a;
  const cudaError_t e = cudaPointerGetAttributes(&a, p);
  if (e != cudaSuccess) (void)cudaGetLastError();  // clear the sticky-free error state of the query
  QS_CHECK_ARG(e == cudaSuccess && (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged),
               std::string(what) + " is not device memory");
  QS_CHECK_ARG(a.type == cudaMemoryTypeManaged || a.device == h->device,
               std::string(what) + " is device memory of GPU " + std::to_string(a.device) +
                   ", not of the handle's GPU " + std::to_string(h->device));
  h->dev_ptr_ok[h->dev_ptr_next] = p;
  h->dev_ptr_ok_device[h->dev_ptr_next] = h->device;
  h->dev_ptr_next = (h->dev_ptr_next + 1) & 3;
}

int qs_apply_1q_dev(qs_handle_t h, void* state, int n, const void* gate_dev, int t) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  qs_check_qubit(t, n, "target");
  check_dev_ptr(h, gate_dev, "gate");
  qs_launch_1q(h, (float2*)state, 1ull << (n - 1), t, G2{}, static_cast<const float2*>(gate_dev));
  QS_API_END(h)
}

int qs_apply_gates_fused_dev(qs_handle_t h, void* state, int n, const void* gates_dev, const void* targets_dev,
                             int n_gates) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(n_gates >= 0, "n_gates must be >= 0");
  if (n_gates == 0) return QS_OK;
  check_dev_ptr(h, gates_dev, "gates");
  QS_CHECK_ARG(((uintptr_t)targets_dev & 3u) == 0, "targets must be 4-byte aligned");
  check_dev_ptr(h, targets_dev, "targets");
  const int T = std::min(n, kFusedMax);
  const uint64_t ntiles = 1ull << (n - T);
  // Below 12 qubits the state is one small tile, which groups of two gates and
  // 512 threads finish sooner; from 12 on k_fused1q_tiles is never behind (ten
  // gates: 16 qubits 11.8 against 13.2 us, 20 qubits 14.2 / 16.2, 24 qubits 115 /
  // 187), in one wave of its two CTAs per SM.
  const bool wide = n >= kFusedMax;
  const size_t smem = (wide ? 2 : 1) * (sizeof(float2) << T);
  if (wide) qs_smem_limit(h, (const void*)k_fused1q_tiles, smem);   // (every call's size is this one)
  const unsigned grid = (unsigned)std::min<uint64_t>(ntiles, (uint64_t)h->sm_count * 2);
  const float2* g = static_cast<const float2*>(gates_dev);
  const int32_t* t = static_cast<const int32_t*>(targets_dev);
  // at most 12 gates per launch, so their distinct targets always fit a tile
  for (int k0 = 0; k0 < n_gates; k0 += kFusedMax) {
    const int K = std::min(kFusedMax, n_gates - k0);
    qs_launch_pdl(h, wide ? k_fused1q_tiles : k_fused1q_dev, dim3(grid), dim3(wide ? kTileThreads : kFusedThreads), smem,
                  (float2*)state, n, g + 4 * k0, t + k0, K, h->dev_status);
    qs_after_launch(h, "k_fused1q");
  }
  QS_API_END(h)
}

int qs_apply_2q_dev(qs_handle_t h, void* state, int n, const void* gate_dev, int q0, int q1) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(n >= 2, "a 2-qubit gate needs n >= 2");
  qs_check_qubit(q0, n, "qubit0");
  qs_check_qubit(q1, n, "qubit1");
  QS_CHECK_ARG(q0 != q1, "qubit0 and qubit1 must differ");
  check_dev_ptr(h, gate_dev, "gate");
  const int lo = std::min(q0, q1), hi = std::max(q0, q1), swap = q0 > q1 ? 1 : 0;
  const float2* gd = static_cast<const float2*>(gate_dev);
  uint64_t nquads = 1ull << (n - 2);
  if (lo == 0) LAUNCH(h, k_2q_lo0, nquads, (float2*)state, nquads, hi, G4{}, gd, swap);
  else LAUNCH(h, k_2q_gen, nquads / 2, (float2*)state, nquads / 2, lo, hi, G4{}, gd, swap);
  QS_API_END(h)
}

int qs_apply_diag1_dev(qs_handle_t h, void* state, int n, const void* diag_dev, int t) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  qs_check_qubit(t, n, "target");
  check_dev_ptr(h, diag_dev, "diag");
  uint64_t nvec = (1ull << n) / 2;
  LAUNCH(h, k_diag1, nvec, (float2*)state, nvec, t, make_float2(0.f, 0.f), make_float2(0.f, 0.f),
         static_cast<const float2*>(diag_dev));
  QS_API_END(h)
}

int qs_apply_mc1q_dev(qs_handle_t h, void* state, int n, const void* gate_dev, const int* controls, int nc, int t) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  qs_check_qubit(t, n, "target");
  check_controls(controls, nc, n);
  check_dev_ptr(h, gate_dev, "gate");
  const float2* gd = static_cast<const float2*>(gate_dev);
  if (nc == 0) { qs_launch_1q(h, (float2*)state, 1ull << (n - 1), t, G2{}, gd); return QS_OK; }
  int all[QS_MAX_CONTROLS + 1];
  uint64_t cmask = 0;
  for (int i = 0; i < nc; ++i) {
    QS_CHECK_ARG(controls[i] != t, "target_qubit must not appear in controls");
    all[i] = controls[i];
    cmask |= 1ull << controls[i];
  }
  all[nc] = t;
  Sorted P = make_sorted(all, nc + 1);
  QS_CHECK_ARG(nc + 1 <= n, "more gate qubits than state qubits");
  uint64_t items = 1ull << (n - nc - 1);
  LAUNCH(h, k_mc1q, items, (float2*)state, items, P, cmask, t, G2{}, gd);
  QS_API_END(h)
}

int qs_apply_2q(qs_handle_t h, void* state, int n, const float* gate, int q0, int q1) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(n >= 2, "a 2-qubit gate needs n >= 2");
  qs_check_qubit(q0, n, "qubit0");
  qs_check_qubit(q1, n, "qubit1");
  QS_CHECK_ARG(q0 != q1, "qubit0 and qubit1 must differ");
  G4 G = load_g4(gate);
  int lo = q0, hi = q1;
  if (q0 > q1) { G = swap_bits(G); lo = q1; hi = q0; }
  uint64_t nquads = 1ull << (n - 2);
  if (lo == 0) LAUNCH(h, k_2q_lo0, nquads, (float2*)state, nquads, hi, G, nullptr, 0);
  else LAUNCH(h, k_2q_gen, nquads / 2, (float2*)state, nquads / 2, lo, hi, G, nullptr, 0);
  QS_API_END(h)
}

int qs_apply_diag1(qs_handle_t h, void* state, int n, const float* diag, int t) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  qs_check_qubit(t, n, "target");
  QS_CHECK_ARG(diag != nullptr, "diag pointer is null");
  uint64_t nvec = (1ull << n) / 2;
  LAUNCH(h, k_diag1, nvec, (float2*)state, nvec, t, f2(diag), f2(diag + 2), nullptr);
  QS_API_END(h)
}

int qs_apply_phase(qs_handle_t h, void* state, int n, float re, float im, int t) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  qs_check_qubit(t, n, "target");
  float2 ph = make_float2(re, im);
  uint64_t npairs = 1ull << (n - 1);
  if (t == 0) LAUNCH(h, k_phase_t0, npairs, (float2*)state, npairs, ph);
  else LAUNCH(h, k_phase_tn, npairs / 2, (float2*)state, npairs / 2, t, ph);
  QS_API_END(h)
}

int qs_apply_diag2(qs_handle_t h, void* state, int n, const float* diag, int q0, int q1) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(n >= 2, "a 2-qubit gate needs n >= 2");
  qs_check_qubit(q0, n, "qubit0");
  qs_check_qubit(q1, n, "qubit1");
  QS_CHECK_ARG(q0 != q1, "qubit0 and qubit1 must differ");
  QS_CHECK_ARG(diag != nullptr, "diag pointer is null");
  G2 D = load_g2(diag);
  int lo = std::min(q0, q1), hi = std::max(q0, q1);
  uint64_t nvec = (1ull << n) / 2;
  LAUNCH(h, k_diag2, nvec, (float2*)state, nvec, lo, hi, D, nullptr);
  QS_API_END(h)
}

int qs_apply_diag2_dev(qs_handle_t h, void* state, int n, const void* diag_dev, int q0, int q1) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(n >= 2, "a 2-qubit gate needs n >= 2");
  qs_check_qubit(q0, n, "qubit0");
  qs_check_qubit(q1, n, "qubit1");
  QS_CHECK_ARG(q0 != q1, "qubit0 and qubit1 must differ");
  check_dev_ptr(h, diag_dev, "diag");
  const int lo = std::min(q0, q1), hi = std::max(q0, q1);
  const uint64_t nvec = (1ull << n) / 2;
  LAUNCH(h, k_diag2, nvec, (float2*)state, nvec, lo, hi, G2{}, static_cast<const float2*>(diag_dev));
  QS_API_END(h)
}

int qs_apply_mc1q(qs_handle_t h, void* state, int n, const float* gate, const int* controls, int nc, int t) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  qs_check_qubit(t, n, "target");
  check_controls(controls, nc, n);
  G2 G = load_g2(gate);
  if (nc == 0) { qs_launch_1q(h, (float2*)state, 1ull << (n - 1), t, G); return QS_OK; }
  int all[QS_MAX_CONTROLS + 1];
  uint64_t cmask = 0;
  for (int i = 0; i < nc; ++i) {
    QS_CHECK_ARG(controls[i] != t, "target_qubit must not appear in controls");
    all[i] = controls[i];
    cmask |= 1ull << controls[i];
  }
  all[nc] = t;
  Sorted P = make_sorted(all, nc + 1);
  QS_CHECK_ARG(nc + 1 <= n, "more gate qubits than state qubits");
  uint64_t items = 1ull << (n - nc - 1);
  LAUNCH(h, k_mc1q, items, (float2*)state, items, P, cmask, t, G, nullptr);
  QS_API_END(h)
}

int qs_apply_mc2q(qs_handle_t h, void* state, int n, const float* gate, const int* controls, int nc, int t0, int t1) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  qs_check_qubit(t0, n, "target0");
  qs_check_qubit(t1, n, "target1");
  QS_CHECK_ARG(t0 != t1, "target0 and target1 must differ");
  check_controls(controls, nc, n);
  QS_CHECK_ARG(nc + 2 <= n, "more gate qubits than state qubits");
  G4 G = load_g4(gate);
  int lo = std::min(t0, t1), hi = std::max(t0, t1);
  int all[QS_MAX_CONTROLS + 2];
  uint64_t cmask = 0;
  for (int i = 0; i < nc; ++i) {
    QS_CHECK_ARG(controls[i] != t0 && controls[i] != t1, "target qubits must not appear in controls");
    all[i] = controls[i];
    cmask |= 1ull << controls[i];
  }
  all[nc] = lo;
  all[nc + 1] = hi;
  Sorted P = make_sorted(all, nc + 2);
  uint64_t items = 1ull << (n - nc - 2);
  LAUNCH(h, k_mc2q, items, (float2*)state, items, P, cmask, lo, hi, G, nullptr);
  QS_API_END(h)
}

int qs_apply_mc2q_dev(qs_handle_t h, void* state, int n, const void* gate_dev, const int* controls, int nc, int t0,
                      int t1) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  qs_check_qubit(t0, n, "target0");
  qs_check_qubit(t1, n, "target1");
  QS_CHECK_ARG(t0 != t1, "target0 and target1 must differ");
  check_controls(controls, nc, n);
  QS_CHECK_ARG(nc + 2 <= n, "more gate qubits than state qubits");
  check_dev_ptr(h, gate_dev, "gate");
  const int lo = std::min(t0, t1), hi = std::max(t0, t1);
  int all[QS_MAX_CONTROLS + 2];
  uint64_t cmask = 0;
  for (int i = 0; i < nc; ++i) {
    QS_CHECK_ARG(controls[i] != t0 && controls[i] != t1, "target qubits must not appear in controls");
    all[i] = controls[i];
    cmask |= 1ull << controls[i];
  }
  all[nc] = lo;
  all[nc + 1] = hi;
  Sorted P = make_sorted(all, nc + 2);
  const uint64_t items = 1ull << (n - nc - 2);
  LAUNCH(h, k_mc2q, items, (float2*)state, items, P, cmask, lo, hi, G4{}, static_cast<const float2*>(gate_dev));
  QS_API_END(h)
}

int qs_apply_mcx(qs_handle_t h, void* state, int n, const int* controls, int nc, int t) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  qs_check_qubit(t, n, "target");
  check_controls(controls, nc, n);
  QS_CHECK_ARG(nc + 1 <= n, "more gate qubits than state qubits");
  if (nc == 0) {
    uint64_t npairs = 1ull << (n - 1);
    if (t == 0) LAUNCH(h, k_x_t0, npairs, (float2*)state, npairs);
    else LAUNCH(h, k_x_tn, npairs / 2, (float2*)state, npairs / 2, t);
    return QS_OK;
  }
  int all[QS_MAX_CONTROLS + 1];
  uint64_t cmask = 0;
  for (int i = 0; i < nc; ++i) {
    QS_CHECK_ARG(controls[i] != t, "target_qubit must not appear in controls");
    all[i] = controls[i];
    cmask |= 1ull << controls[i];
  }
  all[nc] = t;
  Sorted P = make_sorted(all, nc + 1);
  uint64_t items = 1ull << (n - nc - 1);
  LAUNCH(h, k_mcx, items, (float2*)state, items, P, cmask, t);
  QS_API_END(h)
}

int qs_apply_mcswap(qs_handle_t h, void* state, int n, const int* controls, int nc, int t0, int t1) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  qs_check_qubit(t0, n, "target0");
  qs_check_qubit(t1, n, "target1");
  QS_CHECK_ARG(t0 != t1, "target0 and target1 must differ");
  check_controls(controls, nc, n);
  QS_CHECK_ARG(nc + 2 <= n, "more gate qubits than state qubits");
  int all[QS_MAX_CONTROLS + 2];
  uint64_t cmask = 0;
  for (int i = 0; i < nc; ++i) {
    QS_CHECK_ARG(controls[i] != t0 && controls[i] != t1, "target qubits must not appear in controls");
    all[i] = controls[i];
    cmask |= 1ull << controls[i];
  }
  all[nc] = t0;
  all[nc + 1] = t1;
  Sorted P = make_sorted(all, nc + 2);
  uint64_t items = 1ull << (n - nc - 2);
  LAUNCH(h, k_mcswap, items, (float2*)state, items, P, cmask, t0, t1);
  QS_API_END(h)
}

int qs_apply_mcz(qs_handle_t h, void* state, int n, const int* qubits, int k) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(k >= 1 && k <= QS_MAX_CONTROLS + 1 && k <= n, "mcz needs 1..8 qubits");
  QS_CHECK_ARG(qubits != nullptr, "qubits pointer is null");
  uint64_t mask = 0;
  for (int i = 0; i < k; ++i) { qs_check_qubit(qubits[i], n, "mcz"); mask |= 1ull << qubits[i]; }
  Sorted P = make_sorted(qubits, k);
  uint64_t items = 1ull << (n - k);
  LAUNCH(h, k_mcz, items, (float2*)state, items, P, mask);
  QS_API_END(h)
}

}  // extern "C"
