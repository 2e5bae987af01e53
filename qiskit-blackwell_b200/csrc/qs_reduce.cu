// qs_reduce.cu — reductions over a state, accumulated in FP64 in a fixed
// order (no floating-point atomics), so every result is bit-reproducible and
// the same whether a state is processed alone or inside a batch.
//
// Two-stage scheme: stage 1 gives each block a fixed contiguous slice of the
// index range (the slicing depends only on the item count); every thread sums
// a fixed strided subset sequentially, then the block reduces in a fixed tree
// order.  Stage 2 is one block that reduces the per-block partials in order.
#include "qs_api.h"
#include <vector>
#include "qs_common.cuh"
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>

using namespace qs;

namespace {

constexpr int kThreads = 256;
constexpr int kMaxBlocks = 1024;
// Two waves of the three CTAs that fit on each of 148 SMs; a constant, so that the
// order of an expectation value's sums depends on the width alone.
constexpr int kPauliBlocks = 888;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Fixed-order block reduction; the result is valid in thread 0.
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double ws[32];
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) ws[w] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  v = 0.0;
  if (w == 0) {
    v = lane < nw ? ws[lane] : 0.0;
    v = warp_sum(v);
  }
  return v;
}

struct Slicing { int nb; uint64_t per; };
Slicing slice(uint64_t items) {
  uint64_t nb = (items + 4095) / 4096;
  if (nb > kMaxBlocks) nb = kMaxBlocks;
  if (nb < 1) nb = 1;
  return Slicing{(int)nb, (items + nb - 1) / nb};
}

// -------------------------------------------------------------- functors -
// Each functor sees "items" = float4 vectors (two amplitudes).
struct FNorm {
  const float4* s;
  __device__ double operator()(uint64_t i) const {
    float4 v = s[i];
    return (double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z + (double)v.w * v.w;
  }
};

struct FP0 {  // probability of bit t = 0
  const float4* s;
  int t;
  __device__ double operator()(uint64_t i) const {
    float4 v = s[i];
    double a = (double)v.x * v.x + (double)v.y * v.y;
    double b = (double)v.z * v.z + (double)v.w * v.w;
    if (t == 0) return a;
    return ((2 * i) >> t) & 1 ? 0.0 : a + b;
  }
};

struct FZ {  // sum |a_i|^2 (-1)^popc(i & z)
  const float4* s;
  uint64_t z;
  __device__ double operator()(uint64_t i) const {
    float4 v = s[i];
    double a = (double)v.x * v.x + (double)v.y * v.y;
    double b = (double)v.z * v.z + (double)v.w * v.w;
    uint64_t i0 = 2 * i;
    double s0 = (__popcll(i0 & z) & 1) ? -a : a;
    double s1 = (__popcll((i0 + 1) & z) & 1) ? -b : b;
    return s0 + s1;
  }
};

template <class F>
__global__ void k_reduce(F f, uint64_t items, uint64_t per, double* __restrict__ partial) {
  pdl_begin();
  const uint64_t b0 = (uint64_t)blockIdx.x * per;
  const uint64_t e = min(b0 + per, items);
  double acc = 0.0;
  for (uint64_t i = b0 + threadIdx.x; i < e; i += blockDim.x) acc += f(i);
  acc = block_sum(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc;
}

// mode 0: out[0] = sum.  mode 1: out[0] = sum, out[1] = 1/sqrt(sum) (renorm).
__global__ void k_final(const double* __restrict__ partial, int nb, double* __restrict__ out, int mode) {
  pdl_begin();
  double acc = 0.0;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) acc += partial[i];
  acc = block_sum(acc);
  if (threadIdx.x == 0) {
    out[0] = acc;
    if (mode == 1) out[1] = acc > 0.0 ? 1.0 / sqrt(acc) : 0.0;
  }
}

__global__ void k_scale(float4* __restrict__ s, uint64_t nvec, const double* __restrict__ scale) {
  pdl_begin();
  const float f = (float)scale[1];
  for (uint64_t i = gtid(); i < nvec; i += gstride()) {
    float4 v = s[i];
    s[i] = make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
  }
}

__global__ void k_probs(const float4* __restrict__ s, float2* __restrict__ p, uint64_t nvec) {
  pdl_begin();
  for (uint64_t i = gtid(); i < nvec; i += gstride()) {
    float4 v = s[i];
    p[i] = make_float2(v.x * v.x + v.y * v.y, v.z * v.z + v.w * v.w);
  }
}

// Collapse after measuring qubit t: keep amplitudes with bit t == outcome,
// scaled by 1/sqrt(p_outcome); zero the others.  pr[0] = P(bit = 0).
__global__ void k_collapse(float4* __restrict__ s, uint64_t nvec, int t, double u, const double* __restrict__ pr,
                           int* __restrict__ outcome) {
  pdl_begin();
  const double p0 = pr[0];
  const int res = (u < p0) ? 0 : 1;
  const double p = res == 0 ? p0 : 1.0 - p0;
  const float f = p > 1e-30 ? (float)(1.0 / sqrt(p)) : 0.f;
  if (blockIdx.x == 0 && threadIdx.x == 0) *outcome = res;
  for (uint64_t i = gtid(); i < nvec; i += gstride()) {
    float4 v = s[i];
    const uint64_t i0 = 2 * i;
    const int b0 = (int)((i0 >> t) & 1), b1 = (int)(((i0 + 1) >> t) & 1);
    const float f0 = b0 == res ? f : 0.f, f1 = b1 == res ? f : 0.f;
    s[i] = make_float4(v.x * f0, v.y * f0, v.z * f1, v.w * f1);
  }
}

// ----------------------------------------------------------- sampling ----
// The CDF is built in chunks of kChunk amplitudes.  A chunk is split into 32
// contiguous segments of kSeg amplitudes, one per lane; a lane sums its
// segment sequentially in FP64 and the warp scans the 32 segment sums in a
// fixed shuffle order.  The same routine (seg_sum_staged) produces the chunk
// totals (pass 1) and the in-chunk search (pass 3), so both see identical
// values.
constexpr int kSeg = 64;
constexpr int kChunk = 32 * kSeg;

// |a|^2 in FP64, and a segment's running sum: the one expression and order
// that every pass uses, so the chunk totals and the in-chunk search agree bit
// for bit.
__device__ __forceinline__ void seg_add(double& acc, float2 a) { acc += (double)a.x * a.x + (double)a.y * a.y; }

// Lane `lane`'s segment sum of the chunk starting at `c0`: its amplitudes
// c0 + lane * kSeg + k, k = 0..kSeg-1, added by seg_add in order.  The chunk
// is read in coalesced 128-byte runs (a segment is 512 contiguous bytes per
// lane, so loading it lane by lane would touch 32 lines per warp access): the
// warp stages 16 amplitudes of every segment at a time in `buf` (32 rows of
// 17: the pad spreads a row walk over the banks) and each lane adds its row.
__device__ __forceinline__ void seg_stage_load(const float2* __restrict__ s, uint64_t c0, uint64_t n, int lane, int q,
                                               float4 (&r)[8]) {
  // lanes 8k..8k+7 cover one 128-byte run (16 amplitudes of one segment),
  // two amplitudes per lane.  16-byte loads when the state starts on a
  // 16-byte boundary and has an even length (every state of one or more
  // qubits): g is even, so the pair is then either inside it or past its end
  const bool v4 = ((reinterpret_cast<uintptr_t>(s) & 15) == 0) && !(n & 1);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint64_t g = c0 + (uint64_t)(4 * i + (lane >> 3)) * kSeg + 16 * q + 2 * (lane & 7);
    if (v4 && g < n) {
      r[i] = *reinterpret_cast<const float4*>(s + g);
    } else {
      const float2 lo = g < n ? s[g] : make_float2(0.f, 0.f);
      const float2 hi = g + 1 < n ? s[g + 1] : make_float2(0.f, 0.f);
      r[i] = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
  }
}
__device__ __forceinline__ double seg_sum_staged(const float2* __restrict__ s, uint64_t c0, uint64_t n, int lane,
                                                 float2 (*buf)[17]) {
  double acc = 0.0;
  float4 r[8];
  seg_stage_load(s, c0, n, lane, 0, r);
#pragma unroll 1
  for (int q = 0; q < kSeg / 16; ++q) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = 4 * i + (lane >> 3), e = 2 * (lane & 7);
      buf[row][e] = make_float2(r[i].x, r[i].y);
      buf[row][e + 1] = make_float2(r[i].z, r[i].w);
    }
    __syncwarp();
    if (q + 1 < kSeg / 16) seg_stage_load(s, c0, n, lane, q + 1, r);  // in flight while this row is summed
    const uint64_t start = c0 + (uint64_t)lane * kSeg + 16 * q;
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (start + k < n) seg_add(acc, buf[lane][k]);
    __syncwarp();
  }
  return acc;
}

// inclusive warp scan in fixed order
__device__ __forceinline__ double warp_iscan(double v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    double y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  return v;
}

// pass 1: one warp per chunk -> csum[c]
__global__ void k_chunk_sums(const float2* __restrict__ s, uint64_t n, uint64_t nchunks, double* __restrict__ csum) {
  pdl_begin();
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  __shared__ float2 stage[kThreads / 32][32][17];
  for (uint64_t c = warp; c < nchunks; c += nwarps) {
    double v = seg_sum_staged(s, c * kChunk, n, lane, stage[threadIdx.x >> 5]);
    v = warp_iscan(v);
    if (lane == 31) csum[c] = v;
  }
}

// pass 2: exclusive scan of the chunk sums, one block, fixed order.
// cbase[c] = sum_{c' < c} csum[c'];  cbase[nchunks] = total.  The order
// depends only on nchunks and the block size (1024 threads in every launch).
// Each thread owns a contiguous run of `per` chunks; the block walks the runs
// kScanCols columns at a time through a shared tile (one row per thread), so
// csum is read and cbase written in coalesced 64-byte runs while every thread
// still adds its own run in order.  The next columns are fetched into
// registers while the current tile is summed.
constexpr int kScanThreads = 1024;
constexpr int kScanCols = 8;
constexpr size_t kScanSmem = sizeof(double) * kScanThreads * (kScanCols + 1);
using ScanTile = double (*)[kScanCols + 1];

// element m of this thread's share of a tile is row tid / kScanCols +
// m * (kScanThreads / kScanCols), column tid % kScanCols: chunk
// c0 + k0 + m * cstride, with c0 = (tid / kScanCols) * per + tid % kScanCols.
// A state of at most 34 qubits has at most 2^23 chunks: 32-bit indices.
struct ScanCols {
  uint32_t c0, cstride;
  int col;
};
__device__ __forceinline__ ScanCols scan_cols(uint64_t per) {
  const int col = threadIdx.x % kScanCols;
  return {(uint32_t)((threadIdx.x / kScanCols) * per + col), (uint32_t)((kScanThreads / kScanCols) * per), col};
}

__device__ __forceinline__ void scan_tile_fetch(const double* __restrict__ csum, uint64_t nchunks, uint64_t per,
                                                const ScanCols& sc, uint64_t k0, double (&r)[kScanCols]) {
  const bool in_run = k0 + sc.col < per;
#pragma unroll
  for (int m = 0; m < kScanCols; ++m) {
    const uint32_t c = sc.c0 + (uint32_t)k0 + m * sc.cstride;
    r[m] = (in_run && c < nchunks) ? csum[c] : 0.0;
  }
}

__device__ __forceinline__ void scan_tile_put(const double (&r)[kScanCols], ScanTile tile) {
#pragma unroll
  for (int m = 0; m < kScanCols; ++m) {
    const int i = threadIdx.x + kScanThreads * m;
    tile[i / kScanCols][i % kScanCols] = r[m];
  }
}

__device__ __forceinline__ void scan_tile_store(double* __restrict__ cbase, uint64_t nchunks, uint64_t per,
                                                const ScanCols& sc, uint64_t k0, ScanTile tile) {
  const bool in_run = k0 + sc.col < per;
#pragma unroll
  for (int m = 0; m < kScanCols; ++m) {
    const uint32_t c = sc.c0 + (uint32_t)k0 + m * sc.cstride;
    const int i = threadIdx.x + kScanThreads * m;
    if (in_run && c < nchunks) cbase[c] = tile[i / kScanCols][i % kScanCols];
  }
}

__device__ __forceinline__ void chunk_scan_block(const double* __restrict__ csum, uint64_t nchunks,
                                                 double* __restrict__ cbase, double* ws, double& carry, ScanTile tile) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const uint64_t per = (nchunks + kScanThreads - 1) / kScanThreads;
  const uint64_t b = (uint64_t)tid * per, e = min(b + per, nchunks);
  const ScanCols sc = scan_cols(per);
  double r[kScanCols];
  double local = 0.0;
  scan_tile_fetch(csum, nchunks, per, sc, 0, r);
  for (uint64_t k0 = 0; k0 < per; k0 += kScanCols) {
    scan_tile_put(r, tile);
    __syncthreads();
    if (k0 + kScanCols < per) scan_tile_fetch(csum, nchunks, per, sc, k0 + kScanCols, r);
#pragma unroll
    for (int j = 0; j < kScanCols; ++j)
      if (b + k0 + j < e) local += tile[tid][j];
    __syncthreads();
  }
  // block exclusive scan of `local`
  double inc = warp_iscan(local);
  double exc = __shfl_up_sync(0xffffffffu, inc, 1);
  if (lane == 0) exc = 0.0;
  if (lane == 31) ws[w] = inc;
  __syncthreads();
  if (w == 0) {
    const int nw = kScanThreads >> 5;
    double x = lane < nw ? ws[lane] : 0.0;
    double xi = warp_iscan(x);
    double xe = __shfl_up_sync(0xffffffffu, xi, 1);
    if (lane == 0) xe = 0.0;
    __syncwarp();
    if (lane < nw) ws[lane] = xe;  // exclusive warp offsets
    if (lane == nw - 1) carry = xi;
  }
  __syncthreads();
  double run = ws[w] + exc;
  scan_tile_fetch(csum, nchunks, per, sc, 0, r);
  for (uint64_t k0 = 0; k0 < per; k0 += kScanCols) {
    scan_tile_put(r, tile);
    __syncthreads();
    if (k0 + kScanCols < per) scan_tile_fetch(csum, nchunks, per, sc, k0 + kScanCols, r);
#pragma unroll
    for (int j = 0; j < kScanCols; ++j) {
      if (b + k0 + j < e) {
        const double v = tile[tid][j];
        tile[tid][j] = run;
        run += v;
      }
    }
    __syncthreads();
    scan_tile_store(cbase, nchunks, per, sc, k0, tile);
    __syncthreads();
  }
  if (tid == 0) cbase[nchunks] = carry;
}

__global__ void __launch_bounds__(kScanThreads, 1)
    k_chunk_scan(const double* __restrict__ csum, uint64_t nchunks, double* __restrict__ cbase) {
  pdl_begin();
  __shared__ double ws[32];
  __shared__ double carry;
  extern __shared__ double scan_smem[];
  chunk_scan_block(csum, nchunks, cbase, ws, carry, reinterpret_cast<ScanTile>(scan_smem));
}

// pass 3, one shot by one warp: u -> smallest i with cdf[i] >= u, clamped to
// n-1 (reference semantics: sample_sm120.cu:61-68).  Every lane returns it.
__device__ __forceinline__ int64_t sample_one(const float2* __restrict__ s, uint64_t n, uint64_t nchunks,
                                              const double* __restrict__ cbase, double x, float2 (*buf)[17]) {
  const int lane = threadIdx.x & 31;
  // smallest chunk c with cbase[c+1] >= x (nchunks if none): a 32-way search,
  // each lane probing one of 32 evenly spaced chunks per round.  cbase is
  // non-decreasing, so this finds the same chunk as a binary search.
  // Invariant: the answer is in [lo, hi], and cbase[hi+1] >= x if hi < nchunks.
  uint64_t lo = 0, hi = nchunks;
  while (lo < hi) {
    const uint64_t step = (hi - lo + 31) >> 5;
    const uint64_t p = lo + (uint64_t)lane * step;
    const unsigned m = __ballot_sync(0xffffffffu, p < hi && cbase[p + 1] >= x);
    if (m != 0) {
      const int j = __ffs(m) - 1;
      const uint64_t pj = lo + (uint64_t)j * step;
      lo = j ? pj - step + 1 : pj;
      hi = pj;
    } else {
      lo += (hi - 1 - lo) / step * step + 1;  // past the last probed chunk
    }
  }
  if (lo >= nchunks) return (int64_t)(n - 1);
  const uint64_t c = lo;
  double v = seg_sum_staged(s, c * kChunk, n, lane, buf);
  double inc = warp_iscan(v);
  const double base = cbase[c];
  const bool hit = base + inc >= x;
  const unsigned m = __ballot_sync(0xffffffffu, hit);
  if (m == 0) return (int64_t)min((c + 1) * (uint64_t)kChunk, n) - 1;
  const int L = __ffs(m) - 1;
  // lane L walks its segment
  int64_t r = 0;
  if (lane == L) {
    double run = base + (inc - v);
    const uint64_t st = c * kChunk + (uint64_t)L * kSeg;
    uint64_t i = st;
    r = -1;
    for (int q = 0; q < kSeg; ++q, ++i) {
      if (i >= n) break;
      float2 a = s[i];
      run += (double)a.x * a.x + (double)a.y * a.y;
      if (run >= x) { r = (int64_t)i; break; }
    }
    if (r < 0) r = (int64_t)min(st + kSeg, n) - 1;
  }
  return __shfl_sync(0xffffffffu, r, L);
}

__global__ void k_sample(const float2* __restrict__ s, uint64_t n, uint64_t nchunks, const double* __restrict__ cbase,
                         const double* __restrict__ u, int64_t nshots, int64_t* __restrict__ out) {
  pdl_begin();
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  __shared__ float2 stage[kThreads / 32][32][17];
  for (uint64_t k = warp; k < (uint64_t)nshots; k += nwarps) {
    const int64_t result = sample_one(s, n, nchunks, cbase, u[k], stage[threadIdx.x >> 5]);
    if (lane == 0) out[k] = result;
  }
}

// ------------------------------------------------- batched sampling ------
// Many states of any widths in three launches.  Each state's CDF is built and
// searched exactly as qs_sample does it (same chunking, scan order and
// search), and shot k of state t uses value k of seeds[t]'s uniform stream,
// so the shots equal qs_sample's with those uniforms.
struct SampleDesc {
  uint64_t state_off;  // first amplitude of the state
  uint64_t n;          // amplitudes (2^width)
  uint64_t nchunks;
  uint64_t chunk_off;  // prefix sum of nchunks
  uint64_t shot_off;   // prefix sum of shots
  uint64_t seed;
};

// last descriptor whose field `off` is <= g (descriptors sorted by it)
template <uint64_t SampleDesc::*F>
__device__ __forceinline__ int find_desc(const SampleDesc* __restrict__ d, int ns, uint64_t g) {
  int lo = 0, hi = ns - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (d[mid].*F <= g) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__global__ void k_chunk_sums_b(const float2* __restrict__ base, const SampleDesc* __restrict__ d, int ns,
                               uint64_t total_chunks, double* __restrict__ csum) {
  pdl_begin();
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  __shared__ float2 stage[kThreads / 32][32][17];
  for (uint64_t g = warp; g < total_chunks; g += nwarps) {
    const int t = find_desc<&SampleDesc::chunk_off>(d, ns, g);
    const SampleDesc D = d[t];
    const uint64_t c = g - D.chunk_off;
    double v = seg_sum_staged(base + D.state_off, c * kChunk, D.n, lane, stage[threadIdx.x >> 5]);
    v = warp_iscan(v);
    if (lane == 31) csum[g] = v;
  }
}

// one 1024-thread block per state; cbase of state t starts at chunk_off + t
__global__ void __launch_bounds__(kScanThreads, 1)
    k_chunk_scan_b(const double* __restrict__ csum, const SampleDesc* __restrict__ d, double* __restrict__ cbase) {
  pdl_begin();
  __shared__ double ws[32];
  __shared__ double carry;
  extern __shared__ double scan_smem[];
  const SampleDesc D = d[blockIdx.x];
  if (D.shot_off == d[blockIdx.x + 1].shot_off) return;  // no shots: nothing to scan (block-uniform)
  chunk_scan_block(csum + D.chunk_off, D.nchunks, cbase + D.chunk_off + blockIdx.x, ws, carry,
                   reinterpret_cast<ScanTile>(scan_smem));
}

__global__ void k_sample_b(const float2* __restrict__ base, const SampleDesc* __restrict__ d, int ns,
                           uint64_t total_shots, const double* __restrict__ cbase, int64_t* __restrict__ out) {
  pdl_begin();
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  __shared__ float2 stage[kThreads / 32][32][17];
  for (uint64_t g = warp; g < total_shots; g += nwarps) {
    const int t = find_desc<&SampleDesc::shot_off>(d, ns, g);
    const SampleDesc D = d[t];
    const double x = qs_seed_uniform_at(D.seed, g - D.shot_off);
    const int64_t result =
        sample_one(base + D.state_off, D.n, D.nchunks, cbase + D.chunk_off + t, x, stage[threadIdx.x >> 5]);
    if (lane == 0) out[g] = result;
  }
}

// ---------------------------------------------------- Pauli-sum terms ----
// (P_t psi)[i] = i^{|x&z|} (-1)^{popc(j & z)} psi[j], j = i ^ x, for the string
// with masks x, z.  A term's weight is therefore real or i times a real c_t.
// Terms are grouped by X mask: row i of a mask has the weight
// W_x(j) = sum_t c_t (-1)^{popc(j & z_t)} (FP64) on the one gathered psi[j].
//
// A thread holds 2*M amplitudes (qubit 0, and qubits 6 and 7 for M = 4), a
// gather being 16 bytes of which a warp reads 512 in a row.  The parity of the
// index bits outside the registers is taken once per term and thread, the rest
// of the sign is a bit of `pat`.  The masks come in four runs: real / imaginary
// weights, each with even then odd X masks (SWAP: the two amplitudes of a
// gather trade places).
template <class U>
struct alignas(8) PauliMask {
  U x;
  U hbit, hval;             // expectation: threads with (index & hbit) != hval skip the mask
  int32_t t0, tu, t1;       // terms [t0, t1), those before tu of equal sign in all registers
};
template <class U>
struct alignas(8) PauliTerm {
  double c;
  U z;                      // without the bits held in registers
  uint32_t pat;             // signs over the registers: bit 2m + e
};
struct PauliRuns { int r0, r1, i0, end, terms; };  // real even, real odd, imaginary even, imaginary odd

__device__ __forceinline__ uint32_t parity_bit(uint32_t v) { return (uint32_t)__popc(v) << 31; }
__device__ __forceinline__ uint32_t parity_bit(uint64_t v) { return (uint32_t)__popcll(v) << 31; }
__device__ __forceinline__ double flip_if(double v, uint32_t sign) {
  return __hiloint2double(__double2hiint(v) ^ (int)sign, __double2loint(v));
}

// The weights of one mask over a thread's amplitudes; returns whether they are
// all w[0].
template <int M, class U>
__device__ __forceinline__ bool mask_weights(const PauliMask<U>& P, const PauliTerm<U>* __restrict__ st, U j,
                                             double (&w)[2 * M]) {
  double w0 = 0.0;
  for (int t = P.t0; t < P.tu; ++t) w0 += flip_if(st[t].c, parity_bit((U)(j & st[t].z)));
  w[0] = w0;
  if (P.tu == P.t1) return true;
#pragma unroll
  for (int r = 1; r < 2 * M; ++r) w[r] = w0;
  for (int t = P.tu; t < P.t1; ++t) {
    const double c = flip_if(st[t].c, parity_bit((U)(j & st[t].z)));
    const uint32_t pat = st[t].pat;
#pragma unroll
    for (int r = 0; r < 2 * M; ++r) w[r] += flip_if(c, (pat << (31 - r)) & 0x80000000u);
  }
  return false;
}

template <int M, bool IMAG, bool SWAP, class U>
__device__ __forceinline__ void pauli_rows(const PauliMask<U>* __restrict__ sm, const PauliTerm<U>* __restrict__ st,
                                           int b, int e, const float4* __restrict__ x4, U t4, double2 (&acc)[2 * M]) {
  for (int k = b; k < e; ++k) {
    const PauliMask<U> P = sm[k];
    const U j4 = t4 ^ (P.x >> 1);
    float4 v[M];
#pragma unroll
    for (int m = 0; m < M; ++m) v[m] = x4[j4 ^ (U)(m << 5)];
    double w[2 * M];
    const bool same = mask_weights<M, U>(P, st, (U)(j4 << 1), w);
    auto add = [&](int r, double wr) {
      const double vx = (r & 1) ? v[r >> 1].z : v[r >> 1].x, vy = (r & 1) ? v[r >> 1].w : v[r >> 1].y;
      double2& a = acc[SWAP ? r ^ 1 : r];
      if (IMAG) {
        a.x = fma(-wr, vy, a.x);
        a.y = fma(wr, vx, a.y);
      } else {
        a.x = fma(wr, vx, a.x);
        a.y = fma(wr, vy, a.y);
      }
    };
    if (same) {
#pragma unroll
      for (int r = 0; r < 2 * M; ++r) add(r, w[0]);
    } else {
#pragma unroll
      for (int r = 0; r < 2 * M; ++r) add(r, w[r]);
    }
  }
}

// Re sum_i conj(psi_i) W psi_{i^x} over the rows the masks select.
template <int M, bool IMAG, bool SWAP, class U>
__device__ __forceinline__ void pauli_dot(const PauliMask<U>* __restrict__ sm, const PauliTerm<U>* __restrict__ st,
                                          int b, int e, const float4* __restrict__ x4, U t4,
                                          const double2 (&a)[2 * M], double& acc) {
  for (int k = b; k < e; ++k) {
    const PauliMask<U> P = sm[k];
    if (((t4 << 1) & P.hbit) != P.hval) continue;
    const U j4 = t4 ^ (P.x >> 1);
    float4 v[M];
#pragma unroll
    for (int m = 0; m < M; ++m) v[m] = x4[j4 ^ (U)(m << 5)];
    double w[2 * M];
    const bool same = mask_weights<M, U>(P, st, (U)(j4 << 1), w);
    double s[4] = {0.0, 0.0, 0.0, 0.0};   // chains of their own
#pragma unroll
    for (int r = 0; r < 2 * M; ++r) {
      const double2 p = a[SWAP ? r ^ 1 : r];
      const double vx = (r & 1) ? v[r >> 1].z : v[r >> 1].x, vy = (r & 1) ? v[r >> 1].w : v[r >> 1].y;
      if (same) {
        s[r & 1] = fma(IMAG ? p.y : p.x, vx, s[r & 1]);
        s[2 + (r & 1)] = fma(IMAG ? -p.x : p.y, vy, s[2 + (r & 1)]);
      } else {
        s[r & 3] = fma(w[r], IMAG ? fma(p.y, vx, -p.x * vy) : fma(p.x, vx, p.y * vy), s[r & 3]);
      }
    }
    acc = fma(same ? w[0] : 1.0, (s[0] + s[1]) + (s[2] + s[3]), acc);
  }
}

template <int M>
constexpr uint32_t pauli_regs() { return M == 4 ? 0xC1u : 0x01u; }

// The table of a Pauli sum, masks then terms, in shared memory.
template <class U>
__device__ __forceinline__ const PauliTerm<U>* pauli_stage(const uint32_t* __restrict__ table, PauliRuns R,
                                                           PauliMask<U>* sm) {
  const uint32_t words = (uint32_t)((sizeof(PauliMask<U>) * R.end + sizeof(PauliTerm<U>) * R.terms) / 4);
  uint32_t* d = reinterpret_cast<uint32_t*>(sm);
  for (uint32_t k = threadIdx.x; k < words; k += blockDim.x) d[k] = table[k];
  __syncthreads();
  return reinterpret_cast<const PauliTerm<U>*>(sm + R.end);
}

// out = H psi (complex64), accumulated in FP64 per amplitude; blockIdx.y is
// the vector.  S groups of a CTA's threads share its amplitudes, each taking a
// part of every run of masks.
//
// Bound by the FP32-to-FP64 conversions of the gathered amplitudes (16 lanes
// per clock and SM, two per mask and amplitude).  8 vectors of 20 qubits, 256
// random terms: 848 us; 3436 with one amplitude per thread and term (two
// 32-bit POPCs and six FP64 operations each).
template <int M, int S, class U>
__global__ void __launch_bounds__(kThreads, 3)
    k_pauli_apply(const float2* __restrict__ in, float2* __restrict__ out, uint64_t vstride,
                  const uint32_t* __restrict__ table, PauliRuns R, U nthr) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char pauli_smem[];
  constexpr int G = kThreads / S;
  __shared__ double2 part[S > 1 ? S - 1 : 1][S > 1 ? 2 * M : 1][S > 1 ? G : 1];
  auto* sm = reinterpret_cast<PauliMask<U>*>(pauli_smem);
  const PauliTerm<U>* st = pauli_stage(table, R, sm);
  const float4* x4 = reinterpret_cast<const float4*>(in + blockIdx.y * vstride);
  float4* o4 = reinterpret_cast<float4*>(out + blockIdx.y * vstride);
  const int s = threadIdx.x / G;
  auto cut = [&](int b, int e, int k) { return b + (e - b) * k / S; };
  const U g = (U)blockIdx.x * G + threadIdx.x % G;
  const bool has = g < nthr;
  const U t4 = (g >> 5) * (U)(32 * M) + (g & 31);
  double2 acc[2 * M];
#pragma unroll
  for (int r = 0; r < 2 * M; ++r) acc[r] = make_double2(0.0, 0.0);
  if (has) {
    pauli_rows<M, false, false, U>(sm, st, cut(0, R.r0, s), cut(0, R.r0, s + 1), x4, t4, acc);
    pauli_rows<M, false, true, U>(sm, st, cut(R.r0, R.r1, s), cut(R.r0, R.r1, s + 1), x4, t4, acc);
    pauli_rows<M, true, false, U>(sm, st, cut(R.r1, R.i0, s), cut(R.r1, R.i0, s + 1), x4, t4, acc);
    pauli_rows<M, true, true, U>(sm, st, cut(R.i0, R.end, s), cut(R.i0, R.end, s + 1), x4, t4, acc);
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
        const double2 v = part[q][r][threadIdx.x];
        acc[r].x += v.x;
        acc[r].y += v.y;
      }
    }
  }
  if (!has) return;
#pragma unroll
  for (int m = 0; m < M; ++m)
    o4[t4 + (U)(32 * m)] = make_float4((float)acc[2 * m].x, (float)acc[2 * m].y, (float)acc[2 * m + 1].x,
                                       (float)acc[2 * m + 1].y);
}

// <psi|H|psi> partials, one per CTA.  Rows i and i ^ x of a mask contribute
// the same real part, so where x has a bit that a whole warp shares, one of
// the two is evaluated and the weights are doubled on the host.
//
// Bound as k_pauli_apply by conversions: 24 qubits, 64 random terms
// 460 us; 1535 with one amplitude per thread and term.
template <int M, int S, class U>
__global__ void __launch_bounds__(kThreads, 3)
    k_pauli_expect(const float2* __restrict__ psi, const uint32_t* __restrict__ table, PauliRuns R, U nthr,
                   double* __restrict__ partial) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char pauli_smem[];
  constexpr int G = kThreads / S;
  auto* sm = reinterpret_cast<PauliMask<U>*>(pauli_smem);
  const PauliTerm<U>* st = pauli_stage(table, R, sm);
  const float4* x4 = reinterpret_cast<const float4*>(psi);
  const int s = threadIdx.x / G;
  auto cut = [&](int b, int e, int k) { return b + (e - b) * k / S; };
  double acc = 0.0;
  for (U g = (U)blockIdx.x * G + threadIdx.x % G; g < nthr; g += (U)gridDim.x * G) {
    const U t4 = (g >> 5) * (U)(32 * M) + (g & 31);
    double2 a[2 * M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const float4 v = x4[t4 + (U)(32 * m)];
      a[2 * m] = make_double2(v.x, v.y);
      a[2 * m + 1] = make_double2(v.z, v.w);
    }
    pauli_dot<M, false, false, U>(sm, st, cut(0, R.r0, s), cut(0, R.r0, s + 1), x4, t4, a, acc);
    pauli_dot<M, false, true, U>(sm, st, cut(R.r0, R.r1, s), cut(R.r0, R.r1, s + 1), x4, t4, a, acc);
    pauli_dot<M, true, false, U>(sm, st, cut(R.r1, R.i0, s), cut(R.r1, R.i0, s + 1), x4, t4, a, acc);
    pauli_dot<M, true, true, U>(sm, st, cut(R.i0, R.end, s), cut(R.i0, R.end, s + 1), x4, t4, a, acc);
  }
  acc = block_sum(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc;
}

struct PauliUpload { const uint32_t* table; PauliRuns runs; size_t bytes; };

// The largest table: 1024 terms of as many masks.  Up to 32 KiB of it, with the
// static arrays, need no raised limit.
template <class U>
constexpr size_t pauli_largest() { return 1024 * (sizeof(PauliMask<U>) + sizeof(PauliTerm<U>)); }

// Builds the table in scratch after `offset` bytes.  `regs`: the index bits a
// thread holds in registers; `halve`: choose one of the rows i and i ^ x.
template <class U>
PauliUpload pauli_upload(qs_context* h, size_t offset, int n, const uint64_t* x, const uint64_t* z, const double* c,
                         int nterms, uint32_t regs, bool halve) {
  QS_CHECK_ARG(nterms >= 1, "need at least one Pauli term");
  QS_CHECK_ARG(x && z && c, "term pointers are null");
  const uint64_t lim = (1ull << n) - 1ull;
  std::vector<int> order(nterms);
  for (int k = 0; k < nterms; ++k) {
    QS_CHECK_ARG((x[k] & ~lim) == 0 && (z[k] & ~lim) == 0, "Pauli mask has bits beyond n_qubits");
    order[k] = k;
  }
  // real weight: |x & z| even; run 2 * imaginary + odd X mask
  auto run_of = [&](int k) { return 2 * (__builtin_popcountll(x[k] & z[k]) & 1) + (int)(x[k] & 1); };
  // signs of the amplitudes that a thread reads for its outputs: bit 2m + e
  auto pattern = [&](int k) {
    uint32_t pat = 0;
    for (int r = 0; r < 8; ++r) {
      const uint64_t j = (uint64_t)(r & 1) | (((uint64_t)(r >> 1) << 6) ^ (x[k] & regs & ~1ull));
      pat |= (uint32_t)(__builtin_popcountll(j & z[k] & regs) & 1) << r;
    }
    return pat & (regs == 0x01u ? 0x3u : 0xFFu);
  };
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    if (run_of(a) != run_of(b)) return run_of(a) < run_of(b);
    if (x[a] != x[b]) return x[a] < x[b];
    return (pattern(a) == 0) > (pattern(b) == 0);
  });
  std::vector<PauliMask<U>> masks;
  std::vector<PauliTerm<U>> terms;
  int ends[4] = {0, 0, 0, 0};
  for (int u = 0; u < nterms;) {
    const int a = order[u], run = run_of(a);
    PauliMask<U> P{(U)x[a], 0, 0, u, u, u};
    const uint64_t warp_bits = x[a] & ~(uint64_t)(regs | 0x3Eu);
    if (halve && warp_bits) {
      P.hbit = (U)(warp_bits & (~warp_bits + 1));
      P.hval = (masks.size() & 1) ? P.hbit : 0;   // alternate, so that no CTA has all the work
    }
    const double scale = P.hbit ? 2.0 : 1.0;
    for (; u < nterms && run_of(order[u]) == run && x[order[u]] == x[a]; ++u) {
      const int k = order[u];
      const int ny = __builtin_popcountll(x[k] & z[k]) & 3;   // i^ny = +-1 or +-i
      const uint32_t pat = pattern(k);
      terms.push_back(PauliTerm<U>{(ny >= 2 ? -c[k] : c[k]) * scale, (U)z[k] & ~(U)regs, pat});
      if (pat == 0) P.tu = u + 1;
    }
    P.t1 = u;
    masks.push_back(P);
    for (int r = run; r < 4; ++r) ends[r] = (int)masks.size();
  }
  const size_t mb = sizeof(PauliMask<U>) * masks.size(), tb = sizeof(PauliTerm<U>) * terms.size();
  std::vector<char> host(mb + tb);
  std::memcpy(host.data(), masks.data(), mb);
  std::memcpy(host.data() + mb, terms.data(), tb);
  char* d = (char*)h->scratch_get(offset + mb + tb) + offset;
  // From pageable memory the copy returns once it has been staged, so the
  // host vector may go out of scope afterwards.
  QS_CUDA(cudaMemcpyAsync(d, host.data(), mb + tb, cudaMemcpyHostToDevice, h->stream));
  return {(const uint32_t*)d, {ends[0], ends[1], ends[2], ends[3], nterms}, mb + tb};
}

template <int M, int S, class U>
void pauli_apply(qs_context* h, const float2* in, float2* out, uint64_t vstride, int nb, int n, const uint64_t* x,
                 const uint64_t* z, const double* c, int nterms) {
  const PauliUpload T = pauli_upload<U>(h, 0, n, x, z, c, nterms, pauli_regs<M>(), false);
  const uint64_t nthr = (1ull << n) / (2 * M), per = kThreads / S;
  if (T.bytes > 32 * 1024) qs_smem_limit(h, (const void*)k_pauli_apply<M, S, U>, pauli_largest<U>());
  // a CTA holds one vector: no more threads than that has work for
  const unsigned threads = S == 1 ? (unsigned)std::min<uint64_t>(nthr, kThreads) : kThreads;
  qs_launch_pdl(h, k_pauli_apply<M, S, U>, dim3((unsigned)((nthr + per - 1) / per), nb), dim3(threads), T.bytes, in, out,
                vstride, T.table, T.runs, (U)nthr);
  qs_after_launch(h, "k_pauli_apply");
}

}  // namespace

// out_b = H in_b (complex64, FP64 sums) for nb vectors `vstride` amplitudes
// apart; 16-byte aligned, not aliased.
void qs_pauli_apply(qs_context* h, const float2* in, float2* out, uint64_t vstride, int nb, int n, const uint64_t* x,
                    const uint64_t* z, const double* c, int nterms) {
  // Eight amplitudes per thread, or two and the masks over 8 groups of threads:
  // eight cost less in all, but a thread goes through every term (2.4 us + 0.26 per
  // term while the SMs are not full), where two share the terms out and launch four
  // times the threads for each of eight groups (2 us + (8 + 0.25 per term) for each
  // 2^18 amplitudes).  Measured on both sides of the line, us for two / eight: 2^16
  // amplitudes, 8 terms 4.5 / 4.7, 24 terms 6.3 / 8.4; 2^17 amplitudes, 24 terms 9.6 /
  // 8.9, 64 terms 16 / 19; 15 vectors of 14 qubits, 64 terms 27 / 19; 1024 vectors of 8
  // qubits, 64 terms 24.6 / 21.5 (40 in CTAs of 256 threads, of which 32 had work).
  const double amps = std::ldexp((double)nb, n - 16);
  const bool eight = n >= 8 && (amps >= 4.0 || nterms <= 8.0 * amps * amps);
  if (n > 32) pauli_apply<4, 1, uint64_t>(h, in, out, vstride, nb, n, x, z, c, nterms);
  else if (eight) pauli_apply<4, 1, uint32_t>(h, in, out, vstride, nb, n, x, z, c, nterms);
  else pauli_apply<1, 8, uint32_t>(h, in, out, vstride, nb, n, x, z, c, nterms);
}

namespace {

template <class F>
void reduce_to(qs_context* h, F f, uint64_t items, double* d_out, int mode, double* d_partial) {
  Slicing sl = slice(items);
  qs_launch_pdl(h, k_reduce<F>, dim3(sl.nb), dim3(kThreads), 0, f, items, sl.per, d_partial);
  qs_after_launch(h, "k_reduce");
  qs_launch_pdl(h, k_final, dim3(1), dim3(1024), 0, d_partial, sl.nb, d_out, mode);
  qs_after_launch(h, "k_final");
}

// scratch layout for reductions: [0, 16) two doubles out; [64, ...) partials
double* red_out(qs_context* h) { return (double*)h->scratch_get(64 + 8 * kMaxBlocks); }
double* red_part(qs_context* h) { return (double*)((char*)h->scratch_get(64 + 8 * kMaxBlocks) + 64); }

// Leaves <psi|H|psi> in red_out.  The slicing depends on n only.
template <int M, int S, class U>
void pauli_expect(qs_context* h, const float2* psi, int n, const uint64_t* x, const uint64_t* z, const double* c,
                  int nterms) {
  const PauliUpload T = pauli_upload<U>(h, 64 + 8 * kMaxBlocks, n, x, z, c, nterms, pauli_regs<M>(), true);
  const uint64_t nthr = (1ull << n) / (2 * M), per = kThreads / S;
  const int nb = (int)std::min<uint64_t>((nthr + per - 1) / per, kPauliBlocks);
  if (T.bytes > 32 * 1024) qs_smem_limit(h, (const void*)k_pauli_expect<M, S, U>, pauli_largest<U>());
  qs_launch_pdl(h, k_pauli_expect<M, S, U>, dim3(nb), dim3(kThreads), T.bytes, psi, T.table, T.runs, (U)nthr, red_part(h));
  qs_after_launch(h, "k_pauli_expect");
  qs_launch_pdl(h, k_final, dim3(1), dim3(1024), 0, red_part(h), nb, red_out(h), 0);
  qs_after_launch(h, "k_final");
}

double fetch_scalar(qs_context* h, const double* d) {
  double* pin = h->pinned_get(64);
  QS_CUDA(cudaMemcpyAsync(pin, d, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  QS_CUDA(cudaStreamSynchronize(h->stream));
  return pin[0];
}

}  // namespace

extern "C" {

int qs_norm2(qs_handle_t h, const void* state, int n, double* out) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(out != nullptr, "out is null");
  double* o = red_out(h);
  reduce_to(h, FNorm{(const float4*)state}, (1ull << n) / 2, o, 0, red_part(h));
  *out = fetch_scalar(h, o);
  QS_API_END(h)
}

int qs_renorm(qs_handle_t h, void* state, int n) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  double* o = red_out(h);
  const uint64_t nvec = (1ull << n) / 2;
  reduce_to(h, FNorm{(const float4*)state}, nvec, o, 1, red_part(h));
  qs_launch_pdl(h, k_scale, dim3(qs_blocks_for(h, nvec, kThreads)), dim3(kThreads), 0, (float4*)state, nvec, o);
  qs_after_launch(h, "k_scale");
  QS_API_END(h)
}

int qs_probs(qs_handle_t h, const void* state, int n, float* probs) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(probs != nullptr && ((uintptr_t)probs & 7u) == 0, "probs must be a non-null 8-byte aligned pointer");
  const uint64_t nvec = (1ull << n) / 2;
  qs_launch_pdl(h, k_probs, dim3(qs_blocks_for(h, nvec, kThreads)), dim3(kThreads), 0, (const float4*)state, (float2*)probs, nvec);
  qs_after_launch(h, "k_probs");
  QS_API_END(h)
}

int qs_probs_n(qs_handle_t h, const void* states, int64_t n_amps, float* probs) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  QS_CHECK_ARG(states && ((uintptr_t)states & 15u) == 0, "states must be a 16-byte aligned device pointer");
  QS_CHECK_ARG(probs != nullptr && ((uintptr_t)probs & 7u) == 0, "probs must be a non-null 8-byte aligned pointer");
  QS_CHECK_ARG(n_amps >= 0 && (n_amps & 1) == 0, "n_amps must be even and >= 0");
  const uint64_t nvec = (uint64_t)n_amps / 2;
  if (nvec) {
    qs_launch_pdl(h, k_probs, dim3(qs_blocks_for(h, nvec, kThreads)), dim3(kThreads), 0, (const float4*)states, (float2*)probs, nvec);
    qs_after_launch(h, "k_probs");
  }
  QS_API_END(h)
}

int qs_measure(qs_handle_t h, void* state, int n, int t, double u, int* outcome) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  qs_check_qubit(t, n, "target");
  QS_CHECK_ARG(outcome != nullptr, "outcome is null");
  double* o = red_out(h);
  const uint64_t nvec = (1ull << n) / 2;
  reduce_to(h, FP0{(const float4*)state, t}, nvec, o, 0, red_part(h));
  // the kernel writes the outcome straight into the handle's pinned buffer
  // (page-locked host memory is addressable from the device under unified
  // addressing), so no copy is queued between the kernel and the synchronise
  int* pin = reinterpret_cast<int*>(h->pinned_get(64));
  qs_launch_pdl(h, k_collapse, dim3(qs_blocks_for(h, nvec, kThreads)), dim3(kThreads), 0, (float4*)state, nvec, t, u, o, pin);
  qs_after_launch(h, "k_collapse");
  QS_CUDA(cudaStreamSynchronize(h->stream));
  *outcome = *pin;
  QS_API_END(h)
}

int qs_expect_z(qs_handle_t h, const void* state, int n, uint64_t zmask, double* out) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(out != nullptr, "out is null");
  double* o = red_out(h);
  reduce_to(h, FZ{(const float4*)state, zmask}, (1ull << n) / 2, o, 0, red_part(h));
  *out = fetch_scalar(h, o);
  QS_API_END(h)
}

int qs_expect_pauli_sum(qs_handle_t h, const void* state, int n, const uint64_t* x, const uint64_t* z,
                        const double* c, int nterms, double* out) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(out != nullptr, "out is null");
  QS_CHECK_ARG(nterms >= 1 && nterms <= 1024, "n_terms must be in [1, 1024]");
  // as qs_pauli_apply; one vector fills the SMs from 18 qubits on (shots and an
  // expectation value of 64 terms, two against eight amplitudes per thread: 82 us /
  // 93 at 17 qubits, 94 / 92 at 18, 118 / 93 at 19)
  if (n > 32) pauli_expect<4, 1, uint64_t>(h, (const float2*)state, n, x, z, c, nterms);
  else if (n >= 18) pauli_expect<4, 1, uint32_t>(h, (const float2*)state, n, x, z, c, nterms);
  else pauli_expect<1, 8, uint32_t>(h, (const float2*)state, n, x, z, c, nterms);
  double* o = red_out(h);
  *out = fetch_scalar(h, o);
  QS_API_END(h)
}

int qs_apply_pauli_sum(qs_handle_t h, const void* psi, void* out, int n, const uint64_t* x, const uint64_t* z,
                       const double* c, int nterms) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(psi, n);
  qs_check_state(out, n);
  QS_CHECK_ARG(psi != out, "out must not alias psi");
  QS_CHECK_ARG(nterms >= 1 && nterms <= 1024, "n_terms must be in [1, 1024]");
  qs_pauli_apply(h, (const float2*)psi, (float2*)out, 0, 1, n, x, z, c, nterms);
  QS_API_END(h)
}


// Per device, once: the scan kernels' shared-memory limit raised to their
// tile, and the chunk-sum kernels' grids sized to one wave of the CTAs that
// fit on an SM at once (registers and 34 KiB of staging each decide how many),
// so that no second wave runs on part of the SMs while the rest idle.
struct SampleLaunch {
  int sums_per_sm, sums_b_per_sm;
};
static SampleLaunch sample_launch(qs_context* h) {
  static std::mutex mu;
  static std::map<int, SampleLaunch> by_device;
  std::lock_guard<std::mutex> lk(mu);
  auto f = by_device.find(h->device);
  if (f != by_device.end()) return f->second;
  QS_CUDA(cudaFuncSetAttribute(k_chunk_scan, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScanSmem));
  QS_CUDA(cudaFuncSetAttribute(k_chunk_scan_b, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScanSmem));
  SampleLaunch L{0, 0};
  QS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&L.sums_per_sm, k_chunk_sums, kThreads, 0));
  QS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&L.sums_b_per_sm, k_chunk_sums_b, kThreads, 0));
  if (L.sums_per_sm < 1 || L.sums_b_per_sm < 1) throw qs_error(QS_ERR_CUDA, "chunk-sum kernel does not fit on an SM");
  by_device[h->device] = L;
  return L;
}

int qs_sample_batched(qs_handle_t h, const void* states, int n_states, const int32_t* widths,
                      const int64_t* state_offsets, const int64_t* shots, const uint64_t* seeds, int64_t* out) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  QS_CHECK_ARG(n_states >= 0, "n_states must be >= 0");
  if (n_states == 0) return QS_OK;
  QS_CHECK_ARG(states && widths && state_offsets && shots && seeds, "null batch descriptor");
  QS_CHECK_ARG(((uintptr_t)states & 15u) == 0, "states must be 16-byte aligned");
  // descriptors, plus one sentinel holding the totals
  std::vector<SampleDesc> desc(n_states + 1);
  uint64_t chunks = 0, nshots = 0;
  for (int t = 0; t < n_states; ++t) {
    QS_CHECK_ARG(widths[t] >= 1 && widths[t] <= QS_MAX_QUBITS, "state width out of range");
    QS_CHECK_ARG(state_offsets[t] >= 0 && shots[t] >= 0, "negative offset or shot count");
    const uint64_t N = 1ull << widths[t];
    SampleDesc& D = desc[t];
    D.state_off = (uint64_t)state_offsets[t];
    D.n = N;
    D.nchunks = (N + kChunk - 1) / kChunk;
    D.chunk_off = chunks;
    D.shot_off = nshots;
    D.seed = seeds[t];
    chunks += D.nchunks;
    nshots += (uint64_t)shots[t];
  }
  desc[n_states] = SampleDesc{0, 0, 0, chunks, nshots, 0};
  if (nshots == 0) return QS_OK;
  QS_CHECK_ARG(out != nullptr, "out pointer is null");
  const size_t dbytes = ((desc.size() * sizeof(SampleDesc)) + 255) & ~size_t(255);
  char* sc = static_cast<char*>(h->scratch_get(dbytes + sizeof(double) * (2 * chunks + n_states)));
  auto* d_desc = reinterpret_cast<SampleDesc*>(sc);
  double* csum = reinterpret_cast<double*>(sc + dbytes);
  double* cbase = csum + chunks;
  QS_CUDA(cudaMemcpyAsync(d_desc, desc.data(), desc.size() * sizeof(SampleDesc), cudaMemcpyHostToDevice, h->stream));
  const int wpb = kThreads / 32;
  const SampleLaunch L = sample_launch(h);
  qs_launch_pdl(h, k_chunk_sums_b, dim3(qs_blocks_for(h, chunks * 32, kThreads, L.sums_b_per_sm)), dim3(kThreads), 0, 
      (const float2*)states, d_desc, n_states, chunks, csum);
  qs_after_launch(h, "k_chunk_sums_b");
  qs_launch_pdl(h, k_chunk_scan_b, dim3((unsigned)n_states), dim3(kScanThreads), kScanSmem, csum, d_desc, cbase);
  qs_after_launch(h, "k_chunk_scan_b");
  const uint64_t blocks = std::min<uint64_t>((nshots + wpb - 1) / wpb, (uint64_t)h->sm_count * 16);
  qs_launch_pdl(h, k_sample_b, dim3((unsigned)blocks), dim3(kThreads), 0, (const float2*)states, d_desc, n_states, nshots, cbase,
                                                           out);
  qs_after_launch(h, "k_sample_b");
  QS_API_END(h)
}

int qs_sample(qs_handle_t h, const void* state, int n, const double* u, int64_t nshots, int64_t* out) {
  QS_REQUIRE_HANDLE(h);
  QS_API_BEGIN
  qs_check_state(state, n);
  QS_CHECK_ARG(nshots >= 0, "n_shots must be >= 0");
  if (nshots == 0) return QS_OK;
  QS_CHECK_ARG(u != nullptr && out != nullptr, "u/out pointer is null");
  const uint64_t N = 1ull << n;
  const uint64_t nchunks = (N + kChunk - 1) / kChunk;
  double* base = (double*)h->scratch_get(sizeof(double) * (2 * nchunks + 1));
  double* csum = base;
  double* cbase = base + nchunks;
  const int wpb = kThreads / 32;
  const SampleLaunch L = sample_launch(h);
  qs_launch_pdl(h, k_chunk_sums, dim3(qs_blocks_for(h, nchunks * 32, kThreads, L.sums_per_sm)), dim3(kThreads), 0, (const float2*)state, N,
                                                                                     nchunks, csum);
  qs_after_launch(h, "k_chunk_sums");
  qs_launch_pdl(h, k_chunk_scan, dim3(1), dim3(kScanThreads), kScanSmem, csum, nchunks, cbase);
  qs_after_launch(h, "k_chunk_scan");
  const uint64_t blocks = std::min<uint64_t>(((uint64_t)nshots + wpb - 1) / wpb, (uint64_t)h->sm_count * 16);
  qs_launch_pdl(h, k_sample, dim3((unsigned)blocks), dim3(kThreads), 0, (const float2*)state, N, nchunks, cbase, u, nshots, out);
  qs_after_launch(h, "k_sample");
  QS_API_END(h)
}

}  // extern "C"
