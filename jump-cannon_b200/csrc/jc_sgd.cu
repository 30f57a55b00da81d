// SGD pivot-stress layout on B200: "sgd-stress-gpu" (Jacobi move-self) and
// "sgd-stress" (per-pair scatter that moves both endpoints).
//
// Reference behaviour (paths in the jump-cannon repo):
//   crates/graph-compute/src/engines/sgd_stress.rs       settings, SplitMix64,
//       select_pivots :143-175, step :275-318, anneal_eta :324-334,
//       sgd_pair_update :340-366, bfs_distances :372-394
//   crates/graph-compute/src/engines/sgd_stress_gpu.rs   init :165-366, step :368-449
//   crates/graph-compute/src/shaders/sgd_stress.wgsl     sgd_step :34-62
//
// The max-min pivot choice and its per-pivot BFS stay on the host at init, as in
// the reference; random pivots take a device multi-source BFS. Distances are
// stored pivot-major
// (dist[t * n + i]) so that the threads of a warp, one node each, read one
// contiguous row per pivot; u16 when every finite distance fits, else u32,
// with the all-ones value as "unreachable".
//
// Jacobi sweep (sgd_stress.wgsl): node i walks its k pivots in order against
// the start-of-sweep positions; pivot positions are staged in shared memory.
// Bit-identical to the shader's arithmetic (IEEE ops in source order).
//
// Per-pair scatter (sgd_stress.rs semantics on a GPU): the CPU engine draws
// n (node, pivot) samples per sweep from one SplitMix64 stream and moves both
// endpoints sequentially. SplitMix64 is counter based, so sample q of the run
// is computed directly from the stream position; the GPU draws exactly the
// reference's samples. A sweep is split into batches; inside a batch every
// pair update is evaluated against the batch-start positions and the two
// endpoint moves are accumulated in 64-bit fixed point with integer atomics
// (order-independent, so the result is deterministic). Each node then moves
// by the mean of its accumulated moves: a pivot takes part in ~n/(k*batches)
// pairs per batch and summing them would overshoot, averaging keeps each
// pivot's move the size of one pair update. Like the CPU engine it is a
// stochastic method: from the same seed it does not follow the sequential
// trajectory, and it is judged by the stress it converges to.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "jc_common.h"
#include "jc_engine.h"
#include "jc_exact.cuh"
#include "jc_launch.cuh"
#include "jc_params.h"
#include "jc_pool.h"

namespace jc {
namespace sgd {

constexpr uint32_t UNREACH = 0xFFFFFFFFu;
constexpr double FIX_SCALE = 4294967296.0;  // 2^32: fixed-point scale of pair moves

__device__ __forceinline__ float len3(float x, float y, float z) {
  return __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z)));
}

__device__ __forceinline__ uint64_t smix(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Threads a block of the sweep and of the search's levels: small enough that the
// nodes of a small graph spread over the SMs, large enough that an SM's blocks share
// the schedulers evenly. B200, us a step with 100 pivots at 64 / 128 / 256: 5,000
// nodes 14.4 / 12.3 / 14.4, 30,000 16.4 / 16.3 / 14.4, 50,000 18.5 / 18.5 / 20.5, 70,000 22.5
// / 20.5 / 20.5, 90,000 24.6 / 24.6 / 26.6, 140,000 32.8 / 32.8 / 32.7, 200,000 44.2 / 43.0 /
// 43.6, 250,000 53.3 / 51.7 / 51.2. Binds differ by 2 % at most.
constexpr uint32_t NODE_THREADS = 128;

// Node i's term with the pivot at q, hop distance d and mu = min(1, eta / d^2):
// the general operations (any f32 input).
__device__ __forceinline__ void jacobi_term(float& px, float& py, float& pz, const float4 q, float d, float mu) {
  const float ex = __fsub_rn(px, q.x), ey = __fsub_rn(py, q.y), ez = __fsub_rn(pz, q.z);
  const float mag = fmaxf(len3(ex, ey, ez), 1e-6f);
  const float r = __fdiv_rn(__fmul_rn(mu, __fsub_rn(mag, d)), mag);
  px = __fsub_rn(px, __fmul_rn(r, ex));
  py = __fsub_rn(py, __fmul_rn(r, ey));
  pz = __fsub_rn(pz, __fmul_rn(r, ez));
}

// The same term where root and quotient may come from jc_exact.cuh. Below
// 1e-12 the squared distance's root is not exact, but it is under the 1e-6
// clamp (or NaN, which fmaxf drops) as the exact one is.
__device__ __forceinline__ void jacobi_term_in_range(float& px, float& py, float& pz, const float4 q, float d,
                                                     float mu, bool use) {
  const float ex = __fsub_rn(px, q.x), ey = __fsub_rn(py, q.y), ez = __fsub_rn(pz, q.z);
  const float s = __fadd_rn(__fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey)), __fmul_rn(ez, ez));
  const float mag = fmaxf(dev::sqrt_in_range(s), 1e-6f);
  const float r = dev::div_in_range(__fmul_rn(mu, __fsub_rn(mag, d)), mag);
  if (use) {  // (the three subtractions alone are predicated: no branch in the chain)
    px = __fsub_rn(px, __fmul_rn(r, ex));
    py = __fsub_rn(py, __fmul_rn(r, ey));
    pz = __fsub_rn(pz, __fmul_rn(r, ez));
  }
}

// Where that holds: mu >= 2^-44 (eta >= JACOBI_ETA_LO, d < JACOBI_MU_MAX), since
// |mag - d| is 0 or at least 2^-25 of max(mag, 1), so that neither the quotient
// nor its remainders underflow; and every coordinate of the pivots and of the
// node within JACOBI_POS_HI at the sweep's start. A term moves the node along
// its line with the pivot to a distance between mag and d, so its coordinates
// stay within JACOBI_POS_HI + d + rounding and squared distances under 2^60.
constexpr float JACOBI_ETA_LO = 9.5367431640625e-7f;  // 2^-20
constexpr uint32_t JACOBI_MU_MAX = 4096u;
constexpr float JACOBI_POS_HI = 1.34217728e8f;        // 2^27
__device__ __forceinline__ bool jacobi_pos_ok(const float4 p) {
  return fabsf(p.x) <= JACOBI_POS_HI && fabsf(p.y) <= JACOBI_POS_HI && fabsf(p.z) <= JACOBI_POS_HI;
}
constexpr uint32_t JACOBI_PF = 8;

// (unreachable, all ones, and the node itself, 0, are skipped)
template <typename D>
__device__ __forceinline__ bool jacobi_skipped(D dv) {
  return (D)(dv - (D)1) >= (D)~(D)1;
}

// Pivot positions and the (mu, d) table into shared memory; whether the
// in-range terms hold as far as these decide it.
__device__ __forceinline__ bool jacobi_stage(float4* piv, float2* mu_tab, const float4* __restrict__ pin,
                                             const uint32_t* __restrict__ pivots, uint32_t k, uint32_t mu_len,
                                             float eta) {
  bool ok = mu_len != 0u && eta >= JACOBI_ETA_LO;
  for (uint32_t t = threadIdx.x; t < k; t += blockDim.x) {
    const float4 q = pin[pivots[t]];
    ok = ok && jacobi_pos_ok(q);
    piv[t] = q;
  }
  for (uint32_t du = threadIdx.x; du < mu_len; du += blockDim.x) {
    const float d = (float)du;
    mu_tab[du] = make_float2(fminf(1.0f, __fmul_rn(__fdiv_rn(1.0f, __fmul_rn(d, d)), eta)), d);
  }
  return __syncthreads_and(ok);
}

// One Jacobi sweep (sgd_stress.wgsl:34-62); eta comes from the host-computed
// schedule table at the device's sweep counter. The position update is a
// serial chain over the pivots, k links long; a sweep is bound by the
// instructions of the chain where nodes fill the GPU and by its latency where
// they do not, not by the n k 2 B of distances. So:
// - mu = min(1, eta / d^2) depends only on the hop distance d and the sweep's
//   eta and is tabulated beside d for d < mu_len (the same operations, once
//   per block), which takes a division and a conversion out of a link;
// - the root and the quotient come without range tests and calls, correctly
//   rounded both (jc_exact.cuh): bit-identical to the general operations;
// - the next JACOBI_PF distances are in flight during a group's links, and a
//   skipped pivot only predicates the three subtractions, so a link holds no
//   branch.
// About 47 instructions a link, 71 % of issue slots used at 250,000 nodes.
// B200, us a step with 200 pivots, before and after: 500 x 500 grid 135 -> 98;
// random geometric graphs of 200,000 nodes 119 -> 84, of 70,000 55 -> 35; of
// 30,011 with 100 pivots 29 -> 14. Two nodes per thread in packed f32
// operations gave 95 (grid) but for the moves it needs, and was not kept.
template <typename D>
__global__ void __launch_bounds__(NODE_THREADS)
k_jacobi(const float4* __restrict__ pin, float4* __restrict__ pout, const uint32_t* __restrict__ pivots,
         const D* __restrict__ dist, uint32_t n, uint32_t k, const float* __restrict__ eta_table, uint32_t n_eta,
         const uint32_t* __restrict__ sweep_ctr, uint32_t mu_len) {
  extern __shared__ float4 piv[];
  float2* mu_tab = reinterpret_cast<float2*>(piv + k);  // (mu, d)
  const uint32_t sw = *sweep_ctr;
  const float eta = eta_table[sw < n_eta ? sw : n_eta - 1];
  const bool block_ok = jacobi_stage(piv, mu_tab, pin, pivots, k, mu_len, eta);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 p4 = pin[i];
  float px = p4.x, py = p4.y, pz = p4.z;
  if (!block_ok || !jacobi_pos_ok(p4)) {
    for (uint32_t t0 = 0; t0 < k; t0 += JACOBI_PF) {
      D dv[JACOBI_PF];
#pragma unroll
      for (uint32_t u = 0; u < JACOBI_PF; ++u) dv[u] = t0 + u < k ? dist[(size_t)(t0 + u) * n + i] : (D)0;
#pragma unroll
      for (uint32_t u = 0; u < JACOBI_PF; ++u) {
        if (jacobi_skipped(dv[u])) continue;
        const float d = (float)dv[u];
        jacobi_term(px, py, pz, piv[t0 + u], d, fminf(1.0f, __fmul_rn(__fdiv_rn(1.0f, __fmul_rn(d, d)), eta)));
      }
    }
    pout[i] = make_float4(px, py, pz, 0.0f);
    return;
  }
  const uint32_t top = mu_len - 1u;
  const D* row = dist;  // the next group's first row
  uint32_t t = 0;
  D nx[JACOBI_PF];
#pragma unroll
  for (uint32_t u = 0; u < JACOBI_PF; ++u) nx[u] = u < k ? (row + (size_t)u * n)[i] : (D)0;
  for (; t + JACOBI_PF <= k; t += JACOBI_PF) {
    D dv[JACOBI_PF];
    row += (size_t)JACOBI_PF * n;
#pragma unroll
    for (uint32_t u = 0; u < JACOBI_PF; ++u) {
      dv[u] = nx[u];
      nx[u] = t + JACOBI_PF + u < k ? (row + (size_t)u * n)[i] : (D)0;
    }
#pragma unroll
    for (uint32_t u = 0; u < JACOBI_PF; ++u) {
      const float2 md = mu_tab[min((uint32_t)dv[u], top)];
      jacobi_term_in_range(px, py, pz, piv[t + u], md.y, md.x, !jacobi_skipped(dv[u]));
    }
  }
#pragma unroll
  for (uint32_t u = 0; u < JACOBI_PF; ++u) {
    if (t + u >= k) break;
    const float2 md = mu_tab[min((uint32_t)nx[u], top)];
    jacobi_term_in_range(px, py, pz, piv[t + u], md.y, md.x, !jacobi_skipped(nx[u]));
  }
  pout[i] = make_float4(px, py, pz, 0.0f);
}

// A sweep's n samples, drawn in one pass: sample q = sweep * n + t is (node i,
// pivot j, hop distance as f32 bits; 0 for a skipped pair: the node itself, or
// unreachable). They do not depend on the positions, and drawing them inside a
// batch put two 64-bit remainders and a cache-missing distance read into each
// batch's chain of round trips.
template <typename D>
__global__ void __launch_bounds__(256)
k_pairs_draw(uint4* __restrict__ samples, const uint32_t* __restrict__ pivots, const D* __restrict__ dist, uint32_t n,
             uint32_t k, uint64_t s0, const uint32_t* __restrict__ sweep_ctr, uint32_t sweep) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const uint64_t q = (uint64_t)(*sweep_ctr + sweep) * n + t;
  const uint64_t G = 0x9E3779B97F4A7C15ull;
  const uint32_t i = (uint32_t)(smix(s0 + (2 * q + 1) * G) % n);
  const uint32_t pidx = (uint32_t)(smix(s0 + (2 * q + 2) * G) % k);
  const uint32_t j = pivots[pidx];
  const D du = dist[(size_t)pidx * n + i];
  const float hop = (i == j || du == (D)~(D)0) ? 0.0f : (float)du;
  samples[t] = make_uint4(i, j, __float_as_uint(hop), 0u);
}

// The pair update against positions a (node) and b (pivot): the pivot's move in
// fixed point; the node's is its negative.
__device__ __forceinline__ void pair_move(const float4 a, const float4 b, float d, float eta, long long* f) {
  const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y), dz = __fsub_rn(a.z, b.z);
  const float mag = fmaxf(len3(dx, dy, dz), 1e-6f);
  const float w = __fdiv_rn(1.0f, __fmul_rn(d, d));
  const float mu = fminf(__fmul_rn(w, eta), 1.0f);
  const float r = __fdiv_rn(__fmul_rn(__fmul_rn(0.5f, mu), __fsub_rn(mag, d)), mag);
  f[0] = __double2ll_rn((double)__fmul_rn(r, dx) * FIX_SCALE);
  f[1] = __double2ll_rn((double)__fmul_rn(r, dy) * FIX_SCALE);
  f[2] = __double2ll_rn((double)__fmul_rn(r, dz) * FIX_SCALE);
}

__device__ __forceinline__ void pair_add(long long* acc, uint32_t v, const long long* f, bool neg) {
  unsigned long long* o = reinterpret_cast<unsigned long long*>(acc + 3 * (size_t)v);
#pragma unroll
  for (int c = 0; c < 3; ++c) atomicAdd(o + c, (unsigned long long)(neg ? -f[c] : f[c]));
}

// Node v moves by the mean of its `c` accumulated moves.
__device__ __forceinline__ float4 pair_moved(float4 p, const long long* a, uint32_t c) {
  const double inv = 1.0 / (FIX_SCALE * (double)c);
  p.x = __fadd_rn(p.x, (float)((double)a[0] * inv));
  p.y = __fadd_rn(p.y, (float)((double)a[1] * inv));
  p.z = __fadd_rn(p.z, (float)((double)a[2] * inv));
  return p;
}

// A sweep is 64 batches of two short kernels, each a few dependent round trips,
// so both are launched as programmatic dependents: a kernel is placed and reads
// its samples while the one before drains, and waits for it (all of its writes)
// before it touches positions or sums; the draw and the step's end are ordinary
// launches. (A cluster of eight CTAs that kept a whole sweep in one
// launch with barriers between the phases was slower, 569 us a sweep at 200,000
// nodes: every phase waits for the adds of 4,096 threads to drain.) B200, us a
// sweep, before (samples drawn in the batch, a pass over all nodes to apply) and
// after: 200,000 nodes 388 -> 238 (296 without the early placement), 30,000 382
// -> 224, 1,000 27 -> 18, 1 M 599 -> 426.

// One batch: every pair against the batch-start positions, both moves added in
// fixed point.
__global__ void __launch_bounds__(128)
k_pairs(const uint4* __restrict__ samples, uint32_t count, const float4* pos, long long* acc, uint32_t* cnt,
        const float* __restrict__ eta_table, uint32_t n_eta, const uint32_t* __restrict__ sweep_ctr, uint32_t sweep) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const uint32_t sw = *sweep_ctr + sweep;
  const float eta = eta_table[sw < n_eta ? sw : n_eta - 1];
  const uint4 p = samples[t];
  dev::dependent_launch_wait();
  const float hop = __uint_as_float(p.z);
  if (!(hop > 0.0f)) return;
  long long f[3];
  pair_move(pos[p.x], pos[p.y], hop, eta, f);
  pair_add(acc, p.x, f, true);
  pair_add(acc, p.y, f, false);
  atomicAdd(&cnt[p.x], 1u);
  atomicAdd(&cnt[p.y], 1u);
}

// The batch's end: each node it touched moves by the mean of its moves and is
// cleared. A thread per sample endpoint; the one that takes the node's count
// owns it (the others find 0), so no pass over all n nodes looks for the few
// that moved. Sums and position are read beside the count: only the owner
// writes them, after its own reads.
__global__ void __launch_bounds__(128)
k_pairs_apply(const uint4* __restrict__ samples, uint32_t count, float4* pos, long long* acc, uint32_t* cnt) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 2 * count) return;
  const uint4 s = samples[t >> 1];
  dev::dependent_launch_wait();
  if (!(__uint_as_float(s.z) > 0.0f)) return;
  const uint32_t v = (t & 1u) ? s.y : s.x;
  long long* m = acc + 3 * (size_t)v;
  const long long f[3] = {__ldcg(m), __ldcg(m + 1), __ldcg(m + 2)};
  const float4 p = __ldcg(pos + v);
  const uint32_t c = atomicExch(cnt + v, 0u);
  if (c == 0) return;
  pos[v] = pair_moved(p, f, c);
  m[0] = 0;
  m[1] = 0;
  m[2] = 0;
}

// The end of a step's sweeps: the last sweep's output to the engine's positions
// and the read-back array, and the sweep counter (one launch).
__global__ void __launch_bounds__(256)
k_step_end(const float4* v, uint32_t n, float4* pos, float* __restrict__ xyz, uint32_t* ctr, uint32_t sweeps) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *ctr += sweeps;
  if (i >= n) return;
  const float4 p = v[i];
  if (v != pos) pos[i] = p;
  xyz[3 * (size_t)i] = p.x;
  xyz[3 * (size_t)i + 1] = p.y;
  xyz[3 * (size_t)i + 2] = p.z;
}

__global__ void k_pack(const float4* __restrict__ v, uint32_t n, float* __restrict__ xyz) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 p = v[i];
  xyz[3 * (size_t)i] = p.x;
  xyz[3 * (size_t)i + 1] = p.y;
  xyz[3 * (size_t)i + 2] = p.z;
}

// ------------------------------------------------- multi-source BFS --
// Hop distances from all k pivots at once: every node keeps one bit per pivot
// (the pivots that have reached it) and one per pivot that reached it in the
// previous level (the frontier). A level is one pull pass: node i ORs its
// neighbours' frontier words, keeps the bits it has not seen, and records the
// level as its distance to those pivots. Exact BFS distances, independent of
// thread order. A node holds `stride` words of 64 pivots, WB of them (one or
// two 16-byte loads per neighbour) per pass over its row.
//
// A level is a few dependent round trips per node (row bounds, ids, frontier
// words), so four neighbours' words are in flight, a node that every pivot has
// reached gathers nothing, and a gather ends once it holds every bit still wanted.
// Distances go straight into their
// 16-bit rows (u32 from level 65,535 on). Levels are launched MS_CHUNK at a
// time without waiting; one after the last growing level returns at once.
// B200, random geometric graphs, us a level: 30,011 nodes with 100 pivots 16 -> 7,
// 200,000 with 200 pivots 37 -> 22. A whole bind (host copies in it): 5.0 -> 1.7
// ms and 27 -> 12; R-MAT scale 18 (hub rows, 6 levels) 310 -> 24.
constexpr int MS_CHUNK = 32;
using word_t = unsigned long long;

template <typename D>
__global__ void k_msbfs_seed(uint32_t n, uint32_t k, uint32_t stride, const uint32_t* __restrict__ piv,
                             word_t* __restrict__ visited, word_t* __restrict__ front, D* __restrict__ dist) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= k) return;
  const uint32_t v = piv[p];
  const word_t bit = 1ull << (p & 63u);
  atomicOr(&visited[(size_t)v * stride + (p >> 6)], bit);
  atomicOr(&front[(size_t)v * stride + (p >> 6)], bit);
  dist[(size_t)p * n + v] = 0;
}

template <int WB>
struct Words {
  word_t w[WB];
};
template <int WB>
__device__ __forceinline__ Words<WB> load_words(const word_t* p) {
  Words<WB> r;
  if constexpr (WB == 1) {
    r.w[0] = *p;
  } else {
#pragma unroll
    for (int q = 0; q < WB / 2; ++q) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p + 2 * q);
      r.w[2 * q] = v.x;
      r.w[2 * q + 1] = v.y;
    }
  }
  return r;
}
template <int WB>
__device__ __forceinline__ void store_words(word_t* p, const Words<WB>& r) {
  if constexpr (WB == 1) {
    *p = r.w[0];
  } else {
#pragma unroll
    for (int q = 0; q < WB / 2; ++q)
      *reinterpret_cast<ulonglong2*>(p + 2 * q) = make_ulonglong2(r.w[2 * q], r.w[2 * q + 1]);
  }
}

// *last: the highest level at which some node grew (0: the seeds).
template <typename D, int WB>
__global__ void __launch_bounds__(NODE_THREADS)
k_msbfs_level(uint32_t n, uint32_t k, uint32_t stride, const uint32_t* __restrict__ off,
              const uint32_t* __restrict__ nbr, const word_t* __restrict__ front, word_t* __restrict__ next,
              word_t* __restrict__ visited, D* __restrict__ dist, uint32_t level, uint32_t* last) {
  if (*(volatile uint32_t*)last + 1u < level) return;  // the level before added nothing
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  bool grew = false;
  if (i < n) {
    const uint32_t e0 = off[i], e1 = off[i + 1];
    for (uint32_t w0 = 0; w0 < stride; w0 += WB) {
      word_t* vis = visited + (size_t)i * stride + w0;
      const Words<WB> seen = load_words<WB>(vis);
      Words<WB> want, acc;
      word_t missing = 0;
#pragma unroll
      for (int q = 0; q < WB; ++q) {
        const uint32_t p0 = (w0 + q) * 64u;  // pivots [p0, p0 + 64) of this word
        const word_t all = p0 + 64u <= k ? ~0ull : (p0 < k ? (1ull << (k - p0)) - 1ull : 0ull);
        want.w[q] = all & ~seen.w[q];
        acc.w[q] = 0ull;
        missing |= want.w[q];
      }
      uint32_t e = e0;
      for (; missing && e + 4 <= e1; e += 4) {
        uint32_t id[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) id[u] = __ldg(nbr + e + u);
        Words<WB> f[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) f[u] = load_words<WB>(front + (size_t)id[u] * stride + w0);
        missing = 0;
#pragma unroll
        for (int q = 0; q < WB; ++q) {
          acc.w[q] |= f[0].w[q] | f[1].w[q] | f[2].w[q] | f[3].w[q];
          missing |= want.w[q] & ~acc.w[q];
        }
      }
      if (missing && e < e1) {  // one to three left, together
        uint32_t id[3];
#pragma unroll
        for (int u = 0; u < 3; ++u) id[u] = __ldg(nbr + min(e + u, e1 - 1u));
        Words<WB> f[3];
#pragma unroll
        for (int u = 0; u < 3; ++u) f[u] = load_words<WB>(front + (size_t)id[u] * stride + w0);
#pragma unroll
        for (int q = 0; q < WB; ++q) acc.w[q] |= f[0].w[q] | f[1].w[q] | f[2].w[q];
      }
      Words<WB> now;
      word_t any = 0;
#pragma unroll
      for (int q = 0; q < WB; ++q) {
        now.w[q] = acc.w[q] & want.w[q];
        any |= now.w[q];
      }
      store_words<WB>(next + (size_t)i * stride + w0, now);
      if (!any) continue;
      grew = true;
#pragma unroll
      for (int q = 0; q < WB; ++q) {
        acc.w[q] = seen.w[q] | now.w[q];
        for (word_t nb = now.w[q]; nb; nb &= nb - 1ull)
          dist[(size_t)((w0 + q) * 64u + (uint32_t)__ffsll((long long)nb) - 1u) * n + i] = (D)level;
      }
      store_words<WB>(vis, acc);
    }
  }
  if (__syncthreads_or(grew) && threadIdx.x == 0) atomicMax(last, level);
}

__global__ void k_dist_widen(const uint16_t* __restrict__ d16, size_t count, uint32_t* __restrict__ d32) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  d32[t] = d16[t] == 0xFFFFu ? UNREACH : (uint32_t)d16[t];
}

// ============================================================== host ==
// sgd_stress.rs:372-394
static void bfs(uint32_t n, const uint32_t* off, const uint32_t* nbr, uint32_t src, uint32_t* dist,
                std::vector<uint32_t>& q) {
  std::fill(dist, dist + n, UNREACH);
  q.clear();
  dist[src] = 0;
  q.push_back(src);
  for (size_t h = 0; h < q.size(); ++h) {
    uint32_t v = q[h], dv = dist[v];
    for (uint32_t e = off[v]; e < off[v + 1]; ++e) {
      uint32_t u = nbr[e];
      if (dist[u] == UNREACH) {
        dist[u] = dv + 1;
        q.push_back(u);
      }
    }
  }
}

// sgd_stress.rs:324-334
static float anneal_eta(uint64_t sweep, float eta_max, float eta_min, uint32_t n_anneal) {
  if (n_anneal == 0) return eta_min;
  float t = (float)sweep / (float)n_anneal;
  if (t >= 1.0f) return eta_min;
  float ratio = std::fmax(eta_min / eta_max, 1e-9f);
  return eta_max * std::pow(ratio, t);
}

template <typename T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0;
  void alloc(size_t c) {
    if (p && c <= n) return;
    free();
    c = std::max<size_t>(c, 1);
    JC_CUDA_CHECK(cudaMalloc(&p, c * sizeof(T)));
    n = c;
  }
  void free() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
  ~DBuf() { free(); }
};

inline uint32_t cdiv(uint64_t a, uint64_t b) { return (uint32_t)((a + b - 1) / b); }

class SgdEngine : public Engine {
 public:
  explicit SgdEngine(bool jacobi) : jacobi_(jacobi) {
    desc_.id = jacobi ? "sgd-stress-gpu" : "sgd-stress";
    desc_.kind = 1;
    desc_.display_name = jacobi ? "SGD stress (B200, Jacobi pivot)" : "SGD stress (B200, per-pair scatter)";
    desc_.description =
        jacobi ? "Pivot stress by SGD (s_gd2 step, Ortmann sparse pivots): one thread per node slides itself "
                 "along its k pivot terms against start-of-sweep positions (Jacobi), pivot positions "
                 "staged in shared memory, distances pivot-major."
               : "Pivot stress by SGD with the s_gd2 pair update moving both endpoints: the reference "
                 "engine's own random (node, pivot) samples, evaluated in parallel batches with "
                 "deterministic fixed-point accumulation.";
    desc_.needs_edges = 1;
    desc_.needs_cpu_positions = 1;
    desc_.needs_gpu_positions_buffer = 0;
  }
  ~SgdEngine() override { release(); }

  const jc_descriptor& descriptor() const override { return desc_; }

  void set_params(const char* json) override {
    decode_sgd(json, &s_, desc_.id);
    drop_graph();
  }

  void init(uint32_t n, const uint32_t* off, const uint32_t* nbr, uint64_t nnz, const float* xyz) override {
    validate_csr(n, off, nbr, nnz, xyz);
    ensure_stream();
    initialized_ = false;
    drop_graph();
    n_ = n;
    // select_pivots (sgd_stress.rs:143-175) with the engine's SplitMix64.
    SplitMix64 rng(s_.seed);
    k_ = n == 0 ? 0 : std::min(std::max(s_.n_pivots, 1u), n);
    pivots_.clear();
    host_dist_valid_ = true;
    if (s_.random_pivots && n && k_) {
      init_random_pivots(n, off, nbr, nnz, xyz, rng);
      return;
    }
    std::vector<uint32_t> dist32((size_t)k_ * n);
    if (n && k_) {
      std::vector<uint32_t> min_d(n, UNREACH), q;
      q.reserve(n);
      uint32_t next = (uint32_t)rng.below(n);
      for (uint32_t t = 0; t < k_; ++t) {
        uint32_t* d = &dist32[(size_t)t * n];
        bfs(n, off, nbr, next, d, q);
        uint32_t best = next, best_d = 0;
        for (uint32_t v = 0; v < n; ++v) {
          uint32_t dv = d[v];
          if (dv != UNREACH && dv < min_d[v]) min_d[v] = dv;
          uint32_t cover = min_d[v];
          if (cover != UNREACH && cover > best_d) { best_d = cover; best = v; }
        }
        pivots_.push_back(next);
        next = best;
      }
    }
    stream_state_ = rng.state;  // position of the pair-sampling stream
    host_dist_ = dist32;
    uint32_t maxd = 0;
    for (uint32_t d : dist32)
      if (d != UNREACH) maxd = std::max(maxd, d);
    finish_init(n, xyz, maxd, &dist32);
  }

  // k distinct uniformly random pivots (a partial Fisher-Yates shuffle on the
  // engine's SplitMix64) and their hop distances by the device multi-source BFS.
  void init_random_pivots(uint32_t n, const uint32_t* off, const uint32_t* nbr, uint64_t nnz, const float* xyz,
                          SplitMix64& rng) {
    std::vector<uint32_t> idx(n);
    for (uint32_t i = 0; i < n; ++i) idx[i] = i;
    for (uint32_t t = 0; t < k_; ++t) std::swap(idx[t], idx[t + (uint32_t)rng.below(n - t)]);
    pivots_.assign(idx.begin(), idx.begin() + k_);
    stream_state_ = rng.state;
    // words per node: 1, 2 or a multiple of 4 (16-byte loads)
    uint32_t W = (k_ + 63u) / 64u;
    if (W > 2) W = (W + 3u) / 4u * 4u;
    const size_t words = (size_t)n * W, cells = (size_t)k_ * n;
    // the graph, and one bit per (node, pivot) seen, in the frontier and in the next
    // one: a block of the pool, given back at the end of the bind (a bind of 30,011 nodes
    // with 100 pivots 1.80 ms; 1.72 with the buffers kept by every engine, 2.40 with
    // cudaMalloc and cudaFree)
    const auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t seen_b = up(sizeof(word_t) * words), off_b = up(sizeof(uint32_t) * ((size_t)n + 1)),
                 nbr_b = up(sizeof(uint32_t) * std::max<uint64_t>(nnz, 1));
    const PoolBlock work(3 * seen_b + off_b + nbr_b + 256);
    word_t *vis = reinterpret_cast<word_t*>(work.p), *fa = reinterpret_cast<word_t*>(work.p + seen_b),
           *fb = reinterpret_cast<word_t*>(work.p + 2 * seen_b);
    uint32_t* goff = reinterpret_cast<uint32_t*>(work.p + 3 * seen_b);
    uint32_t* gnbr = reinterpret_cast<uint32_t*>(work.p + 3 * seen_b + off_b);
    uint32_t* last = reinterpret_cast<uint32_t*>(work.p + 3 * seen_b + off_b + nbr_b);
    piv_.alloc(k_);
    dist16_.alloc(cells);
    JC_CUDA_CHECK(cudaMemcpyAsync(goff, off, sizeof(uint32_t) * ((size_t)n + 1), cudaMemcpyHostToDevice, stream_));
    if (nnz) JC_CUDA_CHECK(cudaMemcpyAsync(gnbr, nbr, sizeof(uint32_t) * nnz, cudaMemcpyHostToDevice, stream_));
    JC_CUDA_CHECK(cudaMemcpyAsync(piv_.p, pivots_.data(), sizeof(uint32_t) * k_, cudaMemcpyHostToDevice, stream_));
    JC_CUDA_CHECK(cudaMemsetAsync(vis, 0, sizeof(word_t) * words, stream_));
    JC_CUDA_CHECK(cudaMemsetAsync(fa, 0, sizeof(word_t) * words, stream_));
    JC_CUDA_CHECK(cudaMemsetAsync(dist16_.p, 0xFF, sizeof(uint16_t) * cells, stream_));
    JC_CUDA_CHECK(cudaMemsetAsync(last, 0, 4, stream_));
    k_msbfs_seed<uint16_t><<<cdiv(k_, 256), 256, 0, stream_>>>(n, k_, W, piv_.p, vis, fa, dist16_.p);
    auto launch = [&](auto* dist, uint32_t level) {
      using D = std::remove_pointer_t<decltype(dist)>;
      const uint32_t blocks = cdiv(n, NODE_THREADS);
      if (W == 1)
        k_msbfs_level<D, 1><<<blocks, NODE_THREADS, 0, stream_>>>(n, k_, W, goff, gnbr, fa, fb, vis, dist, level, last);
      else if (W == 2)
        k_msbfs_level<D, 2><<<blocks, NODE_THREADS, 0, stream_>>>(n, k_, W, goff, gnbr, fa, fb, vis, dist, level, last);
      else
        k_msbfs_level<D, 4><<<blocks, NODE_THREADS, 0, stream_>>>(n, k_, W, goff, gnbr, fa, fb, vis, dist, level, last);
      std::swap(fa, fb);
    };
    bool wide = false;
    uint32_t level = 1, maxd = 0;
    for (;;) {
      for (int c = 0; c < MS_CHUNK; ++c, ++level) {
        if (level == 0xFFFFu) {  // the first distance that 16 bits cannot hold
          wide = true;
          dist32_.alloc(cells);
          k_dist_widen<<<(unsigned)((cells + 255) / 256), 256, 0, stream_>>>(dist16_.p, cells, dist32_.p);
        }
        if (wide) launch(dist32_.p, level);
        else launch(dist16_.p, level);
      }
      JC_CUDA_CHECK(cudaGetLastError());
      JC_CUDA_CHECK(cudaMemcpyAsync(&maxd, last, 4, cudaMemcpyDeviceToHost, stream_));
      JC_CUDA_CHECK(cudaStreamSynchronize(stream_));
      if (maxd + 1 < level) break;  // the last level launched added nothing
    }
    host_dist_.clear();
    host_dist_valid_ = false;  // copied back on demand (stress and pivot read-outs)
    finish_init(n, xyz, maxd, nullptr);
  }

  // The rest of init, from the pivot distances: host rows (dist32 != null)
  // or rows already on the device (dist16_, or dist32_ when some distance does
  // not fit 16 bits).
  void finish_init(uint32_t n, const float* xyz, uint32_t maxd, const std::vector<uint32_t>* dist32) {
    wide_ = maxd >= 0xFFFFu;
    // eta schedule, one entry per sweep up to the end of annealing
    float eta_max = s_.eta_max, eta_min = s_.eta_min;
    if (s_.auto_eta && maxd > 0) {
      eta_max = (float)maxd * (float)maxd;
      eta_min = 0.01f;
    }
    n_eta_ = s_.n_anneal_steps + 1;
    std::vector<float> eta(n_eta_);
    for (uint32_t w = 0; w < n_eta_; ++w) eta[w] = anneal_eta(w, eta_max, eta_min, s_.n_anneal_steps);
    max_dist_ = maxd;
    // device buffers
    pos_a_.alloc(n); pos_b_.alloc(n); xyz_.alloc((size_t)3 * n); piv_.alloc(k_); eta_.alloc(n_eta_);
    ctr_.alloc(1);
    if (!dist32) {
      // (on the device already: multi-source BFS)
    } else if (wide_) {
      dist32_.alloc((size_t)k_ * n);
      if (k_ && n)
        JC_CUDA_CHECK(cudaMemcpyAsync(dist32_.p, dist32->data(), sizeof(uint32_t) * k_ * n, cudaMemcpyHostToDevice,
                                      stream_));
    } else {
      std::vector<uint16_t> d16(dist32->size());
      for (size_t t = 0; t < d16.size(); ++t) d16[t] = (*dist32)[t] == UNREACH ? 0xFFFFu : (uint16_t)(*dist32)[t];
      dist16_.alloc((size_t)k_ * n);
      if (k_ && n)
        JC_CUDA_CHECK(cudaMemcpyAsync(dist16_.p, d16.data(), sizeof(uint16_t) * k_ * n, cudaMemcpyHostToDevice, stream_));
    }
    if (!jacobi_) {
      acc_.alloc((size_t)3 * std::max<uint32_t>(n, 1));
      cnt_.alloc(std::max<uint32_t>(n, 1));
      samples_.alloc(n);
      JC_CUDA_CHECK(cudaMemsetAsync(acc_.p, 0, sizeof(long long) * 3 * std::max<uint32_t>(n, 1), stream_));
      JC_CUDA_CHECK(cudaMemsetAsync(cnt_.p, 0, sizeof(uint32_t) * std::max<uint32_t>(n, 1), stream_));
    }
    std::vector<float> pos4((size_t)4 * n, 0.0f);
    for (uint32_t i = 0; i < n; ++i)
      for (int c = 0; c < 3; ++c) pos4[4 * (size_t)i + c] = xyz[3 * (size_t)i + c];
    if (n) {
      JC_CUDA_CHECK(cudaMemcpyAsync(pos_a_.p, pos4.data(), sizeof(float4) * n, cudaMemcpyHostToDevice, stream_));
      JC_CUDA_CHECK(cudaMemcpyAsync(xyz_.p, xyz, sizeof(float) * 3 * n, cudaMemcpyHostToDevice, stream_));
    }
    if (k_) JC_CUDA_CHECK(cudaMemcpyAsync(piv_.p, pivots_.data(), sizeof(uint32_t) * k_, cudaMemcpyHostToDevice, stream_));
    JC_CUDA_CHECK(cudaMemcpyAsync(eta_.p, eta.data(), sizeof(float) * n_eta_, cudaMemcpyHostToDevice, stream_));
    JC_CUDA_CHECK(cudaMemsetAsync(ctr_.p, 0, sizeof(uint32_t), stream_));
    JC_CUDA_CHECK(cudaStreamSynchronize(stream_));
    // (the sweeps read one of them)
    if (wide_) dist16_.free();
    else dist32_.free();
    initialized_ = true;
  }

  void step(float* out) override { step_many(1, out); }

  void step_many(uint32_t iters, float* out) override {
    require_init();
    if (n_ == 0 || k_ == 0 || iters == 0) return;
    ensure_graph();
    for (uint32_t s = 0; s < iters; ++s) JC_CUDA_CHECK(cudaGraphLaunch(gexec_, stream_));
    if (out) JC_CUDA_CHECK(cudaMemcpyAsync(out, xyz_.p, sizeof(float) * 3 * n_, cudaMemcpyDeviceToHost, stream_));
    JC_CUDA_CHECK(cudaStreamSynchronize(stream_));
  }

  void positions(float* out) override {
    require_init();
    if (n_ == 0) return;
    JC_CUDA_CHECK(cudaMemcpyAsync(out, xyz_.p, sizeof(float) * 3 * n_, cudaMemcpyDeviceToHost, stream_));
    JC_CUDA_CHECK(cudaStreamSynchronize(stream_));
  }

  void time_steps(uint32_t iters, float* total_ms, float* phase_ms4) override {
    require_init();
    if (phase_ms4)
      for (int k = 0; k < 4; ++k) phase_ms4[k] = 0.0f;
    if (n_ == 0 || k_ == 0 || iters == 0) {
      if (total_ms) *total_ms = 0.0f;
      return;
    }
    ensure_graph();
    cudaEvent_t e0, e1;
    JC_CUDA_CHECK(cudaEventCreate(&e0));
    JC_CUDA_CHECK(cudaEventCreate(&e1));
    JC_CUDA_CHECK(cudaEventRecord(e0, stream_));
    for (uint32_t s = 0; s < iters; ++s) JC_CUDA_CHECK(cudaGraphLaunch(gexec_, stream_));
    JC_CUDA_CHECK(cudaEventRecord(e1, stream_));
    JC_CUDA_CHECK(cudaEventSynchronize(e1));
    float ms = 0.0f;
    JC_CUDA_CHECK(cudaEventElapsedTime(&ms, e0, e1));
    if (total_ms) *total_ms = ms;
    if (phase_ms4) phase_ms4[1] = ms / (float)iters;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
  }

  uint32_t launches_per_step() const override { return launches_; }

  uint32_t node_count() const override { return n_; }
  void enqueue_steps(uint32_t iters) override {
    require_init();
    if (n_ == 0 || k_ == 0) return;
    ensure_graph();
    for (uint32_t s = 0; s < iters; ++s) JC_CUDA_CHECK(cudaGraphLaunch(gexec_, stream_));
  }
  const float* device_xyz() const override { return xyz_.p; }
  cudaStream_t cuda_stream() const override { return stream_; }

  // Stress of the current layout over the engine's (node, pivot) terms:
  // raw Σ w (|x_i - x_j| - d)^2 and the scale-normalized value, w = 1/d^2, in
  // f64 as crates/graph-layouts/src/metrics.rs:31-76 defines them.
  void stress(double* raw, double* normalized) override {
    require_init();
    fetch_host_dist();
    std::vector<float> xyz((size_t)3 * n_);
    positions(xyz.data());
    auto dist_ij = [&](uint32_t i, uint32_t j) {
      double dx = (double)(xyz[3 * (size_t)i] - xyz[3 * (size_t)j]);
      double dy = (double)(xyz[3 * (size_t)i + 1] - xyz[3 * (size_t)j + 1]);
      double dz = (double)(xyz[3 * (size_t)i + 2] - xyz[3 * (size_t)j + 2]);
      return std::sqrt(dx * dx + dy * dy + dz * dz);
    };
    // Fixed-order sums (independent of the thread count): every pivot row is
    // cut into the same CHUNKS ranges, each summed in node order, and the
    // chunk partials are added in chunk order, pivot after pivot.
    constexpr int64_t CHUNKS = 64;
    const int64_t span = ((int64_t)n_ + CHUNKS - 1) / CHUNKS;
    std::vector<double> part(4 * CHUNKS);
    double num = 0, den = 0, wd2 = 0, rs = 0;
    for (uint32_t t = 0; t < k_; ++t) {
      const uint32_t j = pivots_[t];
      const uint32_t* row = &host_dist_[(size_t)t * n_];
#pragma omp parallel for schedule(static)
      for (int64_t c = 0; c < CHUNKS; ++c) {
        double a = 0, b = 0, w2 = 0, r2 = 0;
        const int64_t lo = c * span, hi = std::min<int64_t>((int64_t)n_, lo + span);
        for (int64_t ii = lo; ii < hi; ++ii) {
          const uint32_t i = (uint32_t)ii, du = row[i];
          if (i == j || du == UNREACH || du == 0) continue;
          const double d = (double)du, w = 1.0 / (d * d), big = dist_ij(i, j);
          a += w * d * big;
          b += w * big * big;
          w2 += w * d * d;
          r2 += w * (big - d) * (big - d);
        }
        part[4 * c] = a; part[4 * c + 1] = b; part[4 * c + 2] = w2; part[4 * c + 3] = r2;
      }
      for (int64_t c = 0; c < CHUNKS; ++c) {
        num += part[4 * c]; den += part[4 * c + 1]; wd2 += part[4 * c + 2]; rs += part[4 * c + 3];
      }
    }
    if (raw) *raw = rs;
    if (!normalized) return;
    if (den <= 0.0 || wd2 <= 0.0) {
      *normalized = 0.0;
      return;
    }
    const double alpha = num / den;
    double acc = 0;
    for (uint32_t t = 0; t < k_; ++t) {
      const uint32_t j = pivots_[t];
      const uint32_t* row = &host_dist_[(size_t)t * n_];
#pragma omp parallel for schedule(static)
      for (int64_t c = 0; c < CHUNKS; ++c) {
        double a = 0;
        const int64_t lo = c * span, hi = std::min<int64_t>((int64_t)n_, lo + span);
        for (int64_t ii = lo; ii < hi; ++ii) {
          const uint32_t i = (uint32_t)ii, du = row[i];
          if (i == j || du == UNREACH || du == 0) continue;
          const double d = (double)du, w = 1.0 / (d * d), r = alpha * dist_ij(i, j) - d;
          a += w * r * r;
        }
        part[c] = a;
      }
      for (int64_t c = 0; c < CHUNKS; ++c) acc += part[c];
    }
    *normalized = acc / wd2;
  }

  // Pivot ids (k) and hop distances (k x n, pivot-major, 0xFFFFFFFF =
  // unreachable); either pointer may be null. Returns k.
  uint32_t pivots(uint32_t* piv, uint32_t* dist) override {
    require_init();
    if (piv && k_) std::memcpy(piv, pivots_.data(), sizeof(uint32_t) * k_);
    if (dist && k_ && n_) {
      fetch_host_dist();
      std::memcpy(dist, host_dist_.data(), sizeof(uint32_t) * k_ * n_);
    }
    return k_;
  }

  uint64_t state_size() override { return 8 + (uint64_t)16 * n_; }
  void save_state(void* buf) override {
    require_init();
    uint8_t* b = (uint8_t*)buf;
    uint32_t sw = 0;
    JC_CUDA_CHECK(cudaMemcpyAsync(&sw, ctr_.p, 4, cudaMemcpyDeviceToHost, stream_));
    if (n_) JC_CUDA_CHECK(cudaMemcpyAsync(b + 8, pos_a_.p, sizeof(float4) * n_, cudaMemcpyDeviceToHost, stream_));
    JC_CUDA_CHECK(cudaStreamSynchronize(stream_));
    std::memcpy(b, &n_, 4);
    std::memcpy(b + 4, &sw, 4);
  }
  void load_state(const void* buf, uint64_t len) override {
    require_init();
    if (len != state_size()) fail(JC_ERR_ARG, "state size mismatch");
    const uint8_t* b = (const uint8_t*)buf;
    uint32_t n, sw;
    std::memcpy(&n, b, 4);
    std::memcpy(&sw, b + 4, 4);
    if (n != n_) fail(JC_ERR_ARG, "state is for a graph with a different node count");
    JC_CUDA_CHECK(cudaMemcpyAsync(ctr_.p, &sw, 4, cudaMemcpyHostToDevice, stream_));
    if (n_) {
      JC_CUDA_CHECK(cudaMemcpyAsync(pos_a_.p, b + 8, sizeof(float4) * n_, cudaMemcpyHostToDevice, stream_));
      k_pack<<<cdiv(n_, 256), 256, 0, stream_>>>(pos_a_.p, n_, xyz_.p);
      JC_CUDA_CHECK(cudaGetLastError());
    }
    JC_CUDA_CHECK(cudaStreamSynchronize(stream_));
  }

 private:
  bool jacobi_;
  jc_descriptor desc_{};
  SgdSettings s_;
  uint32_t n_ = 0, k_ = 0, n_eta_ = 1, launches_ = 0, max_dist_ = 0;
  bool wide_ = false, initialized_ = false;
  uint64_t stream_state_ = 0;
  std::vector<uint32_t> pivots_;
  std::vector<uint32_t> host_dist_;  // k x n pivot distances (for the stress read-out)
  bool host_dist_valid_ = true;

  void fetch_host_dist() {
    if (host_dist_valid_) return;
    host_dist_.resize((size_t)k_ * n_);
    if (k_ && n_) {
      if (wide_) {
        JC_CUDA_CHECK(cudaMemcpyAsync(host_dist_.data(), dist32_.p, sizeof(uint32_t) * k_ * n_,
                                      cudaMemcpyDeviceToHost, stream_));
        JC_CUDA_CHECK(cudaStreamSynchronize(stream_));
      } else {
        std::vector<uint16_t> d16((size_t)k_ * n_);
        JC_CUDA_CHECK(cudaMemcpyAsync(d16.data(), dist16_.p, sizeof(uint16_t) * k_ * n_, cudaMemcpyDeviceToHost,
                                      stream_));
        JC_CUDA_CHECK(cudaStreamSynchronize(stream_));
        for (size_t t = 0; t < d16.size(); ++t) host_dist_[t] = d16[t] == 0xFFFFu ? UNREACH : d16[t];
      }
    }
    host_dist_valid_ = true;
  }
  cudaStream_t stream_ = nullptr;
  cudaGraphExec_t gexec_ = nullptr;
  DBuf<float4> pos_a_, pos_b_;
  DBuf<float> xyz_, eta_;
  DBuf<uint32_t> piv_, ctr_, dist32_, cnt_;
  DBuf<uint16_t> dist16_;
  DBuf<long long> acc_;
  DBuf<uint4> samples_;  // one sweep's pairs

  void ensure_stream() {
    if (!stream_) {
      int dev_count = 0;
      if (cudaGetDeviceCount(&dev_count) != cudaSuccess || dev_count == 0)
        fail(JC_ERR_CUDA, "no CUDA device is available");
      JC_CUDA_CHECK(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    }
  }
  void release() {
    drop_graph();
    if (stream_) {
      cudaStreamSynchronize(stream_);
      cudaStreamDestroy(stream_);
      stream_ = nullptr;
    }
  }
  void drop_graph() {
    if (gexec_) {
      cudaGraphExecDestroy(gexec_);
      gexec_ = nullptr;
    }
  }
  void require_init() const {
    if (!initialized_) fail(JC_ERR_STATE, std::string(desc_.id) + " step called before successful init");
  }

  template <typename D>
  int enqueue_sweeps(const D* dist) {
    const uint32_t n = n_, k = k_;
    const uint32_t sweeps = std::max(s_.sweeps_per_step, 1u);
    int L = 0;
    if (jacobi_) {
      // sgd_stress_gpu.rs:377-428: one eta per step, `sweeps` ping-pong sweeps.
      // the mu table covers distances up to the largest one when it fits in 32 KB
      const uint32_t mu_len = max_dist_ + 1 <= JACOBI_MU_MAX ? max_dist_ + 1 : 0u;
      // (rounded to whole 16 bytes; the 200 KB below leave room for the table)
      const size_t smem = sizeof(float4) * k + sizeof(float2) * mu_len;
      if (sizeof(float4) * k + sizeof(float) * mu_len > 200 * 1024)
        fail(JC_ERR_ARG, "too many pivots for the shared-memory pivot stage");
      // (the limit belongs to the kernel, not to one engine: always the most any launch takes)
      if (smem > 48 * 1024)
        JC_CUDA_CHECK(cudaFuncSetAttribute(k_jacobi<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           200 * 1024 + (int)(sizeof(float) * JACOBI_MU_MAX)));
      float4* in = pos_a_.p;
      float4* out = pos_b_.p;
      for (uint32_t s = 0; s < sweeps; ++s) {
        k_jacobi<D><<<cdiv(n, NODE_THREADS), NODE_THREADS, smem, stream_>>>(in, out, piv_.p, dist, n, k, eta_.p, n_eta_,
                                                                            ctr_.p, mu_len);
        std::swap(in, out);
        ++L;
      }
      k_step_end<<<cdiv(n, 256), 256, 0, stream_>>>(in, n, pos_a_.p, xyz_.p, ctr_.p, sweeps);
      ++L;
    } else {
      // sgd_stress.rs:287-315: per sweep, eta(sweep), n samples, sweep += 1.
      // Default: batches of max(256, n/64) samples (at most 64 per sweep).
      uint32_t batches = s_.scatter_batches ? s_.scatter_batches : cdiv(n, std::max(256u, cdiv(n, 64)));
      batches = std::max(1u, std::min(batches, n));
      const uint32_t per = cdiv(n, batches);
      for (uint32_t s = 0; s < sweeps; ++s) {
        k_pairs_draw<D><<<cdiv(n, 256), 256, 0, stream_>>>(samples_.p, piv_.p, dist, n, k, stream_state_, ctr_.p, s);
        ++L;
        for (uint32_t q0 = 0; q0 < n; q0 += per) {
          const uint32_t cnt = std::min(per, n - q0);
          launch_chained(q0 > 0, stream_, cdiv(cnt, 128), 128, 0, k_pairs, (const uint4*)samples_.p + q0, cnt, (const float4*)pos_a_.p,
                     acc_.p, cnt_.p, (const float*)eta_.p, n_eta_, (const uint32_t*)ctr_.p, s);
          launch_chained(true, stream_, cdiv(2 * (uint64_t)cnt, 128), 128, 0, k_pairs_apply, (const uint4*)samples_.p + q0, cnt,
                     pos_a_.p, acc_.p, cnt_.p);
          L += 2;
        }
      }
      k_step_end<<<cdiv(n, 256), 256, 0, stream_>>>(pos_a_.p, n, pos_a_.p, xyz_.p, ctr_.p, sweeps);
      ++L;
    }
    JC_CUDA_CHECK(cudaGetLastError());
    return L;
  }

  void ensure_graph() {
    if (gexec_) return;
    int L = 0;
    cudaGraph_t g = record_graph(
        stream_, [&] { L = wide_ ? enqueue_sweeps<uint32_t>(dist32_.p) : enqueue_sweeps<uint16_t>(dist16_.p); });
    cudaError_t e = cudaGraphInstantiate(&gexec_, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) fail(JC_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
    launches_ = (uint32_t)L;
  }
};

}  // namespace sgd

Engine* make_sgd_engine(bool jacobi) { return new sgd::SgdEngine(jacobi); }

}  // namespace jc
