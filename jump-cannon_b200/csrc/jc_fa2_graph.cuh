// Octrees of a batch of small graphs, one CTA per graph, or of one small graph.
//
// Included by jc_fa2.cu after the device helpers it reuses (TNode, DevState,
// KParams, Forest, body_key, key_after, lcp_levels, the prefix-length index). A
// batch's step needs no order between graphs, only inside each: where the largest
// graph's keys fit a CTA's shared memory, one launch builds every tree (root cell,
// keys, sort, prefix lengths, nodes, centres of mass) instead of the forest's
// device-wide passes, which move every key through memory seven times and give
// each phase a launch of its own. The walk, attraction and speed kernels that
// follow are the forest's. A graph's nodes lie together and in pre-order; which
// graph's come first is left to the order of arrival, as nothing reads across
// trees. Same cells, sums and roundings as the forest path (fa2_bh.rs:768-967).
//
// Bound by latency: a graph's sort passes and the levels of its tree follow one
// another. So a thread takes one cell, not one body's whole path of them, a
// cell's children are found in shared memory and their centres loaded together,
// and four CTAs of 64 registers stay on an SM (more of fewer registers: 233 us a
// step -> 237 with 48, 253 with 40). B200, us a step (theta 0.8, all phases),
// forest and this: 1,000 graphs of 50 to 2,000 bodies 408 -> 233, 100 of them 185 ->
// 122, 500 of 20 to 500 111 -> 90, 300 of 1,000 to 4,000 528 -> 320, 60 of 4,097 to
// 8,000 418 -> 307, 1,000 of 50 to 8,000 1,156 -> 801, 3 of 7,000 to 8,000 184 -> 183:
// there the longest graph's chain has caught up, so this ends at 8,192 bodies.

// (included inside namespace jc::fa2)

// Totals of the trees of one step; the last CTA hands them to DevState and
// zeroes them for the next step.
struct GraphTally {
  uint32_t cursor;  // nodes taken
  uint32_t done;    // CTAs finished
  uint32_t n_invalid;
  uint32_t dropped;
  uint32_t max_depth;
};

constexpr uint32_t GB_MAX_N = 8192;   // bodies of the largest graph
// Runs of keys with equal top words up to this long are ordered by counting, each entry
// against its run; a longer one, or one where GB_TIES others share an entry's next 32
// bits too (each such pair reads a whole key), sends the graph through the sort of whole
// keys. B200, us of this phase in one CTA, a thread a run of up to 32 and now: clusters of
// 100 bodies, 2,000 bodies 44 -> 13, 8,000 229 -> 51 (a batch's step 639 -> 294, and 350
// by the forest's kernels); uniform layouts of 8,000 2.8 -> 2.3. (A bitonic network over
// whole keys in place of the sixteen passes: 85 us for 8,000 bodies, where these take 80.)
constexpr uint32_t GB_RUN = 128, GB_TIES = 16;
// Threads a graph by the largest one: 256, from 2,048 bodies 512, from 4,096 1,024.
// us a step: 1,000 graphs to 2,000 bodies 233 with 256 threads, 269 with 512; 300 to
// 4,000 379 with 256, 319 with 512; 1,000 to 4,096 421 with 512, 520 with 1,024; 60 to
// 8,000 379 with 512, 307 with 1,024.
constexpr uint32_t GB_SMALL = 2048;
constexpr uint32_t GB_MIDDLE = 4096;
// A single graph: one launch on one SM instead of eleven over all of them. B200, us a
// step, those and this with 256, 512 and 1,024 threads: 20 bodies 47, 29, 31, 37; 400
// 66, 41, 40, 45; 1,000 78, 53, 51, 55; 2,000 86, 78, 70, 72; 3,000 97, 125, 89, 91;
// 4,000 103, 154, 109, 108.
constexpr uint32_t GB_SINGLE_N = 3072, GB_SINGLE_256 = 256, GB_SINGLE_512 = GB_SINGLE_N;
// The largest graph that T threads take.
constexpr uint32_t gb_max_n(int T) { return T == 256 ? GB_SMALL : T == 512 ? GB_MIDDLE : GB_MAX_N; }
static_assert(GB_SINGLE_256 <= GB_SMALL && GB_SINGLE_N <= GB_MIDDLE, "a single graph's sizes too");
constexpr int GB_DEPTHS = 33;        // cell depths 0..32

template <int T>
struct GraphShared {
  uint32_t scan[32];
  uint32_t dstart[GB_DEPTHS + 1];
  uint32_t dcnt[GB_DEPTHS];
  float box[T / 32][6];
  float4 root;
  float size2[GB_DEPTHS];  // (cell side)^2 by depth
  unsigned long long zf;
  uint32_t n_invalid;
  uint32_t n_run;
  uint32_t long_run;  // a run past GB_RUN (set before the counting)
  uint32_t tied;      // an entry with GB_TIES ties (set by it)
  uint32_t dropped;
  uint32_t leaf_depth;
  uint32_t base;
};

// Shared words per launch: two key arrays, two 16-bit permutations, digit counts.
inline uint32_t gb_items(uint32_t biggest) { return std::max(512u, (biggest + 1u + 255u) / 256u * 256u); }
inline size_t gb_smem(uint32_t items, int threads) { return 12 * (size_t)items + 4 * 256 * (size_t)(threads / 32); }

template <int T>
__device__ __forceinline__ uint32_t gb_scan(uint32_t x, uint32_t* total, uint32_t* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t v = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
    if (lane >= o) v += y;
  }
  if (lane == 31) sh[w] = v;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int k = 0; k < T / 32; ++k) {
    const uint32_t t = sh[k];
    before += k < w ? t : 0u;
    all += t;
  }
  __syncthreads();
  *total = all;
  return before + v - x;
}

// One stable pass over the byte at `shift`: every warp counts the digits of its
// own run of entries, the counts become first positions, and the warp places its
// entries 32 at a time in order.
template <int T>
__device__ __forceinline__ void gb_pass(const uint32_t* kin, const uint16_t* vin, uint32_t* kout, uint16_t* vout,
                                        uint32_t n, int shift, uint32_t* wcnt, uint32_t* scan, uint32_t* err) {
  constexpr uint32_t W = T / 32;
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (uint32_t k = threadIdx.x; k < 256u * W; k += T) wcnt[k] = 0;
  __syncthreads();
  const uint32_t chunk = (n + 32u * W - 1u) / (32u * W) * 32u;
  const uint32_t b0 = min(n, w * chunk), b1 = min(n, b0 + chunk);
  uint32_t* wc = wcnt + 256u * w;
  for (uint32_t i = b0 + lane; i < b1; i += 32) atomicAdd(&wc[(kin[i] >> shift) & 0xFFu], 1u);
  __syncthreads();
  uint32_t c = 0, total;
  if (threadIdx.x < 256)
    for (uint32_t k = 0; k < W; ++k) c += wcnt[256u * k + threadIdx.x];
  uint32_t run = gb_scan<T>(c, &total, scan);
  if (threadIdx.x < 256)
    for (uint32_t k = 0; k < W; ++k) {
      const uint32_t x = wcnt[256u * k + threadIdx.x];
      wcnt[256u * k + threadIdx.x] = run;
      run += x;
    }
  __syncthreads();
  const uint32_t below = (1u << lane) - 1u;
  for (uint32_t i0 = b0; i0 < b1; i0 += 32) {
    const uint32_t i = i0 + lane;
    const bool ok = i < b1;
    const uint32_t k = ok ? kin[i] : 0u;
    const uint32_t d = ok ? (k >> shift) & 0xFFu : 256u;
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
    const uint32_t at = ok ? wc[d] : 0u;
    __syncwarp();
    if (ok && (peers & below) == 0u) wc[d] = at + (uint32_t)__popc(peers);
    __syncwarp();
    const uint32_t dst = at + (uint32_t)__popc(peers & below);
    if (ok && JC_IN_BOUNDS(dst, n, err)) {
      kout[dst] = k;
      vout[dst] = vin[i];
    }
  }
  __syncthreads();
}

template <int T>
__global__ void __launch_bounds__(T, 1024 / T)
k_graph_build(const float4* __restrict__ pos, const float* __restrict__ degf, Forest F,
              const uint32_t* __restrict__ order, ulonglong2* key, uint32_t* __restrict__ val,
              uint32_t* __restrict__ first_total, TNode* nodes, uint32_t* cells, KParams P, DevState* st,
              GraphTally* tally, uint32_t items, uint32_t* kids) {
  extern __shared__ __align__(1024) unsigned char gb_raw[];
  __shared__ GraphShared<T> S;
  uint32_t* k0 = reinterpret_cast<uint32_t*>(gb_raw);
  uint32_t* k1 = k0 + items;
  uint32_t* wcnt = k1 + items;
  uint16_t* v0 = reinterpret_cast<uint16_t*>(wcnt + 256 * (T / 32));
  uint16_t* v1 = v0 + items;
  const uint32_t tid = threadIdx.x;
  const int lane = tid & 31, w = tid >> 5;
  const bool single = F.n_graphs == 1;
  const uint32_t g = single ? 0u : order[blockIdx.x];
  const uint32_t B = single ? 0u : F.graph_off[g];
  const uint32_t n = single ? P.n : F.graph_off[g + 1] - B;
  key += B;
  val += B;
  pos += B;
  degf += B;
  // ---- root cell (k_bbox_roots' arithmetic) ----------------------------
  {
    float r[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
    for (uint32_t i = tid; i < n; i += T) {
      const float4 p = pos[i];
      const float v[3] = {p.x, p.y, p.z};
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (isfinite(v[k])) {
          r[k] = fminf(r[k], v[k]);
          r[3 + k] = fmaxf(r[3 + k], v[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        r[k] = fminf(r[k], __shfl_xor_sync(0xFFFFFFFFu, r[k], o));
        r[3 + k] = fmaxf(r[3 + k], __shfl_xor_sync(0xFFFFFFFFu, r[3 + k], o));
      }
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < 6; ++k) S.box[w][k] = r[k];
    if (tid < GB_DEPTHS) S.dcnt[tid] = 0;
    __syncthreads();
    if (tid == 0) {
#pragma unroll
      for (int k = 0; k < 3; ++k)
        for (int ww = 0; ww < T / 32; ++ww) {
          r[k] = fminf(r[k], S.box[ww][k]);
          r[3 + k] = fmaxf(r[3 + k], S.box[ww][3 + k]);
        }
      if (!isfinite(r[0]))
        for (int k = 0; k < 3; ++k) { r[k] = -1.0f; r[3 + k] = 1.0f; }
      float half =
          __fmul_rn(fmaxf(fmaxf(__fsub_rn(r[3], r[0]), __fsub_rn(r[4], r[1])), __fsub_rn(r[5], r[2])), 0.5f);
      if (!isfinite(half) || half <= 0.0f) half = 1.0f;
      const float4 root = make_float4(__fmul_rn(0.5f, __fadd_rn(r[0], r[3])), __fmul_rn(0.5f, __fadd_rn(r[1], r[4])),
                                      __fmul_rn(0.5f, __fadd_rn(r[2], r[5])), __fmul_rn(half, 1.05f));
      float h = root.w;
      for (int d = 0; d < GB_DEPTHS; ++d) {  // halved once per level, as child_center does
        const float side = __fmul_rn(h, 2.0f);
        S.size2[d] = __fmul_rn(side, side);
        h = __fmul_rn(h, 0.5f);
      }
      S.root = root;
      S.zf = flat_z_bits(r[2], r[5], root);
      S.n_invalid = 0;
      S.n_run = 0;
      S.long_run = 0;
      S.tied = 0;
      S.dropped = 0;
      S.leaf_depth = 0;
    }
    __syncthreads();
  }
  // ---- keys: 21 levels in the high word, 11 in the low word -------------
  {
    const float4 root = S.root;
    const uint64_t zf = S.zf;
    uint32_t inval = 0;
    for (uint32_t i = tid; i < n; i += T) {
      const float4 p = pos[i];
      uint64_t hi = 0, lo = 0;
      if (isfinite(p.x) && isfinite(p.y) && isfinite(p.z)) {
        body_key(p, root.x, root.y, root.z, root.w, zf, 21, hi, lo);
      } else {
        hi = 1ull << 63;
        ++inval;
      }
      key[i] = make_ulonglong2(hi, lo);
      k0[i] = (uint32_t)(hi >> 32);
      v0[i] = (uint16_t)i;
    }
    if (inval) atomicAdd(&S.n_invalid, inval);
    __syncthreads();
  }
  const uint32_t N = n - S.n_invalid;
  // ---- sort: the top 32 bits, then the runs of equal tops (k_seg_fix) ----
  for (int p = 0; p < 4; ++p)
    gb_pass<T>(p & 1 ? k1 : k0, p & 1 ? v1 : v0, p & 1 ? k0 : k1, p & 1 ? v0 : v1, n, 8 * p, wcnt, S.scan, &st->error);
  // A thread an entry: its place in its run is the number of the run's entries
  // before it, by the key's next 32 bits in shared memory (whole keys only where
  // those tie). A thread a run, sorting up to 32 entries, kept the CTA waiting for
  // its longest runs (see GB_RUN).
  auto whole = [&](uint32_t a) {
    const uint32_t v = v0[a];
    return JC_IN_BOUNDS(v, n, &st->error) ? key[v] : make_ulonglong2(0ull, 0ull);
  };
  uint16_t* const entry = reinterpret_cast<uint16_t*>(wcnt);  // the entries in runs, in any order
  for (uint32_t a0 = 0; a0 < N; a0 += T) {
    const uint32_t a = a0 + tid, top = a < N ? k0[a] : 0u;
    const bool in = a < N && ((a > 0 && k0[a - 1] == top) || (a + 1 < N && k0[a + 1] == top));
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, in);
    if (m == 0u) continue;  // (the warp's)
    if (a + GB_RUN < N && k0[a + GB_RUN] == top) S.long_run = 1u;
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(&S.n_run, (uint32_t)__popc(m));
    at = __shfl_sync(0xFFFFFFFFu, at, 0) + (uint32_t)__popc(m & ((1u << lane) - 1u));
    if (in) {
      entry[at] = (uint16_t)a;
      k1[a] = (uint32_t)whole(a).x;
    }
  }
  __syncthreads();
  const uint32_t n_run = S.n_run;
  if (n_run && !S.long_run) {
    for (uint32_t q = tid; q < n_run; q += T) {
      const uint32_t a = entry[q], top = k0[a], low = k1[a], body = v0[a];
      const ulonglong2 own = whole(a);
      uint32_t left = 0, right = 0, before = 0, ties = 0;
      while (ties < GB_TIES && left < a && k0[a - left - 1] == top) {
        ++left;
        const uint32_t x = k1[a - left];
        before += x < low ? 1u : 0u;
        if (x == low) {
          ++ties;
          before += key_after(whole(a - left), v0[a - left], own, body) ? 0u : 1u;
        }
      }
      while (ties < GB_TIES && a + right + 1 < N && k0[a + right + 1] == top) {
        ++right;
        const uint32_t x = k1[a + right];
        before += x < low ? 1u : 0u;
        if (x == low) {
          ++ties;
          before += key_after(own, body, whole(a + right), v0[a + right]) ? 1u : 0u;
        }
      }
      if (ties >= GB_TIES) {
        S.tied = 1u;
        break;
      }
      v1[a - left + before] = (uint16_t)body;
    }
    __syncthreads();
    if (!S.tied)
      for (uint32_t q = tid; q < n_run; q += T) v0[entry[q]] = v1[entry[q]];
    __syncthreads();
  }
  if (S.long_run || S.tied) {
    // the whole order, stably by the four words of the key from body order
    for (int word = 0; word < 4; ++word) {
      for (uint32_t i = tid; i < n; i += T) {
        const uint32_t v = word ? v0[i] : i;
        const ulonglong2 k = JC_IN_BOUNDS(v, n, &st->error) ? key[v] : make_ulonglong2(0ull, 0ull);
        const uint64_t x = word < 2 ? k.y : k.x;
        k0[i] = word & 1 ? (uint32_t)(x >> 32) : (uint32_t)x;
        v0[i] = (uint16_t)v;
      }
      __syncthreads();
      for (int p = 0; p < 4; ++p)
        gb_pass<T>(p & 1 ? k1 : k0, p & 1 ? v1 : v0, p & 1 ? k0 : k1, p & 1 ? v0 : v1, n, 8 * p, wcnt, S.scan,
                   &st->error);
    }
  }
  // ---- prefix lengths (k_count) in place of the spare keys ----------------
  const uint32_t nl = lcp_index_bytes(n);
  int8_t* const L = reinterpret_cast<int8_t*>(k1);
  const LcpIndex X{L, L + nl, L + nl + nl / 32, nl / 32, nl / 1024};
  for (uint32_t a = tid; a < nl; a += T) {  // (T divides nl)
    auto load = [&](uint32_t b) {
      const uint32_t v = b < N ? v0[b] : 0u;
      return b < N && JC_IN_BOUNDS(v, n, &st->error) ? key[v] : make_ulonglong2(0ull, 0ull);
    };
    const ulonglong2 ka = load(a);
    ulonglong2 kb;
    kb.x = __shfl_down_sync(0xFFFFFFFFu, ka.x, 1);
    kb.y = __shfl_down_sync(0xFFFFFFFFu, ka.y, 1);
    if (lane == 31) kb = load(a + 1);
    const int next = a + 1 < N ? lcp_levels(ka.x, ka.y, kb.x, kb.y) : -1;
    X.L[a] = (int8_t)next;
    const int mn = __reduce_min_sync(0xFFFFFFFFu, next);
    if (lane == 0) X.m1[a >> 5] = (int8_t)mn;
    if (a < n) val[a] = B + v0[a];
  }
  __syncthreads();
  if (tid < 32) {  // (at most 8 blocks of 1024: one 32-byte row of m2)
    int mn = 127;
    if (tid < X.n2)
      for (int k = 0; k < 32; ++k) mn = min(mn, (int)X.m1[32 * tid + k]);
    X.m2[tid] = (int8_t)mn;
  }
  // ---- node counts -> first node of each body (k0) ------------------------
  uint32_t* const first = k0;
  uint32_t tot;
  {
    const uint32_t per = (n + T - 1) / T;
    const uint32_t a0 = min(n, tid * per), a1 = min(n, a0 + per);
    auto count = [&](uint32_t a) -> uint32_t {
      if (a >= N) return 0u;
      const int prev = a > 0 ? (int)X.L[a - 1] : -1;
      return prev == 32 ? 0u : 1u + (uint32_t)max(0, max(0, (int)X.L[a]) - prev);
    };
    uint32_t sum = 0, drop = 0;
    for (uint32_t a = a0; a < a1; ++a) {
      const uint32_t c = count(a);
      sum += c;
      drop += a < N && c == 0u ? 1u : 0u;
    }
    if (drop) atomicAdd(&S.dropped, drop);
    uint32_t run = gb_scan<T>(sum, &tot, S.scan);
    for (uint32_t a = a0; a < a1; ++a) {
      first[a] = run;
      run += count(a);
    }
    if (tid == 0) {
      first[n] = tot;
      S.base = atomicAdd(&tally->cursor, tot);
      if (!single) F.tree_root[g] = tot ? S.base : END;
    }
  }
  __syncthreads();
  const uint32_t base = S.base;
  bool bad = false;
  if (tot && (uint64_t)base + tot <= P.tree_cap) {
    // ---- cells by depth ------------------------------------------------------
    // Body a opens the cells of depths prev + 1 .. top. Their owners are listed by
    // depth (in shared memory where they fit), so that the searches below take a
    // thread a cell; by body, a warp waits for its longest path.
    auto opened = [&](uint32_t a, int& prev) {
      prev = a > 0 ? (int)X.L[a - 1] : -1;
      return prev == 32 ? 0 : max(0, max(0, (int)X.L[a]) - prev);
    };
    for (uint32_t a = tid; a < N; a += T) {
      int prev;
      const int k = opened(a, prev);
      for (int j = 0; j < k; ++j) atomicAdd(&S.dcnt[min(prev + 1 + j, GB_DEPTHS - 1)], 1u);
    }
    __syncthreads();
    if (w == 0) {
      const uint32_t c = S.dcnt[lane];
      uint32_t v = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += y;
      }
      const uint32_t last = S.dcnt[GB_DEPTHS - 1];
      __syncwarp();
      S.dstart[lane] = v - c;
      S.dcnt[lane] = v - c;  // scatter cursors
      if (lane == 31) {
        S.dstart[GB_DEPTHS - 1] = v;
        S.dcnt[GB_DEPTHS - 1] = v;
        S.dstart[GB_DEPTHS] = v + last;
      }
    }
    __syncthreads();
    const uint32_t n_cells = S.dstart[GB_DEPTHS];
    const bool listed = n_cells <= items;
    for (uint32_t a = tid; a < N; a += T) {
      int prev;
      const int k = opened(a, prev);
      for (int j = 0; j < k; ++j) {
        const uint32_t q = atomicAdd(&S.dcnt[min(prev + 1 + j, GB_DEPTHS - 1)], 1u);
        if (!JC_IN_BOUNDS(q, n_cells, &st->error)) continue;
        if (listed) v1[q] = (uint16_t)a;
        else cells[base + q] = a;
      }
    }
    __syncthreads();
    // a listed cell's node, inside the graph
    auto cell = [&](uint32_t q, int d, uint32_t& a) {
      a = listed ? (uint32_t)v1[q] : cells[base + q];
      const int prev = a > 0 ? (int)X.L[a - 1] : -1;
      return first[a] + (uint32_t)(d - prev - 1);
    };
    // ---- pre-order nodes (k_fill) -------------------------------------------
    const bool linked = tot <= 512u * (T / 32);
    uint16_t* const link = reinterpret_cast<uint16_t*>(wcnt);  // each node's rope, in the graph, in place of the counts
    for (uint32_t q = tid; q < n_cells; q += T) {
      int d = 0;  // the last depth that starts at or before q
#pragma unroll
      for (int o = 32; o > 0; o >>= 1)
        if (d + o < GB_DEPTHS && S.dstart[d + o] <= q) d += o;
      uint32_t a;
      const uint32_t v = cell(q, d, a);
      const uint32_t e = d == 0 ? N - 1u : lcp_next_below(X, a, d);
      if (e >= N || v >= tot) {
        bad = true;
        break;
      }
      const uint32_t sk = first[e + 1];
      nodes[base + v].meta = make_int4(sk >= tot ? (int)END : (int)(base + sk), -1, __float_as_int(S.size2[d]), d);
      if (linked) link[v] = (uint16_t)sk;
    }
    uint32_t leaf_depth = 0;
    for (uint32_t a = tid; a < N; a += T) {
      const uint32_t f1 = first[a + 1];
      if (f1 <= first[a]) continue;  // a dropped duplicate
      const uint32_t body = v0[a], leaf = f1 - 1u;
      if (leaf >= tot || !JC_IN_BOUNDS(body, n, &st->error)) {
        bad = true;
        break;
      }
      const int prev = a > 0 ? (int)X.L[a - 1] : -1;
      const uint32_t ld = (uint32_t)(max(prev, max(0, (int)X.L[a])) + 1);
      leaf_depth = max(leaf_depth, ld);
      const float4 p = pos[body];
      nodes[base + leaf].meta = make_int4(f1 >= tot ? (int)END : (int)(base + f1), (int)(B + body), 0, (int)ld);
      nodes[base + leaf].cm = make_float4(p.x, p.y, p.z, fmaxf(degf[body], 1e-3f));
      if (linked) link[leaf] = (uint16_t)f1;
    }
    leaf_depth = __reduce_max_sync(0xFFFFFFFFu, leaf_depth);
    if (lane == 0 && leaf_depth) atomicMax(&S.leaf_depth, leaf_depth);
    bad = __syncthreads_or(bad);
    // ---- centres of mass, deepest cells first --------------------------------
    // The CTA owns the whole tree, so a barrier between levels takes the place
    // of k_com's climbs and arrival counters. A cell's children come from the
    // ropes in shared memory, so that their centres are loaded together; a tree
    // that outgrows them follows the ropes of its nodes.
    if (!bad) {
      for (int d = GB_DEPTHS - 1; d >= 0; --d) {
        const uint32_t b0 = S.dstart[d], b1 = S.dstart[d + 1];
        if (b0 == b1) continue;  // (uniform)
        for (uint32_t q = b0 + tid; q < b1; q += T) {
          uint32_t a;
          const uint32_t v = cell(q, d, a);
          if (!JC_IN_BOUNDS(v, tot, &st->error)) continue;
          const TNode* const t = nodes + base;
          float mass = 0.0f, sx = 0.0f, sy = 0.0f, sz = 0.0f;
          auto add = [&](const float4 c) {
            mass = __fadd_rn(mass, c.w);
            sx = __fadd_rn(sx, __fmul_rn(c.x, c.w));
            sy = __fadd_rn(sy, __fmul_rn(c.y, c.w));
            sz = __fadd_rn(sz, __fmul_rn(c.z, c.w));
          };
          if (__builtin_expect(linked, 1)) {
            const uint32_t end = link[v];
            uint32_t c = v + 1;
            for (int half = 0; half < 2 && (kids || c < end); ++half) {
              float4 kid[4];
              uint32_t id[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                id[i] = END;
                if (c < end) {
                  id[i] = c;
                  kid[i] = t[c].cm;
                  c = link[c];
                }
              }
              if (kids) reinterpret_cast<uint4*>(kids)[2 * (size_t)v + half] = make_uint4(id[0], id[1], id[2], id[3]);
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (id[i] != END) add(kid[i]);
            }
            if (c != end) bad = true;
          } else {
            // (one load a child, and four of its list a store: with single stores a
            // tree of 3,000 bodies in close pairs took 140 us of these, now 79)
            const uint32_t end = (uint32_t)t[v].meta.x;
            uint32_t c = base + v + 1;
#pragma unroll 1
            for (int half = 0; half < 2 && (kids || c != end); ++half) {
              uint32_t id[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                id[i] = END;
                if (c == end || bad) continue;
                if (c - base >= tot) {
                  bad = true;
                  continue;
                }
                float4 cm;
                int4 meta;
                load_node_c(nodes + c, cm, meta);
                id[i] = c - base;
                add(cm);
                bad = (uint32_t)meta.x <= c;
                c = (uint32_t)meta.x;
              }
              if (kids) reinterpret_cast<uint4*>(kids)[2 * (size_t)v + half] = make_uint4(id[0], id[1], id[2], id[3]);
            }
            if (c != end) bad = true;
          }
          if (mass > 0.0f) {
            sx = __fdiv_rn(sx, mass);
            sy = __fdiv_rn(sy, mass);
            sz = __fdiv_rn(sz, mass);
          }
          nodes[base + v].cm = make_float4(sx, sy, sz, mass);
        }
        __syncthreads();
      }
    }
    if (bad) set_error(st, JC_ERR_DEVICE_TIMEOUT);
  }
  // ---- totals: the last CTA hands them over ---------------------------------
  if (tid == 0) {
    if (S.n_invalid) atomicAdd(&tally->n_invalid, S.n_invalid);
    if (S.dropped) atomicAdd(&tally->dropped, S.dropped);
    if (S.leaf_depth) atomicMax(&tally->max_depth, S.leaf_depth);
    __threadfence();
    if (atomicAdd(&tally->done, 1u) == gridDim.x - 1u) {
      __threadfence();
      const uint32_t total = __ldcg(&tally->cursor), inv = __ldcg(&tally->n_invalid), drop = __ldcg(&tally->dropped);
      st->n_invalid = inv;
      st->n_valid = P.n - inv;
      st->dropped = drop;
      st->max_depth = __ldcg(&tally->max_depth);
      st->n_inter = 0;
      st->n_open = 0;
      *first_total = total;
      uint32_t warn = 0;
      if (inv) warn |= JC_WARN_NONFINITE;
      if (drop) warn |= JC_WARN_DEPTH_CAP;
      if (total > P.ref_cap) warn |= JC_WARN_REF_CAPACITY;
      if (warn) atomicOr(&st->warn, warn);
      st->n_tree = total > P.tree_cap ? 0u : total;
      if (total > P.tree_cap) set_error(st, JC_ERR_CAPACITY);
      tally->cursor = 0;
      tally->done = 0;
      tally->n_invalid = 0;
      tally->dropped = 0;
      tally->max_depth = 0;
    }
  }
}
