// core.cuh -- BC of the label-free index over a core graph (part of tree.cu).
//
// Where long shortcuts make the elimination tree too wide for labels, its first steps are still
// cheap: vertices of degree at most kCoreDegree are eliminated, least degree first, as long as their
// subtree stays a bottom (see k_bottom).  What is left is the core, a graph of 30 % of the vertices
// with shortcut lengths and path counts on its arcs; every eliminated vertex lies in a bottom whose
// separator is in the core.  So a source's sweep and dependency pass (k_sweep_rows and
// k_dependency_cta_pipe on the whole graph) are needed on the core alone:
//
//   k_core_up      U rows of a source that lies in a bottom: the core is entered at its separator
//   k_core_sweep   distances and path counts of the core, one CTA per source
//   k_core_rows    those as rows of a group's sources side by side
//   k_bottom       all bottoms, down and up
//   k_core_dep     dependencies of the core, waves in reverse, and the flow through its arcs
//   k_core_back    the flow back through the source's own bottom
//   k_fold, k_unpack
//
// The vertices have numbers of their own ("cid"): the core first, in vertex order, then the bottoms
// in preorder.  An edge belongs to its end of the larger number, so the lists serve k_bottom and the
// unpacking as they are.
#pragma once

// Degree up to 3, 4, 5, 6: 42, 30, 24, 20 % of the vertices stay, with 4.8 to 8 arcs each; 5,003
// vertices, all sources 2.23, 1.95, 2.05, 2.21 ms, 200k, 4,096 sources 64.4, 52.0, 53.6, 57.0 ms, 1M, 2,048
// sources 314, 166, 159, 167 ms.
constexpr int kCoreDegree = 4;
constexpr int kCoreCrowd = 64;  // no vertex next to a longer list is eliminated: it would be searched each time
constexpr int kCoreSort = 1024;                         // frontiers from here on are visited in vertex order,
constexpr int kCoreBuckets = 1024;                      // by so many ranges of vertices
// Threads per CTA, 2,048 per SM in any case.  A frontier is some tens of vertices of a small core and
// some hundreds of a large one; larger CTAs leave threads idle, smaller ones mean more sources at a time
// than L2 holds.  256, 512, 1,024 threads, 4,096 sources: 1.91, 2.46, 4.04 ms (5k vertices), 6.4, 6.7,
// 8.9 ms (25k: 7.5k in the core), 55.8, 52.7, 52.3 ms (200k), 640, 426, 329 ms (1M); a single source
// of 200k 6.4, 3.9, 2.8 ms.
constexpr int kCoreSmall = 8192;
constexpr int kCoreLarge = 40000;
constexpr int kCoreDelta = 2;                           // the core's bucket width in the graph's (1, 2, 3: within 2 %)
constexpr int kCoreChain = kBottomRows + 1;             // ancestors in a bottom, and the source itself
constexpr int kCoreH = kCoreChain + kBottomRows;        // rows of U: those by depth, then the separator

// An eliminated vertex's entries and the arcs of the core, on the host.
struct CoreShape {
  int32_t nc = 0, nbot = 0;
  std::vector<int32_t> cid_of, tid_of;                  // tid -> cid and back
  std::vector<int32_t> xoff, xtid, eL, eC;              // edges by their end of the larger cid
  std::vector<int32_t> depth, parent, send, tidx_of;
  std::vector<uint8_t> row_of;
  std::vector<int4> bot;
  std::vector<int4> arc, info, more;                    // see CoreArgs
};

struct CoreArgs {
  int nc;
  const int4 *arc;    // per core vertex four int4: eight arcs (head, length), head -1 where absent;
                      // more than eight: the last is (~first, end), arcs [first, end) of more
  const int4 *info;   // the same arcs' (path count, place in B of the flow head -> vertex)
  const int4 *more;   // (head, length, path count, place)
  int64_t E;          // edges: Bd, Bu, Bs follow each other
  int delta, max_rounds;
  int sort_shift, sort_buckets;
  int32_t *dist;      // [slots][nc]
  unsigned long long *word;  // [slots][nc] count | in-degree << 32 | successors << 48, then the bits of (1 + delta) / count
  int32_t *hop, *order, *lcnt;  // [slots][nc] staging; near list, then waves; [slots][2 (nc + 2)] lists, wave starts
  int32_t *waves;     // [slots]
};

__host__ __device__ inline int core_words(int nc) { return (nc + 31) / 32; }

// ------------------------------------------------------------------------------- U rows
// A warp per source: the vertices from the source to its bottom's root, lanes over the entries.
__global__ void __launch_bounds__(128) k_core_up(TreeArgs a) {
  __shared__ int32_t sd[4][32];
  __shared__ uint32_t sc[4][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = blockIdx.x * 4 + warp;
  if (slot >= a.ng * kGroup) return;
  const int s = a.src[min(slot, a.ns - 1)], bi = a.tidx_of[s];
  if (bi >= 0) return;
  int32_t *ud = sd[warp];
  uint32_t *uc = sc[warp];
  ud[lane] = INT_MAX;
  uc[lane] = 0;
  __syncwarp();
  const size_t gbase = (size_t)(slot / kGroup) * a.H * kGroup + slot % kGroup;
  const int4 bt = a.bot[-1 - bi];
  for (int y = s;; y = a.parent[y]) {
    const int row = a.row_of[y];  // (the source may be a leaf: it has no row)
    const int d = y == s ? 0 : ud[row];
    const uint32_t c = y == s ? 1u : uc[row];
    if (lane == 0) {
      const size_t u = gbase + (size_t)(a.depth[y] - 1) * kGroup;
      a.Ud[u] = d;
      a.Uc[u] = c;
    }
    const int e = a.xoff[y] + lane;
    if (e < a.xoff[y + 1] && (unsigned)d < a.dist_lim) {
      const int x = a.ex[e].x;
      const int4 v = a.eup[e];
      const int nd = d + v.y;
      if (nd <= ud[x]) {
        uc[x] = count_of(a, (unsigned long long)c * (unsigned)v.z + (nd == ud[x] ? uc[x] : 0u));
        ud[x] = nd;
      }
    }
    __syncwarp();
    if (y == bt.x) break;
  }
  if (lane < bt.z) {
    const size_t u = gbase + (size_t)(kCoreChain + lane) * kGroup;
    a.Ud[u] = ud[lane];
    a.Uc[u] = uc[lane];
  }
}

// The reverse: flow of a separator vertex that a U row reaches, share by share to the source's
// ancestors, the root first.
__global__ void __launch_bounds__(128) k_core_back(TreeArgs a, CoreArgs c) {
  __shared__ int32_t sd[4][32], path[4][kCoreChain];
  __shared__ uint32_t sc[4][32];
  __shared__ double sf[4][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = blockIdx.x * 4 + warp;
  if (slot >= a.ns || wrapped(a)) return;
  const int s = a.src[slot], bi = a.tidx_of[s];
  if (bi >= 0) return;
  int32_t *ud = sd[warp];
  uint32_t *uc = sc[warp];
  double *f = sf[warp];
  const size_t gbase = (size_t)(slot / kGroup) * a.H * kGroup + slot % kGroup;
  const int4 bt = a.bot[-1 - bi];
  const int depth = a.depth[s];
  if (lane < bt.z) {
    const size_t u = gbase + (size_t)(kCoreChain + lane) * kGroup;
    const size_t x = (size_t)slot * c.nc + a.etr[a.xoff[bt.x] + lane];
    ud[lane] = a.Ud[u];
    uc[lane] = a.Uc[u];
    f[lane] = c.dist[x] == ud[lane] ? (double)uc[lane] * __longlong_as_double((long long)c.word[x]) : 0.0;
  }
  if (lane == 0)
    for (int y = s, j = depth - 1; j >= 0; j--, y = a.parent[y]) path[warp][j] = y;
  __syncwarp();
  for (int j = 0; j < depth; j++) {
    const int y = path[warp][j];
    const size_t u = gbase + (size_t)j * kGroup;
    const int d = a.Ud[u];
    const uint32_t cy = a.Uc[u];
    const int e = a.xoff[y] + lane;
    double z = 0.0;
    if (e < a.xoff[y + 1]) {
      const int x = a.ex[e].x;
      const int4 v = a.eup[e];
      if (d + v.y == ud[x] && f[x] != 0.0) {
        z = share(v.z, cy, uc[x]) * f[x];
        atomicAdd((y == s ? a.Bs : a.Bu) + e, z);
      }
    }
    if (y == s) break;
    z = warp_sum(z);
    if (lane == 0) {
      const int row = a.row_of[y];
      ud[row] = d;
      uc[row] = cy;
      f[row] = z + a.seed[u];
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------------------- core sweep
struct CoreShared {
  int near_len, next_len, far_len, min_kept, tail, over;
};

// Four lanes per vertex, two arcs each: a frontier is some tens to hundreds of vertices, and all of a
// vertex's neighbours are loaded at once.  f(head, length, path count, place) for every arc.
__device__ __forceinline__ int core_more(int4 p, int lane4, int &end) {
  const bool more = lane4 == 3 && p.z < -1;
  end = more ? p.w : 0;
  return more ? ~p.z : 0;
}

// u's distance drops to nd: u joins a list unless it is there (a bit per vertex), and the minimum is
// left to the memory.  A distance read before another thread lowered it costs a visit, no more.
__device__ __forceinline__ void core_relax(int32_t *dist, int u, int nd, int T, int32_t *next, int32_t *far, uint32_t *in_next,
                                           uint32_t *in_far, CoreShared &sh) {
  atomicMin(dist + u, nd);
  const uint32_t bit = 1u << (u & 31);
  if (nd < T) {
    if (!(atomicOr(in_next + (u >> 5), bit) & bit)) next[atomicAdd(&sh.next_len, 1)] = u;
  } else if (!(atomicOr(in_far + (u >> 5), bit) & bit)) {
    far[atomicAdd(&sh.far_len, 1)] = u;
  }
}

// Bound by the latency of scattered loads that miss L1 (73 % of warp stalls; DRAM at 37 % of its rate
// with 16-byte records), so what counts is the footprint: distances are an array of their own, 4 bytes
// per vertex, and list membership is a bit in shared memory instead of a stamp in the record, which
// also leaves the relaxation nothing to wait for (the minimum returns no value).  200k vertices, 4,096
// sources: 44.6 ms with records and stamps, 31.4 ms so; the whole graph's sweep and dependency pass
// 182 ms, all of this path 52.
//
// Near-far buckets, then Kahn waves, as k_sweep_rows, from the source (in the core) or the separator
// of its bottom with the distances and counts of U.  A run that goes wrong in any way -- more passes
// than there can be, a count or distance too large -- sets the wrap word: the general sweep answers.
template <int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) k_core_sweep(TreeArgs a, CoreArgs c) {
  extern __shared__ uint32_t sm_bits[];
  __shared__ CoreShared sh;
  __shared__ int hist[kCoreBuckets];
  __shared__ int red[33];
  const int slot = blockIdx.x, tid = threadIdx.x, nc = c.nc;
  const int s = a.src[slot], bi = a.tidx_of[s];
  int32_t *dist = c.dist + (size_t)slot * nc;
  unsigned long long *word = c.word + (size_t)slot * nc;
  const int words = core_words(nc);
  uint32_t *in_next = sm_bits, *in_far = in_next + words;  // list membership, a bit per vertex
  int32_t *stage = c.hop + (size_t)slot * nc;
  int32_t *near = c.order + (size_t)slot * nc;
  int32_t *next = c.lcnt + (size_t)slot * 2 * (nc + 2), *far = next + (nc + 2);
  if (tid == 0) sh = CoreShared{};
  for (int v = tid; v < nc; v += THREADS) dist[v] = INT_MAX;
  for (int i = tid; i < 2 * words; i += THREADS) in_next[i] = 0;
  __syncthreads();
  const int delta = c.delta;
  int T = delta, pass = 0, round = 0;
  int seed_x = -1, seed_d = 0, seed_c = 1;  // this thread's
  if (bi >= 0) {
    if (tid == 0) seed_x = s;
  } else {
    const int4 bt = a.bot[-1 - bi];
    if (tid < bt.z) {
      const size_t u = ((size_t)(slot / kGroup) * a.H + kCoreChain + tid) * kGroup + slot % kGroup;
      seed_d = a.Ud[u];
      seed_c = (int)a.Uc[u];
      if ((unsigned)seed_d < a.dist_lim) seed_x = a.etr[a.xoff[bt.x] + tid];
    }
  }
  if (seed_x >= 0) {
    dist[seed_x] = seed_d;
    if (seed_d < T) {
      near[atomicAdd(&sh.near_len, 1)] = seed_x;
    } else {
      far[atomicAdd(&sh.far_len, 1)] = seed_x;
      atomicOr(in_far + (seed_x >> 5), 1u << (seed_x & 31));
    }
  }
  __syncthreads();
  bool failed = false;
  for (;;) {
    for (;;) {
      const int len = sh.near_len;
      if (len == 0) break;
      if (++pass > c.max_rounds) {
        failed = true;
        break;
      }
      const bool sorted = len >= kCoreSort;
      if (sorted)
        order_frontier<THREADS, kCoreBuckets>(
            c.sort_shift, c.sort_buckets, [&](int i) { return near[i]; }, len, [&](int i) -> int32_t & { return stage[i]; }, hist,
            red);
      for (int i = tid; i < 4 * len; i += THREADS) {
        const int v = sorted ? stage[i >> 2] : near[i >> 2], q = i & 3;
        const int4 p = __ldg(c.arc + 4 * (size_t)v + q);
        const int dv = dist[v];
        const int d0 = p.x >= 0 ? dist[p.x] : INT_MIN, d1 = p.z >= 0 ? dist[p.z] : INT_MIN;
        if (dv + p.y < d0) core_relax(dist, p.x, dv + p.y, T, next, far, in_next, in_far, sh);
        if (dv + p.w < d1) core_relax(dist, p.z, dv + p.w, T, next, far, in_next, in_far, sh);
        int end;
        for (int e = core_more(p, q, end); e < end; e++) {
          const int4 m = __ldg(c.more + e);
          if (dv + m.y < dist[m.x]) core_relax(dist, m.x, dv + m.y, T, next, far, in_next, in_far, sh);
        }
      }
      __syncthreads();
      const int nlen = sh.next_len;
      int32_t *t = near;
      near = next;
      next = t;
      for (int i = tid; i < nlen; i += THREADS) {
        const int v = near[i];
        atomicAnd(in_next + (v >> 5), ~(1u << (v & 31)));
      }
      __syncthreads();
      if (tid == 0) {
        sh.near_len = nlen;
        sh.next_len = 0;
      }
      __syncthreads();
    }
    if (failed) break;
    int T_old = T;
    T += delta;
    bool moved = false;
    while (!moved) {
      const int flen = sh.far_len;
      if (flen == 0 || ++round > c.max_rounds) break;
      __syncthreads();  // every thread has read far_len
      if (tid == 0) {
        sh.far_len = 0;
        sh.min_kept = INT_MAX;
      }
      __syncthreads();
      constexpr int kTile = 2;
      for (int base = 0; base < flen; base += THREADS * kTile) {
        int u[kTile], du[kTile];
#pragma unroll
        for (int q = 0; q < kTile; q++) {
          const int i = base + q * THREADS + tid;
          u[q] = i < flen ? far[i] : -1;
        }
#pragma unroll
        for (int q = 0; q < kTile; q++) du[q] = u[q] >= 0 ? dist[u[q]] : 0;
        __syncthreads();  // the tile is read before kept entries are written back in front of it
        int mn = INT_MAX;
#pragma unroll
        for (int q = 0; q < kTile; q++) {
          if (u[q] < 0) continue;
          if (du[q] >= T) {
            far[atomicAdd(&sh.far_len, 1)] = u[q];
            mn = min(mn, du[q]);
          } else {
            atomicAnd(in_far + (u[q] >> 5), ~(1u << (u[q] & 31)));
            if (du[q] >= T_old) near[atomicAdd(&sh.near_len, 1)] = u[q];  // (else settled in an earlier bucket)
          }
        }
        mn = __reduce_min_sync(kAll, mn);
        if ((tid & 31) == 0 && mn != INT_MAX) atomicMin(&sh.min_kept, mn);
        __syncthreads();
      }
      moved = sh.near_len > 0;
      if (!moved) {
        T_old = T;
        const int mk = sh.min_kept;
        if (mk != INT_MAX) T = max(T + delta, (mk / delta + 1) * delta);
      }
    }
    if (round > c.max_rounds) failed = true;
    if (failed || !moved) break;
  }
  if (failed) {
    if (tid == 0) *a.wrap = 1;
    return;
  }
  // in-degrees and successors (bits 0..7 of the mask; bit 8: some of the further arcs)
  int32_t *queue = c.order + (size_t)slot * nc;
  bool over = false;
  for (int i = tid; i < ((4 * nc + 31) & ~31); i += THREADS) {
    const bool in = i < 4 * nc;
    const int v = in ? i >> 2 : 0, q = i & 3;
    const int4 p = __ldg(c.arc + 4 * (size_t)v + q);
    const int dv = dist[v];
    const int d0 = p.x >= 0 ? dist[p.x] : INT_MIN, d1 = p.z >= 0 ? dist[p.z] : INT_MIN;
    int cnt = (p.x >= 0 && d0 + p.y == dv) + (p.z >= 0 && d1 + p.w == dv);
    int m = (p.x >= 0 && d0 == dv + p.y) << (2 * q) | (p.z >= 0 && d1 == dv + p.w) << (2 * q + 1);
    int end;
    for (int e = core_more(p, q, end); e < end; e++) {
      const int4 w = __ldg(c.more + e);
      const int dx = dist[w.x];
      cnt += dx + w.y == dv;
      m |= (dx == dv + w.y) << 8;
    }
    cnt += m << 16;
    cnt += __shfl_xor_sync(kAll, cnt, 1);
    cnt += __shfl_xor_sync(kAll, cnt, 2);
    if (in && q == 0) {
      over |= (unsigned)dv >= a.dist_lim;
      word[v] = (unsigned long long)(unsigned)cnt << 32;
      if ((cnt & 0xffff) == 0) queue[atomicAdd(&sh.tail, 1)] = v;
    }
  }
  __syncthreads();
  if (seed_x >= 0 && dist[seed_x] == seed_d) word[seed_x] |= (unsigned)seed_c;
  __syncthreads();
  int L = 0, b = 0, e = sh.tail;
  int32_t *wave = c.lcnt + (size_t)slot * 2 * (nc + 2), *wstart = wave + (nc + 2);
  while (b < e) {
    if (tid == 0) wstart[L] = b;
    const bool sorted = e - b >= kCoreSort;
    if (sorted)
      order_frontier<THREADS, kCoreBuckets>(
          c.sort_shift, c.sort_buckets, [&](int i) { return queue[b + i]; }, e - b, [&](int i) -> int32_t & { return wave[i]; },
          hist, red);
    for (int i = tid; i < 4 * (e - b); i += THREADS) {
      const int v = sorted ? wave[i >> 2] : queue[b + (i >> 2)], q = i & 3;
      if (sorted && q == 0) queue[b + (i >> 2)] = v;
      const int4 p = __ldg(c.arc + 4 * (size_t)v + q), f = __ldg(c.info + 4 * (size_t)v + q);
      const unsigned long long r = word[v];
      const unsigned mask = (unsigned)(r >> 48);
      auto push = [&](int h, int paths) {
        const unsigned long long inc = (r & 0xffffffffull) * (unsigned)paths;
        if (inc > 0x7fffffffull) {
          over = true;
          paths = 0;
        }
        // count += inc, in-degree -= 1
        const unsigned long long old = atomicAdd(word + h, (paths ? inc : 0ull) - (1ull << 32));
        over |= (old & 0xffffffffull) + inc > 0x7fffffffull;
        if (((unsigned)(old >> 32) & 0xffff) == 1u) queue[atomicAdd(&sh.tail, 1)] = h;  // its last predecessor
      };
      if ((mask >> (2 * q)) & 1) push(p.x, f.x);
      if ((mask >> (2 * q)) & 2) push(p.z, f.z);
      if (mask & 256) {
        int end;
        for (int x = core_more(p, q, end); x < end; x++) {
          const int4 m = __ldg(c.more + x);
          if (dist[m.x] == dist[v] + m.y) push(m.x, m.z);
        }
      }
    }
    __syncthreads();
    b = e;
    e = sh.tail;
    L++;
    __syncthreads();  // every thread has read the tail before the next wave moves it
  }
  if (over || e != nc) *a.wrap = 1;
  if (tid == 0) {
    wstart[L] = e;
    c.waves[slot] = L;
  }
}

// distances and counts of a group's sources side by side, delta cleared
__global__ void __launch_bounds__(256) k_core_rows(TreeArgs a, CoreArgs c) {
  __shared__ uint2 tile[32][kGroup + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = blockIdx.y, v0 = blockIdx.x * 32;
  for (int k = warp; k < kGroup; k += 8) {
    const int slot = min(g * kGroup + k, a.ns - 1);
    if (v0 + lane < c.nc) {
      const size_t x = (size_t)slot * c.nc + v0 + lane;
      tile[lane][k] = make_uint2((unsigned)c.dist[x] << a.bits, (unsigned)c.word[x]);
    }
  }
  __syncthreads();
  for (int i = warp; i < 32 && v0 + i < c.nc; i += 8) {
    const size_t o = ((size_t)g * a.NT + v0 + i) * kGroup + 2 * lane;
    const uint2 x = tile[i][2 * lane], y = tile[i][2 * lane + 1];
    *reinterpret_cast<uint2 *>(a.D + o) = make_uint2(x.x, y.x);
    *reinterpret_cast<uint2 *>(a.S + o) = make_uint2(x.y, y.y);
    *reinterpret_cast<double2 *>(a.J + o) = make_double2(0.0, 0.0);
  }
}

// Dependencies, waves in reverse: delta = J (from the bottoms) + sum of the successors' shares.  The
// flow through an arc is added to the edge's total whichever way it runs; those totals give the core's
// own dependencies, too (k_fold), so a vertex costs about one atomic per source, as before.  11.6 ms of
// 52 at 200k vertices and 4,096 sources, 342 us of 1.95 ms for all sources of 5k.
template <int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) k_core_dep(TreeArgs a, CoreArgs c) {
  if (__syncthreads_or(wrapped(a))) return;
  const int slot = blockIdx.x, tid = threadIdx.x, nc = c.nc;
  const int s = a.src[slot];
  const int32_t *dist = c.dist + (size_t)slot * nc;
  unsigned long long *word = c.word + (size_t)slot * nc;
  const int32_t *queue = c.order + (size_t)slot * nc;
  const int32_t *wstart = c.lcnt + (size_t)slot * 2 * (nc + 2) + (nc + 2);
  const double *J = a.J + (size_t)(slot / kGroup) * a.NT * kGroup + slot % kGroup;
  int e = nc;
  for (int L = c.waves[slot] - 1; L >= 0; L--) {
    const int b = wstart[L];
    for (int i = tid; i < ((4 * (e - b) + 31) & ~31); i += THREADS) {
      const bool in = i < 4 * (e - b);
      const int v = queue[in ? b + (i >> 2) : b], q = i & 3;
      const int4 p = __ldg(c.arc + 4 * (size_t)v + q), f = __ldg(c.info + 4 * (size_t)v + q);
      const unsigned long long r = word[v];
      const double j = J[(size_t)v * kGroup];
      const unsigned mask = in ? (unsigned)(r >> 48) : 0u;
      const bool h0 = (mask >> (2 * q)) & 1, h1 = (mask >> (2 * q)) & 2;
      auto rho = [&](int h) { return __longlong_as_double((long long)word[h]); };
      const double sigma = (double)(unsigned)r;
      const double z0 = h0 ? rho(p.x) * (double)f.x : 0.0, z1 = h1 ? rho(p.z) * (double)f.z : 0.0;
      const int64_t own = 2 * c.E;  // flow into the source itself counts apart
      auto add = [&](int place, double z) { atomicAdd(a.Bd + (v == s ? own + (place >= c.E ? place - c.E : place) : place), z * sigma); };
      if (h0) add(f.y, z0);
      if (h1) add(f.w, z1);
      double z = z0 + z1;
      if (mask & 256) {
        int end;
        for (int x = core_more(p, q, end); x < end; x++) {
          const int4 m = __ldg(c.more + x);
          if (dist[m.x] == dist[v] + m.y) {
            const double w = rho(m.x) * (double)m.z;
            add(m.w, w);
            z += w;
          }
        }
      }
      z += __shfl_xor_sync(kAll, z, 1);
      z += __shfl_xor_sync(kAll, z, 2);
      if (in && q == 0) word[v] = (unsigned long long)__double_as_longlong((j + 1.0) / sigma + z);
    }
    __syncthreads();
    e = b;
  }
}

__global__ void k_core_src(const int32_t *__restrict__ tid, const int32_t *__restrict__ cid_of, int ns, int32_t *cid) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ns) cid[i] = cid_of[tid[i]];
}

__global__ void k_core_finish(const double *__restrict__ F, const int32_t *__restrict__ cid_of, double *__restrict__ bc_tid, int n,
                              const int32_t *err) {
  if (result_void(err)) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) bc_tid[t] += 0.5 * F[cid_of[t]];
}

// ------------------------------------------------------------------------------- plan
// f(begin, end) over ranges of [0, count) on a few threads; f does not throw
template <class F>
static void core_ranges(int32_t count, F &&f) {
  const int nt = count < 20000 ? 1 : (int)std::min(8u, std::max(1u, std::thread::hardware_concurrency()));
  std::vector<std::thread> ts;
  ts.reserve((size_t)nt);
  for (int t = 0; t < nt; t++) {
    const int32_t b = (int32_t)((int64_t)count * t / nt), e = (int32_t)((int64_t)count * (t + 1) / nt);
    if (t + 1 < nt) {
      try {
        ts.emplace_back([&f, b, e] { f(b, e); });
        continue;
      } catch (const std::system_error &) {  // no thread to be had
      }
    }
    f(b, e);
  }
  for (std::thread &t : ts) t.join();
}

// The elimination, of paired arcs (Index::arcs_paired); false where no plan is possible (a count past 2^31, a degree past the sweep's, or
// lengths below 1, which a graph has none of but a file might).
static bool core_shape(const Index &ix, CoreShape &s) {
  const int32_t n = ix.n;
  struct Ent {
    int32_t h, L, C;
  };
  struct List {
    int64_t off;
    int32_t len, cap;
  };
  // lists with room for one more entry each; a list that grows past its room moves to the end
  std::vector<List> adj((size_t)n);
  int64_t room = 2 * ((int64_t)ix.arc_off[n] + n), used = (int64_t)ix.arc_off[n] + n;
  std::unique_ptr<Ent[]> pool(new Ent[(size_t)room]);
  std::atomic<bool> ok{true};
  core_ranges(n, [&](int32_t v0, int32_t v1) {
    for (int32_t v = v0; v < v1; v++) {
      const int32_t b = ix.arc_off[v], e = ix.arc_off[v + 1];
      adj[v] = {(int64_t)b + v, e - b, e - b + 1};
      for (int32_t q = b; q < e; q++) {
        if (ix.arc_w[q] < 1) ok = false;
        pool[(int64_t)q + v] = {ix.arc_head[q], ix.arc_w[q], 1};
      }
    }
  });
  if (!ok) return false;
  auto find = [&](int32_t u, int32_t h) {
    for (int32_t q = 0; q < adj[u].len; q++)
      if (pool[adj[u].off + q].h == h) return q;
    return -1;
  };
  // eliminated vertices: entries, state of the subtree; pending roots per live vertex (4 links each)
  std::unique_ptr<Ent[]> xs(new Ent[(size_t)n * kCoreDegree]);
  std::vector<int8_t> nx((size_t)n, -1);  // entries of an eliminated vertex; -1 live, -2 live for good
  std::vector<uint8_t> size((size_t)n, 0), inner((size_t)n, 0), edges((size_t)n, 0);
  std::vector<int32_t> up((size_t)n, -1), head((size_t)n, -1);
  std::unique_ptr<int32_t[]> link(new int32_t[(size_t)n * kCoreDegree]);
  std::vector<std::vector<int32_t>> bucket(kCoreDegree + 1);
  for (int32_t v = n - 1; v >= 0; v--)
    if (adj[v].len >= 1 && adj[v].len <= kCoreDegree) bucket[adj[v].len].push_back(v);
  std::vector<int32_t> kids;
  for (int d = 1; d <= kCoreDegree;) {
    if (bucket[d].empty()) {
      d++;
      continue;
    }
    const int32_t v = bucket[d].back();
    bucket[d].pop_back();
    if (nx[v] != -1 || adj[v].len != d) continue;
    const int k = d;
    bool crowded = false;  // next to a hub: finding v in its list would take long
    for (int i = 0; i < k; i++) crowded |= adj[pool[adj[v].off + i].h].len > kCoreCrowd;
    kids.clear();
    int sz = 1, in = 0, ed = k;
    for (int32_t l = head[v]; l >= 0 && sz <= kBottomVerts; l = link[l]) {
      const int32_t u = l / kCoreDegree;
      if (up[u] >= 0) continue;
      kids.push_back(u);
      sz += size[u];
      in += inner[u];
      ed += edges[u];
    }
    in += !kids.empty();
    if (crowded || sz > kBottomVerts || k + in > kBottomRows || ed > kBottomEdges) {
      nx[v] = -2;
      continue;
    }
    for (int32_t u : kids) up[u] = v;
    size[v] = (uint8_t)sz;
    inner[v] = (uint8_t)in;
    edges[v] = (uint8_t)ed;
    nx[v] = (int8_t)k;
    Ent *x = xs.get() + (size_t)v * kCoreDegree;
    for (int i = 0; i < k; i++) {
      x[i] = pool[adj[v].off + i];
      link[(size_t)v * kCoreDegree + i] = head[x[i].h];
      head[x[i].h] = v * kCoreDegree + i;
    }
    for (int i = 0; i < k; i++) {
      List &a = adj[x[i].h];
      pool[a.off + find(x[i].h, v)] = pool[a.off + a.len - 1];
      a.len--;
      for (int j = 0; j < k; j++) {
        if (j == i) continue;
        const int32_t L = x[i].L + x[j].L;
        const int64_t C = (int64_t)x[i].C * x[j].C;
        const int32_t q = find(x[i].h, x[j].h);
        if (q < 0) {
          if (C > INT_MAX) return false;
          if (a.len == a.cap) {
            if (used + 2 * a.cap > room) {
              room = 2 * room + 2 * a.cap;
              std::unique_ptr<Ent[]> larger(new Ent[(size_t)room]);
              std::copy(pool.get(), pool.get() + used, larger.get());
              pool.swap(larger);
            }
            std::copy(pool.get() + a.off, pool.get() + a.off + a.len, pool.get() + used);
            a.off = used;
            a.cap *= 2;
            used += a.cap;
          }
          pool[a.off + a.len++] = {x[j].h, L, (int32_t)C};
        } else {
          Ent &f = pool[a.off + q];
          if (L > f.L) continue;
          const int64_t sum = L < f.L ? C : C + f.C;
          if (sum > INT_MAX) return false;
          f.L = L;
          f.C = (int32_t)sum;
        }
      }
      if (a.len >= 1 && a.len <= kCoreDegree) {
        bucket[a.len].push_back(x[i].h);
        d = std::min(d, (int)a.len);
      }
    }
  }
  // numbers: the core, then each bottom in preorder
  s.cid_of.resize((size_t)n);
  s.tid_of.resize((size_t)n);
  for (int32_t v = 0; v < n; v++)
    if (nx[v] < 0) {
      s.cid_of[v] = s.nc;
      s.tid_of[s.nc++] = v;
    }
  std::vector<int32_t> child((size_t)n, -1), sibling((size_t)n, -1), stack;
  for (int32_t v = n - 1; v >= 0; v--)
    if (up[v] >= 0) {
      sibling[v] = child[up[v]];
      child[up[v]] = v;
    }
  s.depth.assign((size_t)n, 1);
  s.parent.assign((size_t)n, -1);
  s.send.resize((size_t)n);
  s.tidx_of.resize((size_t)n);
  s.row_of.assign((size_t)n, 0xff);
  for (int32_t c = 0; c < s.nc; c++) {
    s.send[c] = c + 1;
    s.tidx_of[c] = c;
  }
  int32_t at_cid = s.nc;
  for (int32_t v = 0; v < n; v++) {
    if (nx[v] < 0 || up[v] >= 0) continue;
    s.bot.push_back(make_int4(at_cid, size[v], nx[v], nx[v] + inner[v]));
    int row = nx[v];
    stack.assign(1, v);
    while (!stack.empty()) {
      const int32_t t = stack.back();
      stack.pop_back();
      const int32_t c = at_cid++;
      s.cid_of[t] = c;
      s.tid_of[c] = t;
      s.send[c] = c + size[t];
      if (up[t] >= 0) {
        s.parent[c] = s.cid_of[up[t]];
        s.depth[c] = s.depth[s.parent[c]] + 1;
      }
      if (child[t] >= 0) s.row_of[c] = (uint8_t)row++;
      for (int32_t k = child[t]; k >= 0; k = sibling[k]) stack.push_back(k);
    }
  }
  s.nbot = (int32_t)s.bot.size();
  std::stable_sort(s.bot.begin(), s.bot.end(), [](const int4 &x, const int4 &y) { return x.w > y.w; });
  for (int32_t i = 0; i < s.nbot; i++)
    for (int32_t c = s.bot[i].x; c < s.bot[i].x + s.bot[i].y; c++) s.tidx_of[c] = -1 - i;
  // edges, then the core's arcs
  auto list_of = [&](int32_t t) { return nx[t] < 0 ? pool.get() + adj[t].off : xs.get() + (size_t)t * kCoreDegree; };
  auto length_of = [&](int32_t t) { return nx[t] < 0 ? adj[t].len : (int32_t)nx[t]; };
  s.xoff.assign((size_t)n + 1, 0);
  core_ranges(n, [&](int32_t c0, int32_t c1) {
    for (int32_t c = c0; c < c1; c++) {
      const Ent *x = list_of(s.tid_of[c]);
      for (int32_t q = 0; q < length_of(s.tid_of[c]); q++) s.xoff[c + 1] += s.cid_of[x[q].h] < c;
    }
  });
  int64_t total = 0;
  for (int32_t c = 0; c < n; c++) {
    total += s.xoff[c + 1];
    if (total >= INT_MAX / 2) return false;
    s.xoff[c + 1] = (int32_t)total;
  }
  const int32_t E = (int32_t)total;
  s.xtid.resize((size_t)E);
  s.eL.resize((size_t)E);
  s.eC.resize((size_t)E);
  core_ranges(n, [&](int32_t c0, int32_t c1) {
    for (int32_t c = c0; c < c1; c++) {
      Ent *x = list_of(s.tid_of[c]);
      const int32_t k = length_of(s.tid_of[c]);
      std::sort(x, x + k, [&](const Ent &p, const Ent &q) { return s.cid_of[p.h] < s.cid_of[q.h]; });
      for (int32_t q = 0, e = s.xoff[c]; e < s.xoff[c + 1]; q++, e++) {  // (those below c come first)
        s.xtid[e] = s.cid_of[x[q].h];
        s.eL[e] = x[q].L;
        s.eC[e] = x[q].C;
      }
    }
  });
  const int4 none = make_int4(-1, 0, -1, 0);
  s.arc.assign((size_t)s.nc * 4, none);
  s.info.assign((size_t)s.nc * 4, make_int4(0, 0, 0, 0));
  s.more.assign(1, none);  // (~0 would read as an absent arc)
  for (int32_t c = 0; c < s.nc; c++) {
    const int32_t k = adj[s.tid_of[c]].len;
    if (k > 60000) return false;  // (in-degrees are summed in 16 bits)
    if (k <= 8) continue;
    s.arc[(size_t)c * 4 + 3].z = ~(int32_t)s.more.size();
    s.more.resize(s.more.size() + k - 7);
    s.arc[(size_t)c * 4 + 3].w = (int32_t)s.more.size();
  }
  core_ranges(s.nc, [&](int32_t c0, int32_t c1) {
    for (int32_t c = c0; c < c1; c++) {
      const int32_t t = s.tid_of[c], k = adj[t].len, direct = k > 8 ? 7 : k;
      const Ent *x = list_of(t);
      for (int32_t q = 0; q < k; q++) {
        const int32_t h = s.cid_of[x[q].h], own = std::max(h, c), other = std::min(h, c);
        const int32_t e = (int32_t)(std::lower_bound(s.xtid.begin() + s.xoff[own], s.xtid.begin() + s.xoff[own + 1], other) -
                                    s.xtid.begin());
        const int32_t place = c < h ? e : E + e;  // flow from h to c: down (c is the smaller end) or up
        if (q < direct) {
          int4 &p = s.arc[(size_t)c * 4 + q / 2], &f = s.info[(size_t)c * 4 + q / 2];
          (q & 1 ? p.z : p.x) = h;
          (q & 1 ? p.w : p.y) = x[q].L;
          (q & 1 ? f.z : f.x) = x[q].C;
          (q & 1 ? f.w : f.y) = place;
        } else {
          s.more[~s.arc[(size_t)c * 4 + 3].z + q - direct] = make_int4(h, x[q].L, x[q].C, place);
        }
      }
    }
  });
  return s.nc >= 1;
}
