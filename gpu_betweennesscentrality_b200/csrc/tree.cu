// tree.cu -- BC over the elimination tree of libqbc_b200 (label indexes: MHL and H2H).
//
// The label scan computes a source's distances and path counts pair by pair: d(s, t) is a minimum
// over every common ancestor of s and t, hundreds to thousands of label entries per pair
// (MHLQBC.cu:379-392).  For BC the rows of one source are wanted for all targets at once, and then
// the elimination tree gives them with far less work.  X(t) is t's separator: the vertices adjacent
// to t when it was eliminated, all of them ancestors, with shortcut lengths L and path counts C over
// vertices eliminated before t.  The last vertex above t on a path s -> t lies in X(t), so
//
//   D_s(t) = U_s(t)  (+)  (+)_{x in X(t)} D_s(x) (x) (L, C)(t, x)                        (down)
//   U_s(s) = (0, 1),  U_s(x) = (+)_{y below x, x in X(y)} U_s(y) (x) (L, C)(y, x)        (up)
//
// where (+) keeps the least length and adds the counts of ties, (x) adds lengths and multiplies
// counts, and U_s(t) (t an ancestor of s or s itself) holds the paths whose highest vertex is t.
// Every shortest path is counted once.  A pair costs |X(t)| entries instead of h(lca(s, t)): 7.5
// against 229 at 50k vertices, 11.7 against about 1,900 at 1M.
//
// Dependencies (MHLQBC.cu:452-466) are the reverse of that recursion.  delta_s(t) is what t's
// descendants hand up; t hands its flow delta_s(t) + 1 on to the entries its shortest paths come
// from, to each x its share C(t, x) sigma_s(x) / sigma_s(t) -- all of it where one entry is the only
// one, so counts are needed for ties alone.  B(t, x) sums, over all sources, the flow through the
// shortcut itself.  The paths through the inside of a shortcut are unpacked once per call: a shortcut
// (t, x) of least length through y is two shortcuts (y, t), (y, x) ("triangle"), so its share of B
// passes to the two and is dependency of y.  No hop layer, no per-source ordering and no scattered
// gathers are left: all sources visit the vertices in the same order, 32 sources per warp.
//
//   k_up_gather, k_up_rows  U rows: the source's label row, or along its ancestors
//   k_trunk_down            D of the vertices near the root ("trunk"), pieces of a path level by level
//   k_bottom                every small subtree below the trunk, down and up in shared memory
//   k_trunk_up              delta of the trunk, levels in reverse
//   k_up_back               the reverse of the U rows
//   k_fold, k_unpack        B over the triangles, level by level, once per call
//
// Counts are held in 32 bits as in the label rows.  Those wrap where the true count passes 2^31, and
// BC is then defined by the wrapped values; here a product that reaches 2^31 sets the wrap word, the
// kernels leave their results unused, and the call is answered by the label kernels, as are all calls
// after it.  (A sum over entries that a shorter one beats later may set it, too.)
//
// All 50,175 sources of the 50k grid: 239.8 ms by the label kernels (label scan 142, dependency pass
// 77, sorting and gaps), 37.1 ms so; 1,024 sources of 500k 150.8 and 22.1 ms, 6,083 of 6k 3.33 and 1.15.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdlib>
#include <memory>
#include <system_error>
#include <thread>
#include <type_traits>

#include "device_state.h"
#include "frontier.cuh"

namespace qbc {

namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr unsigned kNoKey = 0xffffffffu;
constexpr int kGroup = 64;           // sources a warp takes: two neighbouring ones per lane
constexpr int kPieceLen = 32;        // trunk vertices per piece
// a bottom subtree: rows in shared memory (its separator and its vertices with descendants), vertices, edges
// (12, 16, 20 rows, all sources of 50k: 43.3, 42.5, 43.2 ms)
constexpr int kBottomRows = 16;
constexpr int kBottomVerts = 64;
constexpr int kBottomEdges = 224;
constexpr int kMaxUnpackLevels = 1024;

struct TreeArgs {
  int n, H, NT, bits;
  unsigned dist_lim;               // distances of shortest paths are below it
  unsigned absent;                 // key of a missing entry: above every distance
  const int32_t *xoff;             // [n + 1] edge range of a vertex
  const int2 *ex;                  // per edge (x: trunk index or bottom row, (L << bits) | (i + 1))
  const int4 *eup;                 // per edge (depth(x) - 1, L, path count, tid of x)
  const int32_t *eC;               // per edge path count
  const int32_t *etr;              // per edge trunk index of x (separators of bottom roots)
  const int4 *tmeta;               // per trunk vertex (first edge, end edge, edges inside its piece, tid)
  const int2 *tsub;                // per trunk vertex (subtree end, depth - 1)
  const int4 *piece;               // (first trunk index, end, trunk index of the parent or -1, 0)
  const int32_t *piece_of;         // per trunk vertex
  const int32_t *chain_off;        // per piece: the pieces above it, root first, and itself, as
  const int2 *chain;               // (first trunk index, depth - 1 of that vertex)
  const int32_t *tidx_of;          // per tid: trunk index, or -1 - bottom
  const int4 *bot;                 // bottoms: (root tid, size, separator size, rows)
  const uint8_t *row_of;           // per tid in a bottom: its row, 0xff without descendants
  const int32_t *depth, *parent, *send;
  const int64_t *lab_off;          // label rows (MHL): distances, shifted by lab_bits, and (count, hop)
  const int32_t *lab_dis;
  const int2 *lab_ch;
  int lab_bits;
  const int32_t *src;              // tids of this launch's sources
  int ns, ng;                      // sources, groups of kGroup
  uint32_t *D;                     // [ng][NT][kGroup] distance << bits
  uint32_t *S;
  uint32_t *arg;
  double *J;                       // delta
  int32_t *Ud;                     // [ng][H][kGroup]
  uint32_t *Uc;
  double *seed;                    // flow of the paths whose highest vertex is the ancestor
  double *Bd, *Bu, *Bs;            // per edge: flow on the way down, up, and from x's or y's own source
  double *F;                       // per vertex (tid): dependency
  int32_t *wrap;
};

__device__ __forceinline__ bool wrapped(const TreeArgs &a) { return __ldcg(a.wrap) != 0; }

// Launched by launch_early, a kernel starts while the one before it still runs: what it reads above
// wait_before must be older than that one, and lets the next one start from let_next on.
__device__ __forceinline__ void let_next() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void wait_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ uint32_t count_of(const TreeArgs &a, unsigned long long c) {
  if (c > 0x7fffffffull) {
    *a.wrap = 1;
    return 1u;
  }
  return (uint32_t)c;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(kAll, v, o);
  return v;
}

// c * x / y of counts; 1 where the only entry carries the whole count
__device__ __forceinline__ double share(int c, uint32_t x, uint32_t y) {
  const unsigned long long p = (unsigned long long)(unsigned)c * x;
  return p == y ? 1.0 : (double)p / (double)y;
}

// the two sources of a lane of group g (slots past the end repeat the last source; live tells them apart)
__device__ __forceinline__ void lane_sources(const TreeArgs &a, int g, int lane, int (&s)[2], bool (&live)[2]) {
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int slot = g * kGroup + 2 * lane + k;
    live[k] = slot < a.ns;
    s[k] = a.src[min(slot, a.ns - 1)];
  }
}

// The minimum of a pair is kept as two keys, (distance, entry index) and the same with the index
// complemented; their indices differ where several entries reach it.  arg = smallest index |
// largest << 16: equal for one entry, smallest < largest for exactly two, swapped for more.
__device__ __forceinline__ void key_min2(unsigned &m1, unsigned &m2, unsigned v, unsigned w, unsigned mask) {
  m1 = __vimin3_u32(m1, v, w);
  m2 = __vimin3_u32(m2, v ^ mask, w ^ mask);
}

// ------------------------------------------------------------------------------- up
// U rows from the label rows (MHL): row s is U_s, transposed here so that a group's sources lie
// side by side.
__global__ void __launch_bounds__(1024) k_up_gather(TreeArgs a) {
  __shared__ int sd[kGroup][33];
  __shared__ unsigned sc[kGroup][33];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = blockIdx.x;
  int h[2];
  int64_t off[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int s = a.src[min(g * kGroup + 2 * warp + k, a.ns - 1)];
    h[k] = a.depth[s];
    off[k] = a.lab_off[s];
  }
  for (int j0 = blockIdx.y * 32; j0 < a.H; j0 += gridDim.y * 32) {
    if (!__syncthreads_or(j0 < max(h[0], h[1]))) break;  // past every row of the group
    const int j = j0 + lane;
#pragma unroll
    for (int k = 0; k < 2; k++)
      if (j < h[k]) {
        sd[2 * warp + k][lane] = (int)((unsigned)a.lab_dis[off[k] + j] >> a.lab_bits);
        sc[2 * warp + k][lane] = (unsigned)a.lab_ch[off[k] + j].x;
      }
    __syncthreads();
    if (j0 + warp < a.H) {
      const size_t o = ((size_t)g * a.H + j0 + warp) * kGroup + 2 * lane;
      *reinterpret_cast<int2 *>(a.Ud + o) = make_int2(sd[2 * lane][warp], sd[2 * lane + 1][warp]);
      *reinterpret_cast<uint2 *>(a.Uc + o) = make_uint2(sc[2 * lane][warp], sc[2 * lane + 1][warp]);
    }
    __syncthreads();
  }
}

// U rows without count labels (H2H): a warp follows one source's ancestors, lanes over the separator
// of the current one.  The ancestors of a trunk vertex come a piece at a time (consecutive trunk
// indices), so the pointer chase is one step per piece; the next ancestor's first 32 edges are in
// flight while the current one's are applied.
__global__ void k_up_rows(TreeArgs a) {
  extern __shared__ int32_t sm_up[];
  if (wrapped(a)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int slot = blockIdx.x * nw + warp;
  if (slot >= a.ng * kGroup) return;
  int32_t *ud = sm_up + (size_t)warp * 2 * a.H;
  uint32_t *uc = reinterpret_cast<uint32_t *>(ud + a.H);
  const int s = a.src[min(slot, a.ns - 1)];
  const int h = a.depth[s];
  for (int j = lane; j < h; j += 32) {
    ud[j] = INT_MAX;
    uc[j] = 0;
  }
  __syncwarp();
  if (lane == 0) {
    ud[h - 1] = 0;
    uc[h - 1] = 1;
  }
  __syncwarp();
  int j = h - 1;
  auto first = [&](int e0, int e1) { return e0 + lane < e1 ? __ldg(a.eup + e0 + lane) : make_int4(-1, 0, 0, 0); };
  auto relax = [&](int4 v, int e0, int e1) {
    const int d = ud[j];
    if ((unsigned)d < a.dist_lim) {
      const unsigned c = uc[j];
      for (int e = e0 + lane;;) {
        if (v.x >= 0) {
          const int nd = d + v.y;
          if (nd <= ud[v.x]) {
            uc[v.x] = count_of(a, (unsigned long long)c * (unsigned)v.z + (nd == ud[v.x] ? uc[v.x] : 0u));
            ud[v.x] = nd;
          }
        }
        e += 32;
        if (e >= e1) break;
        v = __ldg(a.eup + e);
      }
    }
    __syncwarp();
    j--;
  };
  int y = s, i = a.tidx_of[y];
  while (i < 0 && j >= 0) {
    const int e0 = a.xoff[y], e1 = a.xoff[y + 1];
    relax(first(e0, e1), e0, e1);
    y = a.parent[y];
    i = y >= 0 ? a.tidx_of[y] : 0;
  }
  while (j >= 0) {
    const int4 pc = a.piece[a.piece_of[i]];
    const int cnt = i - pc.x + 1;
    const int4 m = lane < cnt ? a.tmeta[pc.x + lane] : make_int4(0, 0, 0, 0);
    int e0 = __shfl_sync(kAll, m.x, cnt - 1), e1 = __shfl_sync(kAll, m.y, cnt - 1);
    int4 v = first(e0, e1);
    for (int k = cnt - 1; k >= 0; k--) {
      const int n0 = __shfl_sync(kAll, m.x, max(k - 1, 0)), n1 = __shfl_sync(kAll, m.y, max(k - 1, 0));
      const int4 vn = first(n0, n1);
      relax(v, e0, e1);
      v = vn;
      e0 = n0;
      e1 = n1;
    }
    i = pc.z;
  }
  const size_t gbase = (size_t)(slot / kGroup) * a.H * kGroup + slot % kGroup;
  for (int q = lane; q < h; q += 32) {
    a.Ud[gbase + (size_t)q * kGroup] = ud[q];
    a.Uc[gbase + (size_t)q * kGroup] = uc[q];
  }
}

// The label kernels' source rows (k_src_rows: a source's ancestors, root first, then their subtree
// ends) from the plan: a warp per source, a run of ancestors per step instead of one parent link
// after another (a chain of 477 dependent loads at 50k vertices).
__global__ void k_source_rows(TreeArgs a, int stride, int32_t *rows) {
  const int slot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (slot >= a.ns) return;
  int32_t *lo = rows + (size_t)slot * 2 * stride, *hi = lo + stride;
  int y = a.src[slot], j = a.depth[y] - 1, i = a.tidx_of[y];
  while (i < 0 && j >= 0) {
    if (lane == 0) {
      lo[j] = y;
      hi[j] = a.send[y];
    }
    j--;
    y = a.parent[y];
    i = y >= 0 ? a.tidx_of[y] : 0;
  }
  if (j < 0) return;
  const int pc = a.piece_of[i], c0 = a.chain_off[pc], c1 = a.chain_off[pc + 1];
#pragma unroll 4
  for (int c = c0; c < c1; c++) {
    const int2 run = a.chain[c];
    const int end = c + 1 < c1 ? a.chain[c + 1].y : j + 1;
    if (run.y + lane < end) {
      lo[run.y + lane] = a.tmeta[run.x + lane].w;
      hi[run.y + lane] = a.tsub[run.x + lane].x;
    }
  }
}

// Reverse of the U rows, a CTA per source, root first: the flow of y is its seed plus its share of the
// flow of the separator entries x with U(y) + L = U(x).  Each warp takes a block of 32 ancestors and
// collects the entries that hold (independent loads, the next ancestor's in flight); one warp then
// applies the blocks in order in shared memory, and all add the shortcuts' flow.
// Many sources: four warps, so that more CTAs wait at a time; few: eight, for the shorter wait.
constexpr int kBackHits = 160;  // entries collected per block; a block with more is done by one warp in turns
template <int BW>
struct BackShared {
  int2 hit[BW][kBackHits];  // (edge, x's depth | y's depth << 16)
  double ratio[BW][kBackHits];
  int count[BW];
};

template <int BW>
__global__ void __launch_bounds__(BW * 32) k_up_back(TreeArgs a) {
  extern __shared__ double sm_back[];
  __shared__ BackShared<BW> sh;
  if (__syncthreads_or(wrapped(a))) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nt = blockDim.x;
  const int slot = blockIdx.x;
  double *ub = sm_back;
  int32_t *ud = reinterpret_cast<int32_t *>(ub + a.H), *path = ud + a.H;  // path: trunk index or -1 - tid
  uint32_t *uc = reinterpret_cast<uint32_t *>(path + a.H);
  const int s = a.src[slot], h = a.depth[s];
  const size_t gbase = (size_t)(slot / kGroup) * a.H * kGroup + slot % kGroup;
  for (int q = threadIdx.x; q < h; q += nt) {
    ud[q] = a.Ud[gbase + (size_t)q * kGroup];
    uc[q] = a.Uc[gbase + (size_t)q * kGroup];
    ub[q] = a.seed[gbase + (size_t)q * kGroup];
  }
  {
    int j = h - 1, y = s, i = a.tidx_of[y];
    while (i < 0 && j >= 0) {
      if (threadIdx.x == 0) path[j] = -1 - y;
      j--;
      y = a.parent[y];
      i = y >= 0 ? a.tidx_of[y] : 0;
    }
    if (j >= 0) {  // ancestors in the trunk: a run of trunk indices per piece
      const int pc = a.piece_of[i], c0 = a.chain_off[pc], c1 = a.chain_off[pc + 1];
      for (int c = c0 + warp; c < c1; c += BW) {
        const int2 run = a.chain[c];
        const int end = c + 1 < c1 ? a.chain[c + 1].y : j + 1;
        if (run.y + lane < end) path[run.y + lane] = run.x + lane;
      }
    }
  }
  __syncthreads();
  // the entries of the block's ancestors [q0, q0 + 32) from ancestor `from` on, at most kBackHits;
  // returns the ancestor to go on from (32: all done)
  auto collect = [&](int w, int q0, int from) {
    const int cnt = min(32, h - q0);
    int4 m = make_int4(0, 0, 0, 0);
    bool need = false;  // U(y) is a shortest distance: an ancestor whose row is longer has no seed
    if (lane >= from && lane < cnt) {
      need = ub[q0 + lane] != 0.0 || q0 + lane == h - 1;
      const int p = path[q0 + lane];
      if (need) m = p >= 0 ? a.tmeta[p] : make_int4(a.xoff[-1 - p], a.xoff[-p], 0, 0);
    }
    unsigned todo = __ballot_sync(kAll, need);
    int nh = 0, done = 32;
    int4 v[4];
    auto load = [&](int eb, int e1) {
#pragma unroll
      for (int r = 0; r < 4; r++) v[r] = eb + r * 32 + lane < e1 ? __ldg(a.eup + eb + r * 32 + lane) : make_int4(-1, 0, 0, 0);
    };
    int k = __ffs(todo) - 1, e0 = __shfl_sync(kAll, m.x, max(k, 0)), e1 = __shfl_sync(kAll, m.y, max(k, 0));
    if (todo) load(e0, e1);
    while (todo) {
      const int mark = nh, yq = q0 + k;
      const int d = ud[yq];
      bool full = false;
      int eb = e0;
      do {  // (once for the root, which has none: the next ancestor's entries are loaded here)
        int4 c[4];
#pragma unroll
        for (int r = 0; r < 4; r++) c[r] = v[r];
        if (eb + 128 < e1) load(eb + 128, e1);
        else {  // the next ancestor's first entries
          const unsigned rest = todo & (todo - 1);
          if (rest) {
            const int kn = __ffs(rest) - 1;
            load(__shfl_sync(kAll, m.x, kn), __shfl_sync(kAll, m.y, kn));
          }
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const bool is = c[r].x >= 0 && d + c[r].y == ud[max(c[r].x, 0)];
          const unsigned b = __ballot_sync(kAll, is);
          if (!b) continue;
          const int pos = nh + __popc(b & ((1u << lane) - 1u));
          if (is && pos < kBackHits) {
            sh.hit[w][pos] = make_int2(eb + r * 32 + lane, (int)((unsigned)c[r].x | ((unsigned)yq << 16)));
            sh.ratio[w][pos] = share(c[r].z, uc[yq], uc[c[r].x]);
          }
          nh += __popc(b);
          full |= nh > kBackHits;
        }
        eb += 128;
      } while (eb < e1);
      if (full) {  // this ancestor again in the next turn (alone if it has to be)
        nh = mark;
        done = k;
        break;
      }
      todo &= todo - 1;
      if (todo) {
        k = __ffs(todo) - 1;
        e0 = __shfl_sync(kAll, m.x, k);
        e1 = __shfl_sync(kAll, m.y, k);
      }
    }
    if (lane == 0) sh.count[w] = nh;
    return done;
  };
  auto apply = [&](int w) {  // one lane: an ancestor's flow depends on those before it
    if (lane == 0)
      for (int q = 0; q < sh.count[w]; q++) {
        const int y = sh.hit[w][q].y;
        ub[(unsigned)y >> 16] += sh.ratio[w][q] * ub[y & 0xffff];
      }
    __syncwarp();
  };
  auto add = [&](int w, int first, int step) {
    for (int q = first; q < sh.count[w]; q += step) {
      const int2 t = sh.hit[w][q];
      const double f = sh.ratio[w][q] * ub[t.y & 0xffff];
      if (f != 0.0) atomicAdd(((int)((unsigned)t.y >> 16) == h - 1 ? a.Bs : a.Bu) + t.x, f);
    }
  };
  for (int r0 = 0; r0 < h; r0 += BW * 32) {
    const int q0 = r0 + warp * 32;
    int done = 32;
    if (q0 < h) done = collect(warp, q0, 0);
    else if (lane == 0) sh.count[warp] = 0;
    const bool crowded = __syncthreads_or(done < 32);
    if (!crowded) {
      if (warp == 0)
        for (int w = 0; w < BW; w++) apply(w);
      __syncthreads();
      add(warp, lane, 32);
    } else if (warp == 0) {  // more entries than the lists hold: one warp, list by list
      for (int w = 0; w < BW; w++)
        for (int from = 0; r0 + w * 32 < h && from < 32;) {
          __syncwarp();
          int next = collect(0, r0 + w * 32, from);
          __syncwarp();
          if (next == from && sh.count[0] == 0) {  // one ancestor with more entries than a list: entry by entry
            const int p = path[r0 + w * 32 + from], yq = r0 + w * 32 + from;
            const int4 m = p >= 0 ? a.tmeta[p] : make_int4(a.xoff[-1 - p], a.xoff[-p], 0, 0);
            double up = 0.0;
            for (int e = m.x + lane; e < m.y; e += 32) {
              const int4 v = a.eup[e];
              if (ud[yq] + v.y != ud[v.x]) continue;
              const double f = share(v.z, uc[yq], uc[v.x]) * ub[v.x];
              up += f;
              if (f != 0.0) atomicAdd((yq == h - 1 ? a.Bs : a.Bu) + e, f);
            }
            up = warp_sum(up);
            if (lane == 0) ub[yq] += up;
            __syncwarp();
            next = from + 1;
          } else {
            apply(0);
            add(0, lane, 32);
          }
          from = next;
        }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------- shared pieces
// key of U_s(t) for a lane whose source lies in t's subtree (index 0), else none
__device__ __forceinline__ unsigned up_key(const TreeArgs &a, bool in, size_t uidx) {
  if (!in) return kNoKey;
  const unsigned u = (unsigned)a.Ud[uidx];
  return u < a.dist_lim ? u << a.bits : kNoKey;
}

// Bd(e) += sum over lanes and values of the flows whose entry is e (entry idx > 0 of the vertex whose
// edges start at e0; 0: none), one entry of the warp after another.
template <int K>
__device__ __forceinline__ void add_flows(const TreeArgs &a, int e0, int (&idx)[K], const double (&flow)[K]) {
  const int lane = threadIdx.x & 31;
  for (;;) {
    int mine = 0;
#pragma unroll
    for (int k = 0; k < K; k++) mine = mine ? mine : idx[k];
    const unsigned any = __ballot_sync(kAll, mine != 0);
    if (!any) return;
    const int xl = __shfl_sync(kAll, mine, __ffs(any) - 1);
    double z = 0.0;
#pragma unroll
    for (int k = 0; k < K; k++)
      if (idx[k] == xl) {
        z += flow[k];
        idx[k] = 0;
      }
    z = warp_sum(z);
    if (lane == 0) atomicAdd(a.Bd + e0 + xl - 1, z);
  }
}

// ------------------------------------------------------------------------------- trunk, wide levels
// A CTA takes one piece (a path of at most PL trunk vertices) for one group of sources.  The minima
// over the separator vertices above the piece are independent, a warp per vertex; then one warp
// follows the path over the edges inside the piece in shared memory, while other CTAs fill the SM:
// levels with many pieces are bound by instructions and occupancy, not by the latency of the path.
// Pieces of up to 8 and 16 vertices, most of those below the top, have launches of their own with
// less shared memory and fewer warps to wait for the one on the path.
template <int PL>
struct Wide {
  static constexpr int warps = PL == 8 ? 2 : 4;
};

template <int PL>
struct PieceShared {
  int2 ine[PL * (PL - 1) / 2];  // edges inside the piece: (kGroup * position, key)
  int ineC[PL * (PL - 1) / 2];
  int inoff[PL + 1];
  int4 meta[PL];
  int2 sub[PL];
};

template <int PL>
__device__ __forceinline__ void load_piece(const TreeArgs &a, int start, int len, PieceShared<PL> &p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) {
    const int4 m = lane < len ? a.tmeta[start + lane] : make_int4(0, 0, 0, 0);
    if (lane < len) {
      p.meta[lane] = m;
      p.sub[lane] = a.tsub[start + lane];
    }
    int x = m.z;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int z = __shfl_up_sync(kAll, x, o);
      if (lane >= o) x += z;
    }
    if (lane <= len && lane < PL) p.inoff[lane] = x - m.z;
    if (lane == len - 1) p.inoff[len] = x;
  }
  __syncthreads();
  for (int i = warp; i < len; i += Wide<PL>::warps) {
    const int4 m = p.meta[i];
    if (lane < m.z) {  // at most 31 edges
      const int2 v = a.ex[m.y - m.z + lane];
      p.ine[p.inoff[i] + lane] = make_int2((v.x - start) * kGroup, v.y);
      p.ineC[p.inoff[i] + lane] = a.eC[m.y - m.z + lane];
    }
  }
}

// Minimum keys of a vertex over its entries [e, ee) above the piece, eight or four loaded together.
__device__ __forceinline__ void scan_above(const TreeArgs &a, int e, int ee, size_t gt, unsigned mask, unsigned (&m1)[2],
                                           unsigned (&m2)[2]) {
  if (e >= ee) return;
  const uint32_t *D = a.D + gt;
  int2 w[8];  // the next entries, in flight while the current distances are loaded
#pragma unroll
  for (int q = 0; q < 8; q++) w[q] = __ldg(a.ex + min(e + q, ee - 1));
  auto step = [&](auto count) {  // (the last entry may repeat)
    constexpr int N = decltype(count)::value;
    uint2 d[N];
    unsigned key[N];
#pragma unroll
    for (int q = 0; q < N; q++) {
      d[q] = *reinterpret_cast<const uint2 *>(D + (size_t)w[q].x * kGroup);
      key[q] = (unsigned)w[q].y;
    }
    e += N;
    if (e < ee) {
#pragma unroll
      for (int q = 0; q < N; q++) w[q] = __ldg(a.ex + min(e + q, ee - 1));
    }
#pragma unroll
    for (int q = 0; q < N; q += 2) {
      key_min2(m1[0], m2[0], d[q].x + key[q], d[q + 1].x + key[q + 1], mask);
      key_min2(m1[1], m2[1], d[q].y + key[q], d[q + 1].y + key[q + 1], mask);
    }
  };
  while (e + 4 < ee) step(std::integral_constant<int, 8>{});
  if (e < ee) step(std::integral_constant<int, 4>{});
}

// Counts of a minimum over the entries above the piece (first edge e0, nx of them), its argument
// being smallest | largest << 16; hits: how many entries reach it.
__device__ __forceinline__ void count_above(const TreeArgs &a, int e0, int nx, size_t gt, size_t gu, unsigned mask,
                                            const unsigned (&md)[2], const unsigned (&ar)[2], uint32_t (&cnt)[2],
                                            unsigned (&hits)[2], unsigned &over) {
  int lo = INT_MAX, hi = 0;
  bool tie = false;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int a1 = (int)(ar[k] & 0xffff), a2 = (int)(ar[k] >> 16);
    hits[k] = a1 <= nx;  // (none: no entry above the piece)
    const int e = e0 + a1 - 1;
    unsigned long long c = 0;
    if (a1 == 0) c = a.Uc[gu + k];
    else if (a1 <= nx) c = (unsigned long long)(unsigned)a.eC[e] * a.S[gt + (size_t)a.ex[e].x * kGroup + k];
    over |= c > 0x7fffffffull;
    cnt[k] = (uint32_t)c;
    if (a1 != a2 && a1 <= nx) {
      tie = true;
      lo = min(lo, a1 + 1);
      hi = max(hi, min(a2, nx));
    }
  }
  if (!__any_sync(kAll, tie)) return;
  // several entries: those after the first, up to the last that any lane has
  lo = __reduce_min_sync(kAll, lo);
  hi = __reduce_max_sync(kAll, hi);
  for (int q0 = lo; q0 <= hi; q0 += 8) {
    int2 w[8];
    uint2 d[8];
#pragma unroll
    for (int q = 0; q < 8; q++) w[q] = __ldg(a.ex + e0 + min(q0 + q, hi) - 1);
#pragma unroll
    for (int q = 0; q < 8; q++) d[q] = *reinterpret_cast<const uint2 *>(a.D + gt + (size_t)w[q].x * kGroup);
#pragma unroll
    for (int q = 0; q < 8; q++)
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int a1 = (int)(ar[k] & 0xffff), a2 = (int)(ar[k] >> 16);
        if (q0 + q <= hi && a1 < q0 + q && q0 + q <= a2 && (k ? d[q].y : d[q].x) + ((unsigned)w[q].y & ~mask) == md[k]) {
          const unsigned long long c =
              cnt[k] + (unsigned long long)(unsigned)a.eC[e0 + q0 + q - 1] * a.S[gt + (size_t)w[q].x * kGroup + k];
          over |= c > 0x7fffffffull;
          cnt[k] = (uint32_t)c;
          hits[k]++;
        }
      }
  }
}

template <int PL>
__global__ void __launch_bounds__(Wide<PL>::warps * 32) k_trunk_down(TreeArgs a, int piece0) {
  constexpr int NW = Wide<PL>::warps;
  __shared__ PieceShared<PL> p;
  // per vertex and source: distance and argument (before its turn on the path: the two keys of the
  // minimum above the piece), count (sign bit before its turn: more than two entries reach it)
  __shared__ uint2 sd[PL * 32], sa[PL * 32], sc[PL * 32];
  if (__syncthreads_or(wrapped(a))) return;
  const int4 pc = a.piece[piece0 + blockIdx.x];
  const int start = pc.x, len = pc.y - pc.x, g = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned mask = (1u << a.bits) - 1u;
  uint2 *rd = sd + lane, *ra = sa + lane, *rc = sc + lane;
  int s[2];
  bool live[2];
  lane_sources(a, g, lane, s, live);
  const size_t gt = (size_t)g * a.NT * kGroup + 2 * lane, gu = (size_t)g * a.H * kGroup + 2 * lane;
  load_piece<PL>(a, start, len, p);
  __syncthreads();
  unsigned over = 0;
  for (int i = warp; i < len; i += NW) {
    const int4 m = p.meta[i];
    const int2 sub = p.sub[i];
    const size_t u = gu + (size_t)sub.y * kGroup;
    unsigned m1[2], m2[2], md[2], ar[2], hits[2];
    uint32_t cnt[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      m1[k] = up_key(a, m.w <= s[k] && s[k] < sub.x, u + k);
      m2[k] = m1[k] == kNoKey ? kNoKey : m1[k] ^ mask;
    }
    scan_above(a, m.x, m.y - m.z, gt, mask, m1, m2);
#pragma unroll
    for (int k = 0; k < 2; k++) {
      md[k] = m1[k] & ~mask;
      ar[k] = (m1[k] & mask) | (((m2[k] & mask) ^ mask) << 16);
    }
    count_above(a, m.x, m.y - m.z - m.x, gt, u, mask, md, ar, cnt, hits, over);
    rd[i * 32] = make_uint2(m1[0], m1[1]);
    ra[i * 32] = make_uint2(m2[0], m2[1]);
    rc[i * 32] = make_uint2(cnt[0] | (hits[0] > 2 ? 0x80000000u : 0u), cnt[1] | (hits[1] > 2 ? 0x80000000u : 0u));
  }
  __syncthreads();
  if (warp == 0) {  // along the piece: entries inside it, in order
    for (int i = 0; i < len; i++) {
      const uint2 e1 = rd[i * 32], e2 = ra[i * 32], ec = rc[i * 32];
      const unsigned x1[2] = {e1.x, e1.y}, x2[2] = {e2.x, e2.y};  // above the piece
      unsigned m1[2] = {e1.x, e1.y}, m2[2] = {e2.x, e2.y};
      const int b = p.inoff[i], e = p.inoff[i + 1];
#pragma unroll 4
      for (int q = b; q < e; q++) {
        const int2 v = p.ine[q];
        const uint2 d = rd[v.x >> 1];
        const unsigned w0 = d.x + (unsigned)v.y, w1 = d.y + (unsigned)v.y;
        m1[0] = min(m1[0], w0);
        m2[0] = min(m2[0], w0 ^ mask);
        m1[1] = min(m1[1], w1);
        m2[1] = min(m2[1], w1 ^ mask);
      }
      const int4 m = p.meta[i];
      const int nx = m.y - m.z - m.x;
      unsigned ar[2];
      uint32_t cnt[2] = {ec.x & 0x7fffffffu, ec.y & 0x7fffffffu};
      bool tie = false;
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int a1 = (int)(m1[k] & mask);
        ar[k] = (unsigned)a1 | ((unsigned)a1 << 16);
        tie |= (m1[k] ^ m2[k]) != mask;
        if (a1 > nx) {
          const int q = b + a1 - 1 - nx;
          const uint2 c = rc[p.ine[q].x >> 1];
          const unsigned long long z = (unsigned long long)(unsigned)p.ineC[q] * (k ? c.y : c.x);
          over |= z > 0x7fffffffull;
          cnt[k] = (uint32_t)z;
        }
      }
      if (__any_sync(kAll, tie)) {  // several entries: their counts summed
#pragma unroll
        for (int k = 0; k < 2; k++) {
          if ((m1[k] ^ m2[k]) == mask) continue;
          const unsigned dt = m1[k] & ~mask;
          const uint32_t c0 = (k ? ec.y : ec.x);
          int hits = 0;
          unsigned long long z = 0;
          if ((x1[k] & ~mask) == dt) {  // some above the piece
            hits = (x1[k] ^ x2[k]) == mask ? 1 : c0 >> 31 ? 3 : 2;
            z = c0 & 0x7fffffffu;
          }
          for (int q = b; q < e; q++) {
            const int2 v = p.ine[q];
            const uint2 d = rd[v.x >> 1];
            if ((k ? d.y : d.x) + ((unsigned)v.y & ~mask) != dt) continue;
            const uint2 c = rc[v.x >> 1];
            z += (unsigned long long)(unsigned)p.ineC[q] * (k ? c.y : c.x);
            if (z > 0x7fffffffull) {
              over = 1;
              z = 1;
            }
            hits++;
          }
          cnt[k] = (uint32_t)z;
          const unsigned lo = m1[k] & mask, hi = (m2[k] & mask) ^ mask;
          ar[k] = hits > 2 ? hi | (lo << 16) : lo | (hi << 16);
        }
      }
      rd[i * 32] = make_uint2(m1[0] & ~mask, m1[1] & ~mask);
      ra[i * 32] = make_uint2(ar[0], ar[1]);
      rc[i * 32] = make_uint2(cnt[0], cnt[1]);
    }
  }
  if (over) *a.wrap = 1;
  __syncthreads();
  for (int i = warp; i < len; i += NW) {
    const size_t o = gt + (size_t)(start + i) * kGroup;
    *reinterpret_cast<uint2 *>(a.D + o) = rd[i * 32];
    *reinterpret_cast<uint2 *>(a.S + o) = rc[i * 32];
    *reinterpret_cast<uint2 *>(a.arg + o) = ra[i * 32];
    *reinterpret_cast<double2 *>(a.J + o) = make_double2(0.0, 0.0);
  }
}

// What a trunk vertex does with its flow beyond its piece: the seed of its U row, flow to the entries
// above the piece, and the flow through each of its shortcuts.  one: its argument where it is the
// only one, xi that entry's trunk index.
__device__ __forceinline__ void hand_up(const TreeArgs &a, const int4 m, const int2 sub, size_t gt, size_t gu, unsigned mask,
                                        const int (&s)[2], const int (&si)[2], const bool (&live)[2], const double (&f)[2],
                                        const unsigned (&ar)[2], int (&one)[2], const int (&xi)[2], size_t own) {
  const int nx = m.y - m.z - m.x;
  bool tie = false;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int a1 = (int)(ar[k] & 0xffff), a2 = (int)(ar[k] >> 16);
    tie |= a1 != a2;
    if (live[k] && m.w <= s[k] && s[k] < sub.x) {
      const size_t u = gu + (size_t)sub.y * kGroup + k;
      a.seed[u] = min(a1, a2) != 0 ? 0.0 : a1 == a2 ? f[k] : f[k] * share(1, a.Uc[u], a.S[own + k]);
    }
    if (one[k] > 0 && one[k] <= nx) atomicAdd(a.J + gt + (size_t)xi[k] * kGroup + k, f[k]);
    if (xi[k] == si[k]) {  // flow into the lane's own source counts apart
      atomicAdd(a.Bs + m.x + one[k] - 1, f[k]);
      one[k] = 0;
    }
  }
  add_flows<2>(a, m.x, one, f);
  if (!__any_sync(kAll, tie)) return;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int a1 = (int)(ar[k] & 0xffff), a2 = (int)(ar[k] >> 16);
    if (a1 == a2) continue;
    const uint32_t st = a.S[own + k];
    auto use = [&](int idx) {
      const int e = m.x + idx - 1, x = a.ex[e].x;
      const double w = f[k] * share(a.eC[e], a.S[gt + (size_t)x * kGroup + k], st);
      if (idx <= nx) atomicAdd(a.J + gt + (size_t)x * kGroup + k, w);
      atomicAdd((x == si[k] ? a.Bs : a.Bd) + e, w);
    };
    if (a1 < a2) {
      if (a1 > 0) use(a1);
      use(a2);
    } else {  // more than two entries
      const unsigned dt = a.D[own + k];
      for (int e = m.x; e < m.y; e++) {
        const int2 x = a.ex[e];
        if (a.D[gt + (size_t)x.x * kGroup + k] + ((unsigned)x.y & ~mask) == dt) use(e - m.x + 1);
      }
    }
  }
}

template <int PL>
__global__ void __launch_bounds__(Wide<PL>::warps * 32) k_trunk_up(TreeArgs a, int piece0) {
  constexpr int NW = Wide<PL>::warps;
  __shared__ PieceShared<PL> p;
  __shared__ double2 sf[PL * 32];
  __shared__ uint2 sa[PL * 32], ss[PL * 32];
  if (__syncthreads_or(wrapped(a))) return;
  const int4 pc = a.piece[piece0 + blockIdx.x];
  const int start = pc.x, len = pc.y - pc.x, g = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned mask = (1u << a.bits) - 1u;
  double *rf = &sf[lane].x;  // flow of a vertex: delta + 1 (delta for the source itself)
  uint32_t *ra = &sa[lane].x, *rs = &ss[lane].x;
  int s[2], si[2];
  bool live[2];
  lane_sources(a, g, lane, s, live);
#pragma unroll
  for (int k = 0; k < 2; k++) si[k] = a.tidx_of[s[k]];
  const size_t gt = (size_t)g * a.NT * kGroup + 2 * lane, gu = (size_t)g * a.H * kGroup + 2 * lane;
  load_piece<PL>(a, start, len, p);
  __syncthreads();
  for (int i = warp; i < len; i += NW) {
    const int t = p.meta[i].w;
    const size_t o = gt + (size_t)(start + i) * kGroup;
    const double2 j = __ldcg(reinterpret_cast<const double2 *>(a.J + o));
    const uint2 x = *reinterpret_cast<const uint2 *>(a.arg + o), y = *reinterpret_cast<const uint2 *>(a.S + o);
    // a lane without a source has no flow and no argument
    *reinterpret_cast<double2 *>(rf + i * kGroup) =
        make_double2(live[0] ? j.x + (t != s[0] ? 1.0 : 0.0) : 0.0, live[1] ? j.y + (t != s[1] ? 1.0 : 0.0) : 0.0);
    *reinterpret_cast<uint2 *>(ra + i * kGroup) = make_uint2(live[0] ? x.x : 0u, live[1] ? x.y : 0u);
    *reinterpret_cast<uint2 *>(rs + i * kGroup) = y;
  }
  __syncthreads();
  if (warp == 0) {  // what is handed on inside the piece, deepest vertex first
    for (int i = len - 1; i > 0; i--) {
      const int4 m = p.meta[i];
      if (m.z == 0) continue;
      const int nx = m.y - m.z - m.x, in0 = p.inoff[i] - 1 - nx;
      const uint2 ar = *reinterpret_cast<const uint2 *>(ra + i * kGroup);
      const double2 f2 = *reinterpret_cast<const double2 *>(rf + i * kGroup);
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int a1 = (int)((k ? ar.y : ar.x) & 0xffff), a2 = (int)((k ? ar.y : ar.x) >> 16);
        const double f = k ? f2.y : f2.x;
        if (max(a1, a2) <= nx) continue;
        if (a1 == a2) {
          rf[p.ine[in0 + a1].x + k] += f;
        } else if (a1 < a2) {
          const uint32_t st = rs[i * kGroup + k];
          const int x2 = p.ine[in0 + a2].x + k;
          if (a1 > nx) {
            const int x1 = p.ine[in0 + a1].x + k;
            rf[x1] += share(p.ineC[in0 + a1], rs[x1], st) * f;
          }
          rf[x2] += share(p.ineC[in0 + a2], rs[x2], st) * f;
        } else {  // more than two entries
          const size_t gp = gt + (size_t)start * kGroup + k;
          const unsigned dt = a.D[gp + (size_t)i * kGroup];
          for (int q = p.inoff[i]; q < p.inoff[i + 1]; q++) {
            const int x = p.ine[q].x;
            if (a.D[gp + x] + ((unsigned)p.ine[q].y & ~mask) == dt)
              rf[x + k] += share(p.ineC[q], rs[x + k], rs[i * kGroup + k]) * f;
          }
        }
      }
    }
  }
  __syncthreads();
  for (int i = warp; i < len; i += NW) {  // everything else, a warp per vertex
    const int4 m = p.meta[i];
    const uint2 x = *reinterpret_cast<const uint2 *>(ra + i * kGroup);
    const double2 f2 = *reinterpret_cast<const double2 *>(rf + i * kGroup);
    const unsigned ar[2] = {x.x, x.y};
    const double f[2] = {f2.x, f2.y};
    int one[2], xi[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      one[k] = (ar[k] & 0xffff) == (ar[k] >> 16) ? (int)(ar[k] & 0xffff) : 0;
      xi[k] = one[k] > 0 ? a.ex[m.x + one[k] - 1].x : INT_MIN;
    }
    hand_up(a, m, p.sub[i], gt, gu, mask, s, si, live, f, ar, one, xi, gt + (size_t)(start + i) * kGroup);
  }
}

// ------------------------------------------------------------------------------- trunk, narrow levels
// Levels with few pieces wait for the longest one, so a CTA of 32 warps takes a piece, a warp per
// vertex.  The path is followed vertex by vertex: a vertex's warp publishes its distances and counts,
// and the warps of the vertices below offer them to their running minimum, arguments and count in
// registers.  (One warp walking the path alone takes 23k cycles for the distances and 16k for the
// counts of a full piece.)  256 sources of 50k vertices are 18 levels of 28 us each way, bound by that
// chain (issue 5 %, DRAM below 1 %); 16 or 32 distances of a scan in flight instead of 8 changed nothing
// (1.29, 1.33 and 1.30 ms).  A level starts while the one before it runs (let_next): 1.41 -> 1.34 ms.
struct PieceTable {
  unsigned win[kPieceLen][kPieceLen + 1];  // key of the edge (vertex, earlier vertex), or absent
  int cin[kPieceLen][kPieceLen + 1];       // its count
};

__device__ __forceinline__ void load_table(const TreeArgs &a, int start, int len, PieceTable &p) {
  const int i = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (i >= len) return;
  const int4 m = a.tmeta[start + i];
  p.win[i][lane] = a.absent;
  __syncwarp();
  if (lane < m.z) {  // at most 31 edges inside the piece
    const int2 v = a.ex[m.y - m.z + lane];
    p.win[i][v.x - start] = (unsigned)v.y;
    p.cin[i][v.x - start] = a.eC[m.y - m.z + lane];
  }
}

__global__ void __launch_bounds__(kPieceLen * 32) k_trunk_down_narrow(TreeArgs a, int piece0) {
  __shared__ PieceTable p;
  __shared__ uint2 row_d[2][32], row_c[2][32];
  let_next();
  const int4 pc = a.piece[piece0 + blockIdx.x];
  const int start = pc.x, len = pc.y - pc.x, g = blockIdx.y;
  const int i = threadIdx.x >> 5, lane = threadIdx.x & 31;  // this warp's vertex
  const unsigned mask = (1u << a.bits) - 1u;
  const size_t gt = (size_t)g * a.NT * kGroup + 2 * lane;
  load_table(a, start, len, p);
  unsigned md[2] = {}, ar[2] = {}, hits[2] = {}, over = 0;
  uint32_t cnt[2] = {};
  int s[2];
  bool live[2];
  lane_sources(a, g, lane, s, live);
  const int4 m = a.tmeta[start + min(i, len - 1)];
  const int2 sub = a.tsub[start + min(i, len - 1)];
  wait_before();
  if (__syncthreads_or(wrapped(a))) return;
  if (i < len) {
    const size_t u = ((size_t)g * a.H + sub.y) * kGroup + 2 * lane;
    unsigned m1[2], m2[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      m1[k] = up_key(a, m.w <= s[k] && s[k] < sub.x, u + k);
      m2[k] = m1[k] == kNoKey ? kNoKey : m1[k] ^ mask;
    }
    scan_above(a, m.x, m.y - m.z, gt, mask, m1, m2);
#pragma unroll
    for (int k = 0; k < 2; k++) {
      md[k] = m1[k] & ~mask;
      ar[k] = (m1[k] & mask) | (((m2[k] & mask) ^ mask) << 16);
    }
    count_above(a, m.x, m.y - m.z - m.x, gt, u, mask, md, ar, cnt, hits, over);
  }
  for (int t = 0; t < len; t++) {
    if (t == i) {
      row_d[t & 1][lane] = make_uint2(md[0], md[1]);
      row_c[t & 1][lane] = make_uint2(cnt[0], cnt[1]);
    }
    __syncthreads();  // (also the tables, the first time)
    if (t >= i || i >= len) continue;
    const unsigned key = p.win[i][t];
    if (key == a.absent) continue;
    const uint2 d2 = row_d[t & 1][lane], c2 = row_c[t & 1][lane];
    const unsigned idx = key & mask;
    const int C = p.cin[i][t];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const unsigned d = (k ? d2.y : d2.x) + (key & ~mask);
      if (d > md[k]) continue;
      if (d < md[k]) {
        md[k] = d;
        ar[k] = idx;
        hits[k] = 0;
        cnt[k] = 0;
      }
      const unsigned long long c = (unsigned long long)(unsigned)C * (k ? c2.y : c2.x) + cnt[k];
      over |= c > 0x7fffffffull;
      cnt[k] = (uint32_t)c;
      ar[k] = (ar[k] & 0xffff) | (idx << 16);
      hits[k]++;
    }
  }
  if (over) *a.wrap = 1;
  if (i >= len) return;
#pragma unroll
  for (int k = 0; k < 2; k++)
    if (hits[k] > 2) ar[k] = (ar[k] >> 16) | (ar[k] << 16);
  const size_t o = gt + (size_t)(start + i) * kGroup;
  *reinterpret_cast<uint2 *>(a.D + o) = make_uint2(md[0], md[1]);
  *reinterpret_cast<uint2 *>(a.S + o) = make_uint2(cnt[0], cnt[1]);
  *reinterpret_cast<uint2 *>(a.arg + o) = make_uint2(ar[0], ar[1]);
  *reinterpret_cast<double2 *>(a.J + o) = make_double2(0.0, 0.0);
}

// The same, deepest vertex first: a vertex's warp publishes its flow and arguments, and the warps of
// the vertices above take their share of it.
__global__ void __launch_bounds__(kPieceLen * 32) k_trunk_up_narrow(TreeArgs a, int piece0) {
  __shared__ PieceTable p;
  __shared__ double2 row_f[2][32];
  __shared__ uint2 row_a[2][32], row_s[2][32], row_d[2][32];
  let_next();
  const int4 pc = a.piece[piece0 + blockIdx.x];
  const int start = pc.x, len = pc.y - pc.x, g = blockIdx.y;
  const int i = threadIdx.x >> 5, lane = threadIdx.x & 31;  // this warp's vertex
  const unsigned mask = (1u << a.bits) - 1u;
  const size_t gt = (size_t)g * a.NT * kGroup + 2 * lane, gu = (size_t)g * a.H * kGroup + 2 * lane;
  const size_t own = gt + (size_t)(start + i) * kGroup;
  int4 m = make_int4(0, 0, 0, 0);
  int s[2], si[2], one[2], xi[2];
  bool live[2];
  double f[2] = {};
  unsigned ar[2] = {};
  uint2 st = make_uint2(0, 0), dt = st;
  lane_sources(a, g, lane, s, live);
  if (i < len) {  // (all but the flow is the way down's)
    const uint2 x = *reinterpret_cast<const uint2 *>(a.arg + own);
    st = *reinterpret_cast<const uint2 *>(a.S + own);
    dt = *reinterpret_cast<const uint2 *>(a.D + own);
    m = a.tmeta[start + i];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      si[k] = a.tidx_of[s[k]];
      if (!live[k]) continue;  // a lane without a source has no flow and no argument
      ar[k] = k ? x.y : x.x;
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
      one[k] = (ar[k] & 0xffff) == (ar[k] >> 16) ? (int)(ar[k] & 0xffff) : 0;
      xi[k] = one[k] > 0 ? a.ex[m.x + one[k] - 1].x : INT_MIN;
    }
  }
  load_table(a, start, len, p);
  wait_before();
  if (__syncthreads_or(wrapped(a))) return;
  if (i < len) {
    const double2 j = __ldcg(reinterpret_cast<const double2 *>(a.J + own));
#pragma unroll
    for (int k = 0; k < 2; k++)
      if (live[k]) f[k] = (k ? j.y : j.x) + (m.w != s[k] ? 1.0 : 0.0);
  }
  for (int t = len - 1; t > 0; t--) {
    if (t == i) {
      row_f[t & 1][lane] = make_double2(f[0], f[1]);
      row_a[t & 1][lane] = make_uint2(ar[0], ar[1]);
      row_s[t & 1][lane] = st;
      row_d[t & 1][lane] = dt;
    }
    __syncthreads();  // (also the tables, the first time)
    if (i >= t) continue;
    const unsigned key = p.win[t][i];
    if (key == a.absent) continue;
    const uint2 a2 = row_a[t & 1][lane];
    const double2 f2 = row_f[t & 1][lane];
    const unsigned idx = key & mask;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const unsigned x1 = (k ? a2.y : a2.x) & 0xffff, x2 = (k ? a2.y : a2.x) >> 16;
      if (x1 == x2) {
        if (x1 == idx) f[k] += k ? f2.y : f2.x;
      } else if (x1 > x2 || x1 == idx || x2 == idx) {
        const uint2 s2 = row_s[t & 1][lane], d2 = row_d[t & 1][lane];
        if (x1 < x2 || (k ? dt.y : dt.x) + (key & ~mask) == (k ? d2.y : d2.x))
          f[k] += (k ? f2.y : f2.x) * share(p.cin[t][i], k ? st.y : st.x, k ? s2.y : s2.x);
      }
    }
  }
  if (i < len) hand_up(a, m, a.tsub[start + i], gt, gu, mask, s, si, live, f, ar, one, xi, own);
}

// ------------------------------------------------------------------------------- bottoms
// A whole subtree below the trunk for a group at a time in a warp's shared memory: rows 0..b-1 are
// the root's separator (trunk vertices), then the subtree's vertices with descendants in preorder.
// Down then up, so nothing of the subtree is written to global memory.  Distances are kept shifted (a
// key without its index), and an entry's index in the keys is its row + 1 (0: U), so the row a lane's
// paths come from needs no lookup.  A vertex without descendants (44 % of them) has no row: nobody
// reads it and its flow is 1 per source, so it is done on the way down, and where all lanes hand
// everything to one entry, as most do, only that entry's row and a counter change.  On the way up
// most vertices, too, hand everything to one entry in all lanes (at 50k 1.1 to 1.3 different entries
// per vertex and warp): that entry's flow stays in the finished row and is summed after the pass,
// eight rows at a time, instead of by a warp-wide sum per vertex.
//
// The pass is bound by instruction issue and by the warps that shared memory leaves room for (50k: issue
// 32 to 38 % with 9 to 15 warps per SM, DRAM 5 to 11 %; a third of the time of all sources), so
// shared memory is addressed by 32-bit offsets (ld.shared / st.shared); a row's block holds delta
// (f64), distance, count and argument of the warp's sources.
constexpr int kTieCode = 0xff, kSkipCode = 0xfe;  // arguments that are no row: a tie, a lane without a source
constexpr int kBottomPairs = (kBottomEdges + kBottomVerts) / 2 + 1;
constexpr int kBottomWarps = 2;
constexpr int kLeadFull = 1 << 16;  // deferred sum: every lane, the rows' delta + 1 each
constexpr int kManyCounts = INT_MIN, kLeaf = 1 << 30, kDepthBits = kLeaf - 1;  // in a vertex's fourth word
constexpr int kAhead = 8;           // separator rows of the next group loaded during the way up

struct RowLayout {  // bytes
  static constexpr int D = 512, S = 768, G = 1024, lead = 1088, size = 1104;
};

__device__ __forceinline__ int4 lds128(uint32_t p) {
  int4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(p));
  return v;
}
__device__ __forceinline__ int lds32(uint32_t p) {
  int v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(p));
  return v;
}
__device__ __forceinline__ double lds64(uint32_t p) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(p));
  return v;
}
__device__ __forceinline__ void sts32(uint32_t p, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(p), "r"(v) : "memory"); }
__device__ __forceinline__ void sts64(uint32_t p, double v) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(p), "d"(v) : "memory"); }

// a lane's two neighbouring values in one access
__device__ __forceinline__ void row_load(uint32_t p, uint32_t (&v)[2]) {
  asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(p));
}
__device__ __forceinline__ void row_store(uint32_t p, const uint32_t (&v)[2]) {
  asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(p), "r"(v[0]), "r"(v[1]) : "memory");
}
__device__ __forceinline__ void row_load(uint32_t p, double (&v)[2]) {
  asm volatile("ld.shared.v2.f64 {%0,%1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(p));
}
__device__ __forceinline__ void row_store(uint32_t p, const double (&v)[2]) {
  asm volatile("st.shared.v2.f64 [%0], {%1,%2};" ::"r"(p), "d"(v[0]), "d"(v[1]) : "memory");
}
// the arguments of a lane's sources, a byte each
__device__ __forceinline__ unsigned code_load(uint32_t p) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(p));
  return v;
}
__device__ __forceinline__ void code_store(uint32_t p, unsigned v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(p), "h"((unsigned short)v) : "memory");
}

__global__ void __launch_bounds__(kBottomWarps * 32) k_bottom(TreeArgs a, int first, int rows, int gpc) {
  extern __shared__ int4 sm_b[];
  using R = RowLayout;
  __shared__ int4 ep[kBottomPairs];      // two edges: (x row offset, key) twice
  __shared__ int4 vt[kBottomVerts + 1];  // a vertex: (address of its first pair, end, first edge | edges << 16, depth - 1 | kLeaf | kManyCounts)
  __shared__ int vs[kBottomVerts], sep[kBottomRows];  // subtree end, trunk index
  __shared__ uint8_t emap[kBottomVerts][kBottomRows];  // edge of (vertex, x row)
  __shared__ uint8_t vertex_of[kBottomRows];           // of a row (less b)
  __shared__ uint8_t leaf_units[kBottomWarps][kBottomEdges];  // groups (at most 64) whose leaf handed everything to the edge
  // Launches of one pass (a few classes of rows) read nothing that another of them writes, so they run
  // into each other; block 0 ends after the launch before, and so do the kernels that follow.
  let_next();
  auto end = [] {
    if (blockIdx.x == 0 && blockIdx.y == 0) wait_before();
  };
  if (__syncthreads_or(wrapped(a))) return end();
  const int4 bt = a.bot[first + blockIdx.x];
  const int r = bt.x, m = bt.y, b = bt.z, nr = bt.w - bt.z;  // nr: vertices with descendants
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int ebase = a.xoff[r];
  const uint32_t ep0 = (uint32_t)__cvta_generic_to_shared(ep), vt0 = (uint32_t)__cvta_generic_to_shared(vt);
  if (warp == 0) {  // two vertices per lane
    int e0[2], k[2], pairs[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int t = 2 * lane + q;
      e0[q] = t < m ? a.xoff[r + t] - ebase : 0;
      k[q] = t < m ? a.xoff[r + t + 1] - ebase - e0[q] : 0;
      pairs[q] = t < m ? max(1, (k[q] + 1) >> 1) : 0;  // (the tree's root has no entries: one absent pair)
    }
    int x = pairs[0] + pairs[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int z = __shfl_up_sync(kAll, x, o);
      if (lane >= o) x += z;
    }
    int pos = (int)ep0 + 16 * (x - pairs[0] - pairs[1]);
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int t = 2 * lane + q;
      if (t < m) {
        vt[t] = make_int4(pos, pos + 16 * pairs[q], e0[q] | (k[q] << 16), a.depth[r + t] - 1);
        vs[t] = a.send[r + t];
        const int row = a.row_of[r + t];
        if (row != 0xff) vertex_of[row - b] = (uint8_t)t;
      }
      pos += 16 * pairs[q];
    }
    if (lane == 0) vt[m] = make_int4((int)ep0, (int)ep0, 0, 0);  // read ahead, not used
  }
  for (int i = threadIdx.x; i < b; i += blockDim.x) sep[i] = a.etr[ebase + i];
  for (int i = threadIdx.x; i < kBottomWarps * kBottomEdges; i += blockDim.x) (&leaf_units[0][0])[i] = 0;
  __syncthreads();
  for (int t = warp; t < m; t += nw) {
    const int4 v = vt[t];
    const int e0 = v.z & 0xffff, k = v.z >> 16;
    bool many = false;
    if (lane < max(2, (k + 1) & ~1)) {
      const int2 x = lane < k ? a.ex[ebase + e0 + lane] : make_int2(0, (int)a.absent);
      reinterpret_cast<int2 *>(ep + (((uint32_t)v.x - ep0) >> 4))[lane] = make_int2(x.x * R::size, x.y);
      if (lane < k) {
        many = a.eC[ebase + e0 + lane] > 1;
        emap[t][x.x] = (uint8_t)(e0 + lane);
      }
    }
    many = __any_sync(kAll, many);
    if (lane == 0) vt[t].w |= (many ? kManyCounts : 0) | (vs[t] == r + t + 1 ? kLeaf : 0);
  }
  __syncthreads();
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm_b) + (uint32_t)warp * (uint32_t)rows * R::size;
  const uint32_t bJ = base + lane * 16, bD = base + R::D + lane * 8, bS = base + R::S + lane * 8, bG = base + R::G + lane * 2;
  const unsigned mask = (1u << a.bits) - 1u;
  const int gend = min(a.ng, ((int)blockIdx.y + 1) * gpc);
  // the next group's sources and first separator rows
  int ns[2], nsi[2];
  bool nlive[2];
  uint2 nd[kAhead], nc[kAhead];
  auto load_ahead = [&](int g) {
    lane_sources(a, g, lane, ns, nlive);
    const size_t gt = (size_t)g * a.NT * kGroup + 2 * lane;
#pragma unroll
    for (int q = 0; q < kAhead; q++)
      if (q < b) {
        nd[q] = __ldg(reinterpret_cast<const uint2 *>(a.D + gt + (size_t)sep[q] * kGroup));
        nc[q] = __ldg(reinterpret_cast<const uint2 *>(a.S + gt + (size_t)sep[q] * kGroup));
      }
#pragma unroll
    for (int k = 0; k < 2; k++) nsi[k] = a.tidx_of[ns[k]];
  };
  const int gfirst = blockIdx.y * gpc + warp;
  if (gfirst < gend) load_ahead(gfirst);
  for (int g = gfirst; g < gend; g += nw) {
    int s[2], srow[2], si[2];
    bool live[2];
    const size_t gt = (size_t)g * a.NT * kGroup + 2 * lane, gu = (size_t)g * a.H * kGroup + 2 * lane;
    bool in_any = false, odd = false;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      s[k] = ns[k];
      si[k] = nsi[k];
      live[k] = nlive[k];
      const bool in = r <= s[k] && s[k] < r + m;
      srow[k] = in ? a.row_of[s[k]] : 0xff;  // the row of this lane's own source, if it has one
      in_any |= in;
    }
    const double zero[2] = {};
    const uint32_t none[2] = {};
    if (b == 0) row_store(bD, none);  // the whole tree: an absent entry of its root reads this row
#pragma unroll
    for (int q = 0; q < kAhead; q++)
      if (q < b) {
        const uint32_t d[2] = {nd[q].x, nd[q].y}, c[2] = {nc[q].x, nc[q].y};
        row_store(bD + q * R::size, d);
        row_store(bS + q * R::size, c);
        row_store(bJ + q * R::size, zero);
        const int sp = sep[q];
#pragma unroll
        for (int k = 0; k < 2; k++)
          if (sp == si[k]) srow[k] = q;
      }
    for (int i = kAhead; i < b; i += 4) {  // the separator's other rows, four loads of each in flight
      uint32_t d[4][2], c[4][2];
      int sp[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        sp[q] = sep[min(i + q, b - 1)];
        const uint2 dq = __ldg(reinterpret_cast<const uint2 *>(a.D + gt + (size_t)sp[q] * kGroup));
        const uint2 cq = __ldg(reinterpret_cast<const uint2 *>(a.S + gt + (size_t)sp[q] * kGroup));
        d[q][0] = dq.x;
        d[q][1] = dq.y;
        c[q][0] = cq.x;
        c[q][1] = cq.y;
      }
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (i + q < b) {
          row_store(bD + (i + q) * R::size, d[q]);
          row_store(bS + (i + q) * R::size, c[q]);
          row_store(bJ + (i + q) * R::size, zero);
#pragma unroll
          for (int k = 0; k < 2; k++)
            if (sp[q] == si[k]) srow[k] = i + q;
        }
    }
#pragma unroll
    for (int k = 0; k < 2; k++) odd |= srow[k] != 0xff || !live[k];
    // special: some lane's source lies in this subtree or among its separator, or lanes without a source
    const bool inside = __any_sync(kAll, in_any), special = __any_sync(kAll, odd || in_any);
    unsigned over = 0;

    // What vertex t does with its flows f, distances dt, counts c and arguments x1 (0 afterwards for
    // lanes that are done; else their entry, whose flow through the edge is still to be added).
    auto hand_on = [&](int t, double (&f)[2], unsigned (&x1)[2], const uint32_t (&dt)[2], const uint32_t (&c)[2]) {
      const int4 v = vt[t];
#pragma unroll
      for (int k = 0; k < 2; k++) {
        if (special && live[k] && r + t <= s[k] && s[k] < vs[t]) {
          const size_t u = gu + (size_t)(v.w & kDepthBits) * kGroup + k;
          double sd = x1[k] == 0 ? f[k] : 0.0;
          if (x1[k] == kTieCode && (unsigned)a.Ud[u] == dt[k] >> a.bits) sd = f[k] * share(1, a.Uc[u], c[k]);
          a.seed[u] = sd;
        }
        if (x1[k] - 1 < (unsigned)kBottomRows) {
          const uint32_t xo = bJ + (x1[k] - 1) * R::size + 8 * k;
          sts64(xo, lds64(xo) + f[k]);
          if (special && (int)x1[k] - 1 == srow[k]) {  // flow into the lane's own source counts apart
            atomicAdd(a.Bs + ebase + emap[t][x1[k] - 1], f[k]);
            x1[k] = 0;
          }
        } else if (x1[k] == kTieCode) {
          for (int q = 0; q < v.z >> 16; q++) {
            const int eq = (v.z & 0xffff) + q;
            const unsigned key = (unsigned)lds32(v.x + 8 * q + 4);
            const int xr = (int)(key & mask) - 1;
            const uint32_t xo = (uint32_t)xr * R::size;
            if ((uint32_t)lds32(bD + xo + 4 * k) + (key & ~mask) == dt[k]) {
              const double fl = f[k] * share(a.eC[ebase + eq], (uint32_t)lds32(bS + xo + 4 * k), c[k]);
              sts64(bJ + xo + 8 * k, lds64(bJ + xo + 8 * k) + fl);
              atomicAdd((xr == srow[k] ? a.Bs : a.Bd) + ebase + eq, fl);
            }
          }
          x1[k] = 0;
        } else {
          x1[k] = 0;
        }
      }
    };
    // the first entry that lanes still have (0: none)
    auto leader = [&](const unsigned (&x1)[2]) -> unsigned {
      const unsigned mine = x1[0] ? x1[0] : x1[1], any = __ballot_sync(kAll, mine != 0);
      return any ? __shfl_sync(kAll, mine, __ffs(any) - 1) : 0u;
    };

    uint32_t off = b * R::size;  // of the next row
    int4 v = lds128(vt0), e = lds128(v.x);
    for (int t = 0; t < m; t++) {
      const int4 vn = lds128(vt0 + 16 * (t + 1));
      unsigned m1[2] = {kNoKey, kNoKey}, m2[2] = {kNoKey, kNoKey};
      if (inside) {
        const int se = vs[t];
#pragma unroll
        for (int k = 0; k < 2; k++) {
          m1[k] = up_key(a, r + t <= s[k] && s[k] < se, gu + (size_t)(v.w & kDepthBits) * kGroup + k);
          m2[k] = m1[k] == kNoKey ? kNoKey : m1[k] ^ mask;
        }
      }
      uint32_t pe = v.x;
      do {
        uint32_t d1[2], d2[2];
        row_load(bD + e.x, d1);
        row_load(bD + e.z, d2);
        const int4 ec = e;
        pe += 16;
        if (pe < (uint32_t)v.y) e = lds128(pe);
#pragma unroll
        for (int k = 0; k < 2; k++) key_min2(m1[k], m2[k], d1[k] + (unsigned)ec.y, d2[k] + (unsigned)ec.w, mask);
      } while (pe < (uint32_t)v.y);
      e = lds128(vn.x);
      const bool leaf = v.w & kLeaf;
      if (leaf && !special) {  // (its entries are arcs, one path each: one entry's count needs no check)
        const unsigned x0 = m1[0] & mask;  // one entry for the lane's two sources, and for all lanes?
        const bool one = ((m1[0] ^ m2[0]) == mask) & ((m1[1] ^ m2[1]) == mask) & ((m1[1] & mask) == x0);
        int all = 0;
        __match_all_sync(kAll, one ? x0 : 0x100u + lane, &all);
        if (all) {
          double j[2];
          const uint32_t xo = bJ + (x0 - 1) * R::size;
          row_load(xo, j);
          j[0] += 1.0;
          j[1] += 1.0;
          row_store(xo, j);
          uint8_t *lu = &leaf_units[warp][emap[t][x0 - 1]];
          const uint8_t units = *lu + 1;
          __syncwarp();
          *lu = units;
          v = vn;
          continue;
        }
      }
      unsigned x1[2];
      uint32_t c[2], dt[2];
      unsigned again = 0;  // several entries reach the minimum
#pragma unroll
      for (int k = 0; k < 2; k++) {
        x1[k] = m1[k] & mask;
        dt[k] = m1[k] & ~mask;
        again |= m1[k] ^ m2[k] ^ mask;
        c[k] = (uint32_t)lds32(bS + 4 * k + (max(x1[k], 1u) - 1) * R::size);
      }
      if (inside)
#pragma unroll
        for (int k = 0; k < 2; k++)
          if (x1[k] == 0) c[k] = a.Uc[gu + (size_t)(v.w & kDepthBits) * kGroup + k];
      if (__any_sync(kAll, (again != 0) | (v.w < 0))) {  // or counts above 1: the edges once more
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const bool tk = (m1[k] ^ m2[k]) != mask;
          unsigned long long cc = x1[k] == 0 ? c[k] : 0;
          for (int q = 0; q < v.z >> 16; q++) {
            const unsigned key = (unsigned)lds32(v.x + 8 * q + 4);
            const uint32_t xo = ((key & mask) - 1) * R::size + 4 * k;
            const bool hit = tk ? (uint32_t)lds32(bD + xo) + (key & ~mask) == dt[k] : (key & mask) == x1[k];
            if (hit) cc += (unsigned long long)(unsigned)a.eC[ebase + (v.z & 0xffff) + q] * (uint32_t)lds32(bS + xo);
            if (cc > 0x7fffffffull) {
              over = 1;
              cc = 1;
            }
          }
          c[k] = (uint32_t)cc;
          if (tk) x1[k] = kTieCode;
        }
      }
      if (special)
#pragma unroll
        for (int k = 0; k < 2; k++)
          if (!live[k]) x1[k] = kSkipCode;
      if (!leaf) {
        row_store(bD + off, dt);
        row_store(bS + off, c);
        row_store(bJ + off, zero);
        code_store(bG + off, x1[0] | (x1[1] << 8));
        off += R::size;
      } else {  // several entries, or special
        double f[2];
#pragma unroll
        for (int k = 0; k < 2; k++) f[k] = r + t != s[k] ? 1.0 : 0.0;  // the source itself is no target
        hand_on(t, f, x1, dt, c);
        for (unsigned xl; (xl = leader(x1)) != 0;) {
          int cnt = 0;
#pragma unroll
          for (int k = 0; k < 2; k++) {
            cnt += __popc(__ballot_sync(kAll, x1[k] == xl && f[k] != 0.0));
            if (x1[k] == xl) x1[k] = 0;
          }
          if (lane == 0) atomicAdd(a.Bd + ebase + emap[t][xl - 1], (double)cnt);
        }
      }
      v = vn;
    }
    if (over) *a.wrap = 1;
    if (g + nw < gend) load_ahead(g + nw);
    for (int i = nr - 1; i >= 0; i--) {
      off -= R::size;
      const unsigned code = code_load(bG + off);
      double f[2];
      row_load(bJ + off, f);
      unsigned x1[2] = {code & 0xff, code >> 8};
      int all = 0;
      __match_all_sync(kAll, code, &all);
      if (all && !special && x1[0] == x1[1] && x1[0] <= kBottomRows) {  // (no U without special)
        double j[2];
        const uint32_t xo = (x1[0] - 1) * R::size;
        row_load(bJ + xo, j);
        j[0] += f[0] + 1.0;
        j[1] += f[1] + 1.0;
        row_store(bJ + xo, j);
        sts32(base + off + R::lead, x1[0] | kLeadFull);
        continue;
      }
      const int t = vertex_of[i];
      uint32_t dt[2], c[2];
      row_load(bD + off, dt);
      row_load(bS + off, c);
#pragma unroll
      for (int k = 0; k < 2; k++)
        if (r + t != s[k]) f[k] += 1.0;  // the source itself is no target
      hand_on(t, f, x1, dt, c);
      // two entries wait for the end, a value per lane each; any others now, one after another
      unsigned leads = 0;
      double w[2];
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const unsigned xl = leader(x1);
        w[j] = 0.0;
        leads |= xl << (8 * j);
#pragma unroll
        for (int k = 0; k < 2; k++)
          if (xl && x1[k] == xl) {
            w[j] += f[k];
            x1[k] = 0;
          }
      }
      row_store(bJ + off, w);
      sts32(base + off + R::lead, leads);
      for (unsigned xl; (xl = leader(x1)) != 0;) {
        double z = 0.0;
#pragma unroll
        for (int k = 0; k < 2; k++)
          if (x1[k] == xl) {
            z += f[k];
            x1[k] = 0;
          }
        z = warp_sum(z);
        if (lane == 0) atomicAdd(a.Bd + ebase + emap[t][xl - 1], z);
      }
    }
    __syncwarp();
    // the deferred sums: eight rows at a time, four lanes of eight columns each
    for (int i0 = 0; i0 < nr; i0 += 8) {
      const int i = min(i0 + (lane >> 2), nr - 1);
      const uint32_t ro = base + (b + i) * R::size;
      const unsigned leads = i0 + (lane >> 2) < nr ? (unsigned)lds32(ro + R::lead) : 0;
      double z[2] = {};
      if (leads) {
#pragma unroll
        for (int q = 0; q < 8; q++) {
          double x[2];
          row_load(ro + ((lane & 3) * 8 + q) * 16, x);
          z[0] += x[0];
          z[1] += x[1];
        }
      }
      if (leads & kLeadFull) z[0] += z[1];  // one entry: both values of a lane are its
#pragma unroll
      for (int j = 0; j < 2; j++) {
        z[j] += __shfl_xor_sync(kAll, z[j], 1);
        z[j] += __shfl_xor_sync(kAll, z[j], 2);
        const unsigned x = (leads >> (8 * j)) & 0xff;
        if (x && (lane & 3) == j)
          atomicAdd(a.Bd + ebase + emap[vertex_of[i]][x - 1], leads & kLeadFull ? z[j] + (double)kGroup : z[j]);
      }
    }
    for (int i = 0; i < b; i++) {
      double z[2];
      row_load(bJ + i * R::size, z);
#pragma unroll
      for (int k = 0; k < 2; k++)
        if (z[k] != 0.0) atomicAdd(a.J + gt + (size_t)sep[i] * kGroup + k, z[k]);
    }
    __syncwarp();
  }
  const int ne = a.xoff[r + m] - ebase;
  for (int i = lane; i < ne; i += 32)
    if (leaf_units[warp][i]) atomicAdd(a.Bd + ebase + i, (double)leaf_units[warp][i] * kGroup);
  end();
}

// ------------------------------------------------------------------------------- unpack, finish
// Before the unpacking: a shortcut's flow on the way down is dependency of its upper end, that on the
// way up of its lower end (the flow from an end's own source is not); then one total per edge.
__global__ void k_fold(int64_t E, const int4 *__restrict__ eup, const int32_t *__restrict__ owner, double *Bd,
                       const double *__restrict__ Bu, const double *__restrict__ Bs, double *F, const int32_t *wrap) {
  if (__ldcg(wrap) != 0) return;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  const double d = Bd[e], u = Bu[e];
  if (d != 0.0) atomicAdd(F + eup[e].w, d);
  if (u != 0.0) atomicAdd(F + owner[e], u);
  Bd[e] = d + u + Bs[e];
}

// One triangle: its share of the shortcut's flow passes to the two parts and is dependency of the
// vertex between.
__device__ __forceinline__ void unpack_one(const int4 t, const int32_t *eC, double *B, double *F) {
  double w = __ldcg(B + t.z);
  if (w == 0.0) return;
  const int c1 = eC[t.x], c3 = eC[t.z];
  if (c3 != 1) w *= share(c1, (uint32_t)eC[t.y], (uint32_t)c3);
  atomicAdd(B + t.x, w);
  atomicAdd(B + t.y, w);
  atomicAdd(F + t.w, w);
}

// A level of triangles is final once the levels before it are done: a launch per large level, and
// the small ones at the end by one cluster, a triangle per thread, with cluster barriers between them.
// A level is a chain of latencies (its B, the atomics, the barrier), so the next level's triangle and
// share, which no level changes, are loaded before the barrier: 55 us for the last levels at 50k
// vertices, 94 with one CTA and up to eight triangles per thread.
__global__ void k_unpack(const int4 *__restrict__ tri, int64_t count, const int32_t *__restrict__ eC, double *B, double *F,
                         const int32_t *wrap) {
  if (__ldcg(wrap) != 0) return;
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < count) unpack_one(tri[k], eC, B, F);
}

constexpr int kTailCtas = 8;
constexpr int64_t kTailLevel = kTailCtas * 1024;  // triangles of a level that the cluster takes
__global__ void __cluster_dims__(kTailCtas, 1, 1) __launch_bounds__(1024)
    k_unpack_tail(const int4 *__restrict__ tri, const int64_t *__restrict__ at, int l0, int l1, const int32_t *__restrict__ eC,
                  double *B, double *F, const int32_t *wrap) {
  if (__ldcg(wrap) != 0) return;  // (not written while this kernel runs, so the same for all)
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int4 t = make_int4(0, 0, 0, 0);
  double part = 0.0;  // 0: no triangle
  auto load = [&](int l) {
    const int64_t b = at[l], e = at[l + 1];
    part = 0.0;
    if (b + k >= e) return;
    t = tri[b + k];
    const int c1 = eC[t.x], c3 = eC[t.z];
    part = c3 == 1 ? 1.0 : share(c1, (uint32_t)eC[t.y], (uint32_t)c3);
  };
  load(l0);
  for (int l = l0; l < l1; l++) {
    if (part != 0.0) {
      const double w = __ldcg(B + t.z) * part;
      if (w != 0.0) {
        atomicAdd(B + t.x, w);
        atomicAdd(B + t.y, w);
        atomicAdd(F + t.w, w);
      }
    }
    if (l + 1 == l1) break;
    load(l + 1);
    __threadfence();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// The result of a call is left out where its counts wrapped, and where the error word is set (a source
// id out of range, read here as vertex 0): the call reports that, and the caller's BC stays as it was, as
// with the dependency kernels (see rows_failed).  err: the error word, then the wrap word.
__device__ __forceinline__ bool result_void(const int32_t *err) { return __ldcg(err) != ERR_NONE || __ldcg(err + 1) != 0; }

__global__ void k_finish(const double *__restrict__ F, double *__restrict__ bc_tid, int n, const int32_t *err) {
  if (result_void(err)) return;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) bc_tid[t] += 0.5 * F[t];
}

// ------------------------------------------------------------------------------- plan
// separator entries of each vertex sorted by tid: an entry's place is the number of smaller ones
__global__ void k_sort_edges(const int64_t *__restrict__ soff, const int4 *__restrict__ sep, int n, int32_t *xtid,
                             int32_t *eL, int32_t *eC) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (t >= n) return;
  const int64_t b = soff[t];
  const int k = (int)(soff[t + 1] - b);
  for (int i = lane; i < k; i += 32) {
    const int4 v = sep[b + i];
    int pos = 0;
    for (int j = 0; j < k; j++) pos += __ldg(reinterpret_cast<const int *>(sep + b + j)) < v.x;
    xtid[b + pos] = v.x;
    eL[b + pos] = v.y;
    eC[b + pos] = v.z;
  }
}

// per-edge references once the trunk and bottoms are known; edges that cannot carry a shortest path
// (L above every distance) are clamped so that keys stay in 32 bits
__global__ void k_edge_refs(const int32_t *__restrict__ xoff, const int32_t *__restrict__ xtid, const int32_t *__restrict__ eL,
                            const int32_t *__restrict__ depth, const int32_t *__restrict__ tidx_of, const int4 *__restrict__ bot, const uint8_t *__restrict__ row_of,
                            int n, int bits, int32_t lcap, const int32_t *__restrict__ eC, int2 *ex, int4 *eup,
                            int32_t *etr) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (t >= n) return;
  const int ti = tidx_of[t];
  int4 bt = make_int4(0, 0, 0, 0);
  if (ti < 0) bt = bot[-1 - ti];
  for (int e = xoff[t] + lane; e < xoff[t + 1]; e += 32) {
    const int x = xtid[e];
    int ref = tidx_of[x];
    etr[e] = ref < 0 ? -1 : ref;
    if (ti < 0) {
      if (x >= bt.x) ref = row_of[x];
      else {  // a separator vertex of the bottom's root: its position in the root's list
        int lo = xoff[bt.x], hi = xoff[bt.x + 1];
        const int b0 = lo;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (xtid[mid] < x) lo = mid + 1;
          else hi = mid;
        }
        ref = lo - b0;
      }
    }
    ex[e] = make_int2(ref, (int)(((unsigned)min(eL[e], lcap) << bits) | (unsigned)(ti < 0 ? ref + 1 : e - xoff[t] + 1)));
    eup[e] = make_int4(depth[x] - 1, min(eL[e], lcap), eC[e], x);
  }
}

// edges of a trunk vertex to its own piece: the last of its list
__global__ void k_piece_edges(TreeArgs a, int4 *tmeta) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= a.NT) return;
  const int4 m = tmeta[i];
  const int start = a.piece[a.piece_of[i]].x;
  int c = 0;
  for (int e = m.x + lane; e < m.y; e += 32) c += a.ex[e].x >= start;
  c = __reduce_add_sync(kAll, c);
  if (lane == 0) tmeta[i].z = c;
}

// triangles (y; t, x): shortcut (t, x) of least length through y.  A warp per (y, deeper vertex t),
// from edge E0 on (the edges of a core before it are no eliminated vertex's).
__global__ void k_triangles(const int32_t *__restrict__ xoff, const int32_t *__restrict__ xtid, const int32_t *__restrict__ eL,
                            const int32_t *__restrict__ owner, int64_t E0, int64_t E, int4 *tri, unsigned long long *count,
                            unsigned long long cap) {
  const int64_t e2 = E0 + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (e2 >= E) return;
  const int y = owner[e2], first = xoff[y], t = xtid[e2], l2 = eL[e2];
  const int tb = xoff[t], te = xoff[t + 1];
  for (int e1b = first; e1b < (int)e2; e1b += 32) {
    const int e1 = e1b + lane;
    int e3 = -1;
    if (e1 < (int)e2) {
      const int x = xtid[e1];
      int lo = tb, hi = te;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(xtid + mid) < x) lo = mid + 1;
        else hi = mid;
      }
      if (lo < te && xtid[lo] == x && eL[lo] == eL[e1] + l2) e3 = lo;
    }
    const unsigned hit = __ballot_sync(kAll, e3 >= 0);
    if (!hit) continue;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(count, (unsigned long long)__popc(hit));
    base = __shfl_sync(kAll, base, 0);
    if (e3 >= 0) {
      const unsigned long long pos = base + __popc(hit & ((1u << lane) - 1u));
      if (pos < cap) tri[pos] = make_int4(e1, (int)e2, e3, y);
    }
  }
}

__global__ void k_owner(const int32_t *__restrict__ xoff, int n, int32_t *owner) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (t >= n) return;
  for (int e = xoff[t] + lane; e < xoff[t + 1]; e += 32) owner[e] = t;
}

// level of an edge: one more than the highest level of a shortcut it is a part of
__global__ void k_levels(const int4 *__restrict__ tri, int64_t count, int32_t *lvl, int32_t *changed) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  const int4 t = tri[k];
  const int l = __ldcg(lvl + t.z) + 1;
  if (l > kMaxUnpackLevels) {  // deeper nesting than the plan takes: never settles
    *changed = l;
    return;
  }
  const bool up = atomicMax(lvl + t.x, l) < l;
  const bool up2 = atomicMax(lvl + t.y, l) < l;
  if (up || up2) *changed = l;
}

__global__ void k_level_hist(const int4 *__restrict__ tri, int64_t count, const int32_t *__restrict__ lvl, unsigned long long *hist) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < count) atomicAdd(hist + lvl[tri[k].z], 1ull);
}

__global__ void k_level_scatter(const int4 *__restrict__ tri, int64_t count, const int32_t *__restrict__ lvl,
                                unsigned long long *next, int4 *out) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < count) {
    const int4 t = tri[k];
    out[atomicAdd(next + lvl[t.z], 1ull)] = t;
  }
}

// path counts of the shortcuts recomputed in FP64 from the arcs and the triangles, highest level
// first: where one differs from the 32-bit count, that count has wrapped
__global__ void k_count_arcs(const int32_t *__restrict__ owner, const int32_t *__restrict__ xtid, const int32_t *__restrict__ eL,
                             int64_t E, const int2 *__restrict__ arc_rng, const int2 *__restrict__ arc_hw, double *cd) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  const int2 rng = arc_rng[owner[e]];
  double c = 0.0;
  for (int q = rng.x; q < rng.y; q++) {
    const int2 hw = arc_hw[q];
    if (hw.x == xtid[e] && hw.y == eL[e]) c = 1.0;
  }
  cd[e] = c;
}

__global__ void k_count_triangles(const int4 *__restrict__ tri, int64_t count, double *cd) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  const int4 t = tri[k];
  atomicAdd(cd + t.z, __ldcg(cd + t.x) * __ldcg(cd + t.y));
}

__global__ void k_count_check(const double *__restrict__ cd, const int32_t *__restrict__ eC, int64_t E, int32_t *bad) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < E && (cd[e] != (double)eC[e] || eC[e] < 1)) *bad = 1;
}

inline unsigned blocks_for(int64_t threads, int per) { return (unsigned)std::max<int64_t>(1, (threads + per - 1) / per); }

#include "core.cuh"

}  // namespace

// Host part and device arrays of the plan.
struct TreePlan {
  TreeArgs args{};  // without the per-launch fields
  int nbot = 0, up_warps = 0;
  std::vector<int32_t> level_class;  // 4 per trunk level: first piece, of at most 16, of at most 8 vertices, end
  struct BotClass {
    int first, end, rows;
  };
  std::vector<BotClass> bot_class;
  std::vector<int64_t> tri_first;    // first triangle of each unpack level, end
  int4 *tri = nullptr;
  int64_t *tri_at = nullptr;         // tri_first on the device
  int32_t *owner = nullptr;          // per edge its lower end
  int tail_level = 0;                // levels from here on hold at most kTailLevel triangles each
  int64_t E = 0, bytes = 0;
  bool off = false;  // a count wrapped: the label kernels answer from now on
  CoreArgs core{};   // label-free index: nc > 0, without the scratch
  const int32_t *cid_of = nullptr;
  std::vector<void *> owned;

  char *arena = nullptr;  // one allocation for most arrays: each cudaMalloc and cudaFree costs a build ~0.1 ms
  size_t arena_left = 0;

  void *device(size_t size) {
    void *p = nullptr;
    CK(cudaMalloc(&p, size));
    owned.push_back(p);
    bytes += (int64_t)size;
    return p;
  }
  template <class T>
  T *alloc(size_t count) {
    const size_t size = (std::max<size_t>(count, 1) * sizeof(T) + 255) & ~(size_t)255;
    if (size > arena_left) return (T *)device(size);
    char *p = arena;
    arena += size;
    arena_left -= size;
    return (T *)p;
  }
  template <class T>
  T *upload(const std::vector<T> &v, cudaStream_t st) {
    T *p = alloc<T>(v.size());
    if (!v.empty()) CK(cudaMemcpyAsync(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st));
    return p;
  }
};

void tree_free(DeviceState *d) {
  if (!d->tree) return;
  for (void *p : d->tree->owned) cudaFree(p);
  d->bytes -= d->tree->bytes;
  delete d->tree;
  d->tree = nullptr;
}

// Trunk, pieces and bottoms from the tree (see k_trunk_down and k_bottom).
struct TreeShape {
  std::vector<int32_t> tidx_of;  // tid -> trunk index or -1 - bottom
  std::vector<int4> bot, piece;
  std::vector<uint8_t> row_of;   // tid in a bottom -> row, 0xff without descendants
  std::vector<int32_t> piece_of, level_first, trunk_tid, chain_off;
  std::vector<int2> chain;       // see TreeArgs
};

static TreeShape tree_shape(const Index &ix, const std::vector<int64_t> &soff) {
  const int32_t n = ix.n;
  TreeShape s;
  s.tidx_of.assign((size_t)n, 0);
  std::vector<int32_t> heavy((size_t)n, -1), piece((size_t)n, -1);
  // bottoms: maximal subtrees whose separator and vertices fit the rows
  std::vector<char> is_bot((size_t)n, 0);
  std::vector<int32_t> inner((size_t)n + 1, 0);  // vertices with descendants before t
  for (int32_t t = 0; t < n; t++) inner[t + 1] = inner[t] + (ix.send[t] > t + 1);
  s.row_of.assign((size_t)n, 0xff);
  for (int32_t t = 0; t < n;) {
    const int32_t size = ix.send[t] - t, k = (int32_t)(soff[t + 1] - soff[t]), rows = k + inner[ix.send[t]] - inner[t];
    if (rows <= kBottomRows && size <= kBottomVerts && soff[ix.send[t]] - soff[t] <= kBottomEdges) {
      s.bot.push_back(make_int4(t, size, k, rows));
      for (int32_t x = t; x < ix.send[t]; x++) {
        is_bot[x] = 1;
        if (ix.send[x] > x + 1) s.row_of[x] = (uint8_t)(k + inner[x] - inner[t]);
      }
      t = ix.send[t];
    } else {
      t++;
    }
  }
  std::stable_sort(s.bot.begin(), s.bot.end(), [](const int4 &x, const int4 &y) { return x.w > y.w; });
  for (size_t i = 0; i < s.bot.size(); i++)
    for (int32_t t = s.bot[i].x; t < s.bot[i].x + s.bot[i].y; t++) s.tidx_of[t] = -1 - (int32_t)i;
  // pieces: paths along the child with the largest subtree
  for (int32_t t = n - 1; t > 0; t--)
    if (!is_bot[t]) {
      const int32_t p = ix.parent[t];
      if (heavy[p] < 0 || ix.send[t] - t >= ix.send[heavy[p]] - heavy[p]) heavy[p] = t;
    }
  struct P {
    std::vector<int32_t> v;
    int32_t level;
  };
  std::vector<P> ps;
  int32_t levels = 0;
  for (int32_t t = 0; t < n; t++) {
    if (is_bot[t]) continue;
    const int32_t p = ix.parent[t];
    if (p >= 0 && heavy[p] == t && (int)ps[piece[p]].v.size() < kPieceLen && ps[piece[p]].v.back() == p) {
      piece[t] = piece[p];
    } else {
      piece[t] = (int32_t)ps.size();
      ps.push_back({{}, p < 0 ? 0 : ps[piece[p]].level + 1});
      levels = std::max(levels, ps.back().level + 1);
    }
    ps[piece[t]].v.push_back(t);
  }
  s.level_first.assign((size_t)levels + 1, 0);
  for (const P &p : ps) s.level_first[p.level + 1]++;
  for (int32_t l = 0; l < levels; l++) s.level_first[l + 1] += s.level_first[l];
  std::vector<int32_t> by_level(ps.size());  // by level, longest first
  for (size_t i = 0; i < ps.size(); i++) by_level[i] = (int32_t)i;
  std::stable_sort(by_level.begin(), by_level.end(), [&](int32_t x, int32_t y) {
    return ps[x].level != ps[y].level ? ps[x].level < ps[y].level : ps[x].v.size() > ps[y].v.size();
  });
  s.chain_off.assign(1, 0);
  for (int32_t id : by_level) {
    const int32_t first = (int32_t)s.trunk_tid.size(), np = (int32_t)s.piece.size();
    for (int32_t t : ps[id].v) {
      s.tidx_of[t] = (int32_t)s.trunk_tid.size();
      s.trunk_tid.push_back(t);
      s.piece_of.push_back(np);
    }
    const int32_t par = ix.parent[ps[id].v[0]];
    s.piece.push_back(make_int4(first, (int32_t)s.trunk_tid.size(), par < 0 ? -1 : s.tidx_of[par], 0));
    if (par >= 0) {  // the parent's piece comes first, up to the parent itself
      const int32_t pp = s.piece_of[s.tidx_of[par]], b = s.chain_off[pp], e = s.chain_off[pp + 1];
      for (int32_t c = b; c < e; c++) s.chain.push_back(s.chain[c]);
    }
    s.chain.push_back(make_int2(first, ix.depth[ps[id].v[0]] - 1));
    s.chain_off.push_back((int32_t)s.chain.size());
  }
  return s;
}

// Triangles of the edges [E0, E), level by level; false where their levels do not settle.
template <class F>
static bool build_triangles(TreePlan *p, int64_t E0, int64_t E, const int32_t *xtid, const int32_t *eL, F &&talloc, cudaStream_t st) {
  const TreeArgs &a = p->args;
  p->tri_first.assign(1, 0);
  if (E0 >= E) return true;
  int32_t *lvl = (int32_t *)talloc((size_t)E * 4), *flag = (int32_t *)talloc(16);
  unsigned long long *cnt = (unsigned long long *)talloc(8 * (kMaxUnpackLevels + 2));
  unsigned long long cap = (unsigned long long)E + 1024, found = 0;
  int4 *raw = nullptr;
  for (int round = 0; round < 2; round++) {
    raw = (int4 *)talloc((size_t)cap * 16);
    CK(cudaMemsetAsync(cnt, 0, 8, st));
    k_triangles<<<blocks_for((E - E0) * 32, 256), 256, 0, st>>>(a.xoff, xtid, eL, p->owner, E0, E, raw, cnt, cap);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(&found, cnt, 8, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (found <= cap) break;
    cap = found;
  }
  const int64_t T = (int64_t)found;
  if (T == 0) return true;
  CK(cudaMemsetAsync(lvl, 0, (size_t)E * 4, st));
  bool settled = false;
  for (int round = 0; round <= kMaxUnpackLevels && !settled; round += 4) {
    int32_t ch = 0;
    for (int q = 0; q < 4; q++) {
      if (q == 3) CK(cudaMemsetAsync(flag, 0, 4, st));
      k_levels<<<blocks_for(T, 256), 256, 0, st>>>(raw, T, lvl, flag);
      CK(cudaGetLastError());
    }
    CK(cudaMemcpyAsync(&ch, flag, 4, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    settled = ch == 0;
  }
  if (!settled) return false;
  std::vector<unsigned long long> hist((size_t)kMaxUnpackLevels + 2, 0), first(1, 0);
  CK(cudaMemsetAsync(cnt, 0, 8 * (kMaxUnpackLevels + 2), st));
  k_level_hist<<<blocks_for(T, 256), 256, 0, st>>>(raw, T, lvl, cnt);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(hist.data(), cnt, hist.size() * 8, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  int32_t top = 0;
  while (top < kMaxUnpackLevels && hist[top]) top++;
  for (int l = 0; l < top; l++) {
    p->tri_first.push_back(p->tri_first.back() + (int64_t)hist[l]);
    first.push_back((unsigned long long)p->tri_first.back());
  }
  if (p->tri_first.back() != T) return false;
  p->tri = p->alloc<int4>((size_t)T);
  p->tri_at = p->upload(p->tri_first, st);
  p->tail_level = top;
  while (p->tail_level > 0 && hist[p->tail_level - 1] <= (unsigned long long)kTailLevel) p->tail_level--;
  CK(cudaMemcpyAsync(cnt, first.data(), first.size() * 8, cudaMemcpyHostToDevice, st));
  k_level_scatter<<<blocks_for(T, 256), 256, 0, st>>>(raw, T, lvl, cnt, p->tri);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(st));  // the staging vectors die here
  return true;
}

// Bottoms come with the most rows first: a launch per four rows.
static void bottom_classes(TreePlan *p, const std::vector<int4> &bot) {
  p->nbot = (int)bot.size();
  for (int i = 0; i < p->nbot;) {
    auto rows_of = [&](int q) { return std::max(4, (bot[q].w + 3) & ~3); };
    int e = i;
    while (e < p->nbot && rows_of(e) == rows_of(i)) e++;
    p->bot_class.push_back({i, e, rows_of(i)});
    i = e;
  }
}

// Temporaries of a plan's build: in the per-source scratch, which no call uses yet, as far as it
// reaches, else on their own.
struct PlanScratch {
  char *spare;
  size_t left;
  std::vector<void *> own;
  explicit PlanScratch(DeviceState *d)
      : spare(reinterpret_cast<char *>(d->rec[0])), left((size_t)d->chunk * d->n_pad * sizeof(int4)) {}
  ~PlanScratch() {
    for (void *q : own) cudaFree(q);
  }
  void *operator()(size_t bytes) {
    bytes = (std::max<size_t>(bytes, 16) + 255) & ~(size_t)255;
    if (bytes <= left) {
      char *q = spare;
      spare += bytes;
      left -= bytes;
      return q;
    }
    void *q = nullptr;
    CK(cudaMalloc(&q, bytes));
    own.push_back(q);
    return q;
  }
};

// The plan is the index's now, or gone.
static void plan_done(DeviceState *d, bool keep) {
  if (keep) {
    d->bytes += d->tree->bytes;
  } else {
    d->tree->bytes = 0;
    tree_free(d);
  }
}

// After an exception in a build: no room for the plan means that the general kernels answer.
static void plan_failed(DeviceState *d) {
  plan_done(d, false);
  try {
    throw;
  } catch (const Error &e) {
    if (e.code != QBC_ENOMEM) throw;
    cudaGetLastError();
  }
}

// Builds the plan from the separators (soff on the host; d_soff / d_sep their device copies).  The
// plan is left out, and the label kernels keep answering, where its keys do not fit 32 bits, a
// shortcut count has wrapped, a row does not fit shared memory, or memory is short.
void tree_build(Handle &h, DeviceState *d, const std::vector<int64_t> &soff, const int64_t *d_soff, const int4 *d_sep) {
  NvtxRange nvtx("qbc.tree_plan");
  TraceScope trace("tree plan");
  const Index &ix = h.host;
  tree_free(d);
  const int64_t E = soff[ix.n];
  const int32_t H = ix.tree_height;
  if (ix.kind == IndexKind::CSR || ix.counts_wrapped || E >= INT_MAX || H < 1 || H > 65535) return;
  int bits = 6;  // an entry index (a separator position + 1, or a bottom row + 1) below 2^bits - 1
  while ((1 << bits) - 1 <= ix.tree_width + 1 && bits < 16) bits++;
  const uint64_t lim = 1ull << (32 - bits);
  const uint64_t dmax = 2ull * (uint64_t)std::max(ix.max_label, 0);  // no distance is longer
  if (ix.tree_width >= 65000 || 2 * dmax + 4 >= lim) return;
  auto warps_for = [&](size_t per_warp) {
    int w = 16;
    while (w > 1 && w * per_warp > (size_t)d->smem_optin - 2048) w--;
    return w * per_warp > (size_t)d->smem_optin - 2048 ? 0 : w;
  };
  const int up_warps = warps_for((size_t)H * 8);
  if (!up_warps || (size_t)H * 20 + sizeof(BackShared<8>) > (size_t)d->smem_optin - 2048) return;
  cudaStream_t st = d->s_label;
  auto p = new TreePlan();
  d->tree = p;
  PlanScratch talloc(d);
  bool keep = false;
  try {
    TreeArgs &a = p->args;
    p->E = E;
    p->up_warps = up_warps;
    const int32_t n = ix.n;
    const TreeShape s = tree_shape(ix, soff);
    for (size_t l = 0; l + 1 < s.level_first.size(); l++) {  // (longest first, see tree_shape)
      int32_t q = s.level_first[l];
      p->level_class.push_back(q);
      for (int32_t lim : {16, 8}) {
        while (q < s.level_first[l + 1] && s.piece[q].y - s.piece[q].x > lim) q++;
        p->level_class.push_back(q);
      }
      p->level_class.push_back(s.level_first[l + 1]);
    }
    bottom_classes(p, s.bot);
    a.n = n;
    a.H = H;
    a.NT = (int)s.trunk_tid.size();
    a.bits = bits;
    a.dist_lim = (unsigned)(dmax + 1);
    a.absent = ((unsigned)(lim - 2 - dmax) << bits) | ((1u << bits) - 2u);
    {
      const size_t N = (size_t)n, T = s.trunk_tid.size(), e = (size_t)E;
      p->arena_left = N * (4 + 4 + 1 + 8) + T * (16 + 8 + 4) + (s.piece.size() + s.bot.size()) * 16 + e * (8 + 4 + 4 + 4 + 16 + 24) + 64 * 256;
      p->arena = (char *)p->device(p->arena_left);
    }
    std::vector<int32_t> xoff(soff.begin(), soff.end());
    std::vector<int4> tmeta((size_t)a.NT);
    std::vector<int2> tsub((size_t)a.NT);
    for (int i = 0; i < a.NT; i++) {
      const int32_t t = s.trunk_tid[i];
      tmeta[i] = make_int4(xoff[t], xoff[t + 1], 0, t);
      tsub[i] = make_int2(ix.send[t], ix.depth[t] - 1);
    }
    a.xoff = p->upload(xoff, st);
    int4 *tm = p->upload(tmeta, st);
    a.tmeta = tm;
    a.tsub = p->upload(tsub, st);
    a.piece = p->upload(s.piece, st);
    a.piece_of = p->upload(s.piece_of, st);
    a.chain_off = p->upload(s.chain_off, st);
    a.chain = p->upload(s.chain, st);
    a.tidx_of = p->upload(s.tidx_of, st);
    a.bot = p->upload(s.bot, st);
    a.row_of = p->upload(s.row_of, st);
    a.depth = d->depth;
    a.parent = d->parent;
    a.send = d->send;
    int2 *ex = p->alloc<int2>((size_t)E);
    int32_t *eC = p->alloc<int32_t>((size_t)E), *etr = p->alloc<int32_t>((size_t)E), *owner = p->alloc<int32_t>((size_t)E);
    int4 *eup = p->alloc<int4>((size_t)E);
    a.ex = ex;
    a.eC = eC;
    a.eup = eup;
    p->owner = owner;
    a.etr = etr;
    // the accumulators of a call, cleared together: per edge three, per vertex one
    a.Bd = p->alloc<double>((size_t)E * 3 + (size_t)n);
    a.Bu = a.Bd + E;
    a.Bs = a.Bu + E;
    a.F = a.Bs + E;
    if (d->ch) {
      a.lab_off = d->lab_off;
      a.lab_dis = d->dis;
      a.lab_ch = d->ch;
      a.lab_bits = d->packed_bits;
    }
    a.wrap = d->err + 1;
    CK(cudaMemsetAsync(a.wrap, 0, 4, st));
    int32_t *xtid = (int32_t *)talloc((size_t)E * 4), *eL = (int32_t *)talloc((size_t)E * 4);
    double *cd = a.Bd;  // the edge accumulators are free until the first call
    int32_t *flag = (int32_t *)talloc(16);
    if (E > 0) {
      k_sort_edges<<<blocks_for((int64_t)n * 32, 256), 256, 0, st>>>(d_soff, d_sep, n, xtid, eL, eC);
      CK(cudaGetLastError());
      k_owner<<<blocks_for((int64_t)n * 32, 256), 256, 0, st>>>(a.xoff, n, owner);
      CK(cudaGetLastError());
      const int32_t lcap = (int32_t)(lim - 2 - dmax);
      k_edge_refs<<<blocks_for((int64_t)n * 32, 256), 256, 0, st>>>(a.xoff, xtid, eL, d->depth, a.tidx_of, a.bot, a.row_of, n, bits, lcap, eC,
                                                                  ex, eup, etr);
      CK(cudaGetLastError());
      if (a.NT > 0) {
        k_piece_edges<<<blocks_for((int64_t)a.NT * 32, 256), 256, 0, st>>>(a, tm);
        CK(cudaGetLastError());
      }
      if (build_triangles(p, 0, E, xtid, eL, talloc, st)) {
        const int top = (int)p->tri_first.size() - 1;
        k_count_arcs<<<blocks_for(E, 256), 256, 0, st>>>(owner, xtid, eL, E, d->arc_rng, d->arc_hw, cd);
        CK(cudaGetLastError());
        for (int l = top - 1; l >= 0; l--) {
          const int64_t b = p->tri_first[l], c = p->tri_first[l + 1] - b;
          k_count_triangles<<<blocks_for(c, 256), 256, 0, st>>>(p->tri + b, c, cd);
          CK(cudaGetLastError());
        }
        int32_t bad = 0;
        CK(cudaMemsetAsync(flag, 0, 4, st));
        k_count_check<<<blocks_for(E, 256), 256, 0, st>>>(cd, eC, E, flag);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(&bad, flag, 4, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        keep = bad == 0;
      }
    } else {
      p->tri_first.assign(1, 0);
      keep = true;
    }
    CK(cudaStreamSynchronize(st));  // the staging vectors die here
  } catch (...) {
    return plan_failed(d);
  }
  plan_done(d, keep);
}

// The same for the label-free index (see core.cuh): its plan keeps keys of lengths below lim, of which
// a core distance may take a quarter (checked at each sweep) and a bottom's chain another.
void core_build(Handle &h, DeviceState *d) {
  NvtxRange nvtx("qbc.core_plan");
  TraceScope trace("core plan");
  const Index &ix = h.host;
  tree_free(d);
  const int32_t n = ix.n;
  constexpr int bits = 5;
  static_assert(kBottomRows + 1 < (1 << bits) - 2, "entry index");
  constexpr uint32_t lim = 1u << (32 - bits);
  const int32_t lcap = (int32_t)(lim / (4 * kCoreChain));
  CoreShape s;
  if (!ix.arcs_paired) return;  // the elimination finds an arc's reverse; the sweep of the whole graph answers
  if (!core_shape(ix, s) || (int64_t)s.nc * 4 > (int64_t)n * 3) return;  // (a core that is most of the graph saves nothing)
  if ((size_t)core_words(s.nc) * 8 + 8192 > (size_t)d->smem_optin) return;  // its list bits are in shared memory
  for (size_t e = (size_t)s.xoff[s.nc]; e < s.eL.size(); e++)
    if (s.eL[e] > lcap) return;
  cudaStream_t st = d->s_label;
  auto p = new TreePlan();
  d->tree = p;
  bool keep = false;
  try {
    PlanScratch talloc(d);
    TreeArgs &a = p->args;
    const int64_t E = (int64_t)s.xtid.size(), E0 = s.xoff[s.nc];
    p->E = E;
    bottom_classes(p, s.bot);
    a.n = n;
    a.H = kCoreH;
    a.NT = s.nc;
    a.bits = bits;
    a.dist_lim = lim / 4;
    a.absent = ((lim / 10 * 7) << bits) | ((1u << bits) - 2u);
    p->arena_left = (size_t)n * (7 * 4 + 1 + 8) + s.bot.size() * 16 + (size_t)E * (8 + 4 + 4 + 4 + 16 + 24) +
                    (s.arc.size() * 2 + s.more.size()) * 16 + 64 * 256;
    p->arena = (char *)p->device(p->arena_left);
    a.xoff = p->upload(s.xoff, st);
    a.tidx_of = p->upload(s.tidx_of, st);
    a.bot = p->upload(s.bot, st);
    a.row_of = p->upload(s.row_of, st);
    a.depth = p->upload(s.depth, st);
    a.parent = p->upload(s.parent, st);
    a.send = p->upload(s.send, st);
    p->cid_of = p->upload(s.cid_of, st);
    int32_t *eC = p->upload(s.eC, st);
    CoreArgs &c = p->core;
    c.nc = s.nc;
    c.arc = p->upload(s.arc, st);
    c.info = p->upload(s.info, st);
    c.more = p->upload(s.more, st);
    c.E = E;
    c.max_rounds = 2 * s.nc + 16;
    while (((s.nc - 1) >> c.sort_shift) >= kCoreBuckets) c.sort_shift++;
    c.sort_buckets = ((s.nc - 1) >> c.sort_shift) + 1;
    int2 *ex = p->alloc<int2>((size_t)E);
    int4 *eup = p->alloc<int4>((size_t)E);
    int32_t *etr = p->alloc<int32_t>((size_t)E);
    p->owner = p->alloc<int32_t>((size_t)E);
    a.ex = ex;
    a.eC = eC;
    a.eup = eup;
    a.etr = etr;
    a.Bd = p->alloc<double>((size_t)E * 3 + (size_t)n);
    a.Bu = a.Bd + E;
    a.Bs = a.Bu + E;
    a.F = a.Bs + E;
    a.wrap = d->err + 1;
    CK(cudaMemsetAsync(a.wrap, 0, 4, st));
    int32_t *xtid = (int32_t *)talloc((size_t)E * 4), *eL = (int32_t *)talloc((size_t)E * 4);
    if (E > 0) {
      CK(cudaMemcpyAsync(xtid, s.xtid.data(), (size_t)E * 4, cudaMemcpyHostToDevice, st));
      CK(cudaMemcpyAsync(eL, s.eL.data(), (size_t)E * 4, cudaMemcpyHostToDevice, st));
      k_owner<<<blocks_for((int64_t)n * 32, 256), 256, 0, st>>>(a.xoff, n, p->owner);
      CK(cudaGetLastError());
      k_edge_refs<<<blocks_for((int64_t)n * 32, 256), 256, 0, st>>>(a.xoff, xtid, eL, a.depth, a.tidx_of, a.bot, a.row_of, n, bits,
                                                                  lcap, eC, ex, eup, etr);
      CK(cudaGetLastError());
    }
    keep = build_triangles(p, E0, E, xtid, eL, talloc, st);
    CK(cudaStreamSynchronize(st));  // the staging vectors die here
  } catch (...) {
    return plan_failed(d);
  }
  plan_done(d, keep);
}

// ------------------------------------------------------------------------------- launch
// device bytes of one group of sources
static size_t group_bytes(const TreePlan &p) {
  const TreeArgs &a = p.args;
  if (p.core.nc)  // sweep state, rows of D, S and J, rows of U and the seeds, source and waves
    return ((size_t)a.NT * (4 + 8 + 4 + 4 + 8) + (size_t)a.H * (4 + 4 + 8) + 8) * kGroup;
  return ((size_t)a.NT * (4 + 4 + 4 + 8) + (size_t)a.H * (4 + 4 + 8)) * kGroup;
}

// (piece, group) pairs from which a level is wide: below, the narrow kernels' shorter chain per piece
// counts, above, how many pieces an SM has in flight.  2, 12, 32 and 48 per SM: 1.69, 1.41, 1.43,
// 1.43 ms (50k vertices, 256 sources), 49.3, 49.5, 50.3, 56.6 ms (50k, all; an earlier state), 1.33,
// 1.36, 1.44, 1.73 ms (6k, all).
constexpr int64_t kWideCtas = 148 * 12;

// Groups of sources that the per-source scratch holds, at most kMaxGroups.
constexpr int kMaxGroups = 1024;  // (all sources of 50k in passes of 96 and 192 groups: 19 % and 5 % slower than of 264)
static int groups_fit(const DeviceState *d) {
  const size_t room = (size_t)d->chunk * d->n_pad * sizeof(int4);
  size_t fit = std::min<size_t>(kMaxGroups, room / group_bytes(*d->tree));
  if (d->tree->core.nc)  // the lists of a core vertex take the place of a vertex's
    fit = std::min<size_t>(fit, (size_t)d->chunk * d->n_pad / ((size_t)(d->tree->core.nc + 2) * kGroup));
  return (int)fit;
}

// (source, vertex) pairs from which the plan is the faster path.
//
// MHL: the tree's launches follow the trunk level by level, however few the sources (0.36, 0.43, 0.59, 0.85,
// 1.5 and 5.1 ms for a few sources of 2k, 6k, 21k, 50k, 120k and 500k vertices); the label kernels start
// lower on graphs up to 80k vertices and rise with the pairs.  Time of the tree over that of the label
// kernels, grids of three seeds, calls that wait for their result: 6k vertices 1.11 at 1.5M pairs, 1.10 at
// 2M, 0.97 at 2.75M, 0.91 at 3M; 21k 1.09 at 1.25M, 0.98 at 1.75M; 45k 1.17 at 0.4M, 1.06 at 1.25M, 0.95 at
// 1.5M; 70k 1.03 at 0.2M, 0.97 at 0.8M; 90k to 160k below 1 from the first source; 200k to 350k 0.93 to 1.12
// (1.05 on average) for one source, 0.95 for two.  The lines below join the sizes' crossings, which lie at 1.8M (1.5k), 2.1M (2k), 3.0M (4k),
// 2.7M (6k), 3.2M (8k), 2.4M (12k), 2.1M (16k), 1.8M (21k), 1.4M (30k to 60k) and 0.6M (70k).  (A line from
// 3.6M falling by 68 per vertex cost calls of 30k to 60k vertices up to a fifth.)
// Calls that only enqueue are followed by the guarded label launches: crossings at 2.0M (1.5k), 2.3M (2k),
// 3.4M (4k), 2.8M (6k), 3.4M (8k), 2.6M (12k), 2.3M (16k), 2.0M (21k).  (2M for all sizes: 333 sources of 6k
// 0.36 ms, by the label kernels 0.29.)  From 21k vertices on such calls often overlap with others, where the
// tree's chain has little to offer: 2M.
//
// H2H: the label path counts paths by Kahn waves and is slower from the first source on (1,023 vertices
// 0.194 against 0.241 ms, 20k 0.62 against 1.29).
//
// Label-free: the core from the first source on (one source of 100 vertices 0.163 against 0.177 ms, 400
// 0.19 and 0.27, 5k 0.37 and 0.76, 200k 2.8 and 7.2).
//
// QBC_TREE_MIN_PAIRS overrides all of it for tests.
static int64_t min_pairs(const Handle &h, bool rerun) {
  const char *e = std::getenv("QBC_TREE_MIN_PAIRS");
  if (e && *e) return std::strtoll(e, nullptr, 10);
  const int32_t n = h.host.n;
  if (h.host.kind == IndexKind::CSR) return 0;
  if (h.host.kind == IndexKind::H2H) return rerun ? 1000 : 1 << 20;
  struct Knot {
    int32_t n;
    int64_t pairs;
  };
  static constexpr Knot wait[] = {{0, 1300000}, {4000, 2900000}, {8000, 2900000}, {28000, 1400000}, {60000, 1300000}, {72000, 500000},
                                  {90000, 0}, {180000, 0},    {200000, 360000}};
  static constexpr Knot enqueue[] = {{0, 1600000}, {4000, 3200000}, {8000, 3200000}, {21000, 2 << 20}};
  auto at = [n](const Knot *k, int count) {
    int i = 1;
    while (i < count && k[i].n <= n) i++;
    if (i == count) return k[count - 1].pairs;
    return k[i - 1].pairs + (k[i].pairs - k[i - 1].pairs) * (n - k[i - 1].n) / (k[i].n - k[i - 1].n);
  };
  return rerun ? at(wait, 9) : at(enqueue, 4);
}

bool plan_open(const Handle &h, const DeviceState *d) {
  const Tuning &t = h.tuning;
  if (!d->tree || d->tree->off) return false;
  // a tuning that picks a label or dependency kernel, or the test hook of the label rows' copies, gets it
  if (!t.keep_plan && (t.lanes_per_source || t.split || t.dep_form || t.queue_depth || t.label_warps || t.label_tile ||
                       t.label_passes || t.label_sources || t.label_stream))
    return false;
  const char *hook = std::getenv("QBC_TEST_ROW_WAIT_SPINS");
  if (hook && *hook) return false;
  return groups_fit(d) >= 1;
}

bool use_tree(const Handle &h, const DeviceState *d, int32_t ns, bool rerun) {
  return ns >= 1 && (int64_t)ns * d->n >= min_pairs(h, rerun) && plan_open(h, d);
}

bool tree_source_rows(const DeviceState *d, const int32_t *src, int32_t ns, int32_t stride, int32_t *rows, cudaStream_t st) {
  if (!d->tree || d->tree->core.nc) return false;
  TreeArgs a = d->tree->args;
  a.src = src;
  a.ns = ns;
  k_source_rows<<<blocks_for((int64_t)ns * 32, 128), 128, 0, st>>>(a, stride, rows);
  CK(cudaGetLastError());
  return true;
}

const int32_t *tree_guard(const DeviceState *d) { return d->tree ? d->tree->args.wrap : nullptr; }

bool tree_disable(DeviceState *d) {
  if (!d->tree || d->tree->off) return false;
  d->tree->off = true;
  return true;
}

// The attribute belongs to the function, not to a launch, and other threads launch it for other
// indexes: every launch sets the same limit, the one that the plans are checked against.
template <class K>
static void allow_smem(K kernel, size_t bytes) {
  CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

// The kernel may, if early, start before the one ahead of it in the stream ends (see wait_before).
template <class... A, class... B>
static void launch_early(void (*kernel)(A...), bool early, dim3 grid, int threads, size_t smem, cudaStream_t st,
                         B... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = early ? 1 : 0;
  CK(cudaLaunchKernelEx(&c, kernel, static_cast<A>(args)...));
}

// The bottoms [first, end) of at most `rows` rows: the warps of a CTA share a bottom's edges, and a
// CTA takes more groups one after another while there are CTAs enough.
static void launch_bottom(const TreeArgs &a, bool early, int first, int end, int rows, cudaStream_t st) {
  const int warps = std::min(kBottomWarps, a.ng);
  int gpc = warps;
  while (gpc < 64 && (int64_t)(end - first) * ((a.ng + 2 * gpc - 1) / (2 * gpc)) >= 148 * 24) gpc *= 2;
  static_assert(kBottomWarps * kBottomRows * RowLayout::size <= 36 * 1024, "no opt-in for more than 48 KB");
  const size_t smem = (size_t)warps * rows * RowLayout::size;
  launch_early(k_bottom, early, dim3(end - first, (a.ng + gpc - 1) / gpc), warps * 32, smem, st, a, first, rows, gpc);
}

static void launch_bottoms(DeviceState *d, const TreeArgs &a, cudaStream_t st) {
  const TreePlan &p = *d->tree;
  if (a.ng > 4) {
    // A launch runs into the tail of the one before it: all sources of 2k vertices 0.444 -> 0.394 ms, 6k 6 %
    // less, 50k 2 %, a 5k core graph 3 %.  A large core has so many bottoms that
    // there is no tail to speak of, and the classes are better kept apart (200k + 2 %: 52.6 against 52.2 ms).
    const bool overlap = p.core.nc < kCoreSmall;
    for (const TreePlan::BotClass &c : p.bot_class) {
      launch_bottom(a, overlap && &c != &p.bot_class.front(), c.first, c.end, c.rows, st);
      CK(cudaGetLastError());
      d->launches++;
    }
  } else if (p.nbot) {
    launch_bottom(a, false, 0, p.nbot, p.bot_class[0].rows, st);
    CK(cudaGetLastError());
    d->launches++;
  }
}

// B over the triangles, into F
static void launch_unpack(DeviceState *d, cudaStream_t st) {
  const TreePlan &p = *d->tree;
  const TreeArgs &a = p.args;
  auto launched = [&] {
    CK(cudaGetLastError());
    d->launches++;
  };
  if (p.E > 0) {
    k_fold<<<blocks_for(p.E, 256), 256, 0, st>>>(p.E, a.eup, p.owner, a.Bd, a.Bu, a.Bs, a.F, a.wrap);
    launched();
  }
  const int top = (int)p.tri_first.size() - 1;
  for (int l = 0; l < p.tail_level; l++) {
    const int64_t b = p.tri_first[l], c = p.tri_first[l + 1] - b;
    k_unpack<<<blocks_for(c, 256), 256, 0, st>>>(p.tri + b, c, a.eC, a.Bd, a.F, a.wrap);
    launched();
  }
  if (p.tail_level < top) {
    k_unpack_tail<<<kTailCtas, 1024, 0, st>>>(p.tri, p.tri_at, p.tail_level, top, a.eC, a.Bd, a.F, a.wrap);
    launched();
  }
}

// Threads per CTA of the core's sweep and dependencies; 2,048 per SM in any case.
static int core_threads(const Handle &h, int ns, int nc) {
  const int t = h.tuning.sweep_threads;
  if (t) return t == 2048 ? 512 : t;
  if (ns <= 148 * 2 || nc >= kCoreLarge) return 1024;
  return ns > 148 * 4 && nc < kCoreSmall ? 256 : 512;
}
struct CoreKernels {
  void (*sweep)(TreeArgs, CoreArgs), (*dep)(TreeArgs, CoreArgs);
};
static CoreKernels core_kernels(int threads) {
  switch (threads) {
    case 256: return {k_core_sweep<256, 8>, k_core_dep<256, 8>};
    case 512: return {k_core_sweep<512, 4>, k_core_dep<512, 4>};
    default: return {k_core_sweep<1024, 2>, k_core_dep<1024, 2>};
  }
}

// The label-free index: sweeps over the core, bottoms, dependencies over the core (see core.cuh).
static void launch_core(const Handle &h, DeviceState *d, const int32_t *d_src_tid, int32_t ns, cudaStream_t st) {
  TreePlan &p = *d->tree;
  const int32_t nc = p.core.nc;
  CK(cudaMemsetAsync(p.args.Bd, 0, ((size_t)p.E * 3 + (size_t)p.args.n) * 8, st));
  auto launched = [&] {
    CK(cudaGetLastError());
    d->launches++;
  };
  const int groups = (ns + kGroup - 1) / kGroup, passes = (groups + groups_fit(d) - 1) / groups_fit(d);
  const int fit = (groups + passes - 1) / passes;
  std::pair<cudaEvent_t, cudaEvent_t> ev{};
  for (int32_t off = 0; off < ns; off += fit * kGroup) {
    TreeArgs a = p.args;
    CoreArgs c = p.core;
    a.ns = std::min(fit * kGroup, ns - off);
    a.ng = (a.ns + kGroup - 1) / kGroup;
    const size_t slots = (size_t)a.ng * kGroup, nt = slots * nc, nu = slots * a.H;
    char *w = reinterpret_cast<char *>(d->rec[0]);
    auto take = [&](size_t bytes) {
      char *q = w;
      w += bytes;
      return q;
    };
    c.word = (unsigned long long *)take(nt * 8);
    a.J = (double *)take(nt * 8);
    a.seed = (double *)take(nu * 8);
    a.D = (uint32_t *)take(nt * 4);
    a.S = (uint32_t *)take(nt * 4);
    a.Ud = (int32_t *)take(nu * 4);
    a.Uc = (uint32_t *)take(nu * 4);
    int32_t *cid = (int32_t *)take(slots * 4);
    c.waves = (int32_t *)take(slots * 4);
    c.dist = (int32_t *)take(nt * 4);
    a.src = cid;
    c.hop = d->hop[0];
    c.order = d->order[0];
    c.lcnt = d->lcnt[0];
    c.delta = sweep_delta(h, d) * kCoreDelta;
    const int threads = core_threads(h, a.ns, nc);
    const CoreKernels kernels = core_kernels(threads);
    const size_t smem = (size_t)core_words(nc) * 8;
    allow_smem(kernels.sweep, (size_t)d->smem_optin - 8192);
    if (d->profiling) {
      ev = take_events(d->ev_lab, d->ev_lab_used);
      CK(cudaEventRecord(ev.first, st));
    }
    k_core_src<<<blocks_for(a.ns, 256), 256, 0, st>>>(d_src_tid + off, p.cid_of, a.ns, cid);
    launched();
    k_core_up<<<(unsigned)(slots / 4), 128, 0, st>>>(a);
    launched();
    kernels.sweep<<<a.ns, threads, smem, st>>>(a, c);
    launched();
    k_core_rows<<<dim3((nc + 31) / 32, a.ng), 256, 0, st>>>(a, c);
    launched();
    launch_bottoms(d, a, st);
    if (d->profiling) {
      CK(cudaEventRecord(ev.second, st));
      ev = take_events(d->ev_dp, d->ev_dp_used);
      CK(cudaEventRecord(ev.first, st));
    }
    kernels.dep<<<a.ns, threads, 0, st>>>(a, c);
    launched();
    k_core_back<<<blocks_for(a.ns, 4), 128, 0, st>>>(a, c);
    launched();
    if (d->profiling) CK(cudaEventRecord(ev.second, st));
    d->label_launches++;
    d->dep_launches++;
  }
  launch_unpack(d, st);
  k_core_finish<<<blocks_for(p.args.n, 256), 256, 0, st>>>(p.args.F, p.cid_of, d->bc_tid, p.args.n, d->err);
  launched();
}

void launch_tree(const Handle &h, DeviceState *d, const int32_t *d_src_tid, int32_t ns, cudaStream_t st) {
  if (d->tree->core.nc) return launch_core(h, d, d_src_tid, ns, st);
  TreePlan &p = *d->tree;
  CK(cudaMemsetAsync(p.args.Bd, 0, ((size_t)p.E * 3 + (size_t)p.args.n) * 8, st));
  auto launched = [&] {
    CK(cudaGetLastError());
    d->launches++;
  };
  // passes of equal size
  const int groups = (ns + kGroup - 1) / kGroup, passes = (groups + groups_fit(d) - 1) / groups_fit(d);
  const int fit = (groups + passes - 1) / passes;
  const int levels = (int)p.level_class.size() / 4;
  std::pair<cudaEvent_t, cudaEvent_t> ev{};
  for (int32_t off = 0; off < ns; off += fit * kGroup) {
    TreeArgs a = p.args;
    a.src = d_src_tid + off;
    a.ns = std::min(fit * kGroup, ns - off);
    a.ng = (a.ns + kGroup - 1) / kGroup;
    const size_t nt = (size_t)a.ng * a.NT * kGroup, nu = (size_t)a.ng * a.H * kGroup;
    char *w = reinterpret_cast<char *>(d->rec[0]);
    auto take = [&](size_t bytes) {
      char *q = w;
      w += bytes;
      return q;
    };
    a.J = (double *)take(nt * 8);
    a.seed = (double *)take(nu * 8);
    a.D = (uint32_t *)take(nt * 4);
    a.S = (uint32_t *)take(nt * 4);
    a.Ud = (int32_t *)take(nu * 4);
    a.Uc = (uint32_t *)take(nu * 4);
    a.arg = (uint32_t *)take(nt * 4);
    if (d->profiling) {
      ev = take_events(d->ev_lab, d->ev_lab_used);
      CK(cudaEventRecord(ev.first, st));
    }
    if (a.lab_ch) {
      const int tiles = (a.H + 31) / 32;
      k_up_gather<<<dim3(a.ng, std::max(1, std::min(tiles, 148 * 4 / a.ng))), 1024, 0, st>>>(a);
      launched();
    } else {
      const size_t smem = (size_t)p.up_warps * a.H * 8;
      allow_smem(k_up_rows, (size_t)d->smem_optin - 2048);
      k_up_rows<<<(a.ng * kGroup + p.up_warps - 1) / p.up_warps, p.up_warps * 32, smem, st>>>(a);
      launched();
    }
    for (int l = 0; l < levels; l++) {
      const int32_t *c = p.level_class.data() + 4 * l;
      if ((int64_t)(c[3] - c[0]) * a.ng < kWideCtas) {
        launch_early(k_trunk_down_narrow, l > 0, dim3(c[3] - c[0], a.ng), kPieceLen * 32, 0, st, a, c[0]);
        launched();
        continue;
      }
      if (c[1] > c[0]) {
        k_trunk_down<32><<<dim3(c[1] - c[0], a.ng), Wide<32>::warps * 32, 0, st>>>(a, c[0]);
        launched();
      }
      if (c[2] > c[1]) {
        k_trunk_down<16><<<dim3(c[2] - c[1], a.ng), Wide<16>::warps * 32, 0, st>>>(a, c[1]);
        launched();
      }
      if (c[3] > c[2]) {
        k_trunk_down<8><<<dim3(c[3] - c[2], a.ng), Wide<8>::warps * 32, 0, st>>>(a, c[2]);
        launched();
      }
    }
    launch_bottoms(d, a, st);
    if (d->profiling) {
      CK(cudaEventRecord(ev.second, st));
      ev = take_events(d->ev_dp, d->ev_dp_used);
      CK(cudaEventRecord(ev.first, st));
    }
    for (int l = levels - 1; l >= 0; l--) {
      const int32_t *c = p.level_class.data() + 4 * l;
      if ((int64_t)(c[3] - c[0]) * a.ng < kWideCtas) {
        launch_early(k_trunk_up_narrow, l < levels - 1, dim3(c[3] - c[0], a.ng), kPieceLen * 32, 0, st, a, c[0]);
        launched();
        continue;
      }
      if (c[1] > c[0]) {
        k_trunk_up<32><<<dim3(c[1] - c[0], a.ng), Wide<32>::warps * 32, 0, st>>>(a, c[0]);
        launched();
      }
      if (c[2] > c[1]) {
        k_trunk_up<16><<<dim3(c[2] - c[1], a.ng), Wide<16>::warps * 32, 0, st>>>(a, c[1]);
        launched();
      }
      if (c[3] > c[2]) {
        k_trunk_up<8><<<dim3(c[3] - c[2], a.ng), Wide<8>::warps * 32, 0, st>>>(a, c[2]);
        launched();
      }
    }
    {
      const size_t smem = (size_t)a.H * 20;
      auto kern = a.ns >= 148 * 8 ? k_up_back<4> : k_up_back<8>;
      allow_smem(kern, (size_t)d->smem_optin - 2048 - sizeof(BackShared<8>));
      kern<<<a.ns, a.ns >= 148 * 8 ? 128 : 256, smem, st>>>(a);
      launched();
    }
    if (d->profiling) CK(cudaEventRecord(ev.second, st));
    d->label_launches++;
    d->dep_launches++;
  }
  launch_unpack(d, st);
  k_finish<<<std::min(148 * 4, (p.args.n + 255) / 256), 256, 0, st>>>(p.args.F, d->bc_tid, p.args.n, d->err);
  launched();
}

}  // namespace qbc
