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
// kernels leave their results unused, and the call is answered by the label kernels.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdlib>

#include "device_state.h"

namespace qbc {

namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr unsigned kNoKey = 0xffffffffu;
constexpr int kGroup = 64;           // sources a warp takes: two neighbouring ones per lane
constexpr int kPieceLen = 32;        // trunk vertices per piece
constexpr int kBottomRows = 32;      // shared-memory rows of a bottom subtree (its separator + its vertices)
constexpr int kBottomEdges = 160;    // ... and its edges (grids of 2k to 1M vertices: at most 100)
constexpr int kInPieceEdges = kPieceLen * (kPieceLen - 1) / 2;
constexpr int kMaxUnpackLevels = 1024;

struct TreeArgs {
  int n, H, NT, bits;
  unsigned dist_lim;               // distances of shortest paths are below it
  const int32_t *xoff;             // [n + 1] edge range of a vertex
  const int2 *ex;                  // per edge (x: trunk index or bottom row, (L << bits) | (i + 1))
  const int4 *eup;                 // per edge (depth(x) - 1, L, path count, tid of x)
  const int32_t *eC;               // per edge path count
  const int32_t *etr;              // per edge trunk index of x (separators of bottom roots)
  const int4 *tmeta;               // per trunk vertex (first edge, end edge, edges inside its piece, tid)
  const int2 *tsub;                // per trunk vertex (subtree end, depth - 1)
  const int4 *piece;               // (first trunk index, end, trunk index of the parent or -1, 0)
  const int32_t *piece_of;         // per trunk vertex
  const int32_t *tidx_of;          // per tid: trunk index, or -1 - bottom
  const int4 *bot;                 // bottoms: (root tid, size, separator size, 0)
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
__device__ __forceinline__ void key_min(unsigned &m1, unsigned &m2, unsigned v, unsigned mask) {
  m1 = min(m1, v);
  m2 = min(m2, v ^ mask);
}
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

// Reverse of the U rows, a CTA per source, root first: the flow of y is its seed plus its share of the
// flow of the separator entries x with U(y) + L = U(x).  Each warp takes a block of 32 ancestors and
// collects the entries that hold (independent loads, the next ancestor's in flight); one warp then
// applies the blocks in order in shared memory, and all add the shortcuts' flow.
constexpr int kBackWarps = 8;
constexpr int kBackHits = 192;  // entries collected per block; a block with more is done by one warp in turns
struct BackShared {
  int2 hit[kBackWarps][kBackHits];  // (edge, x's depth | y's depth << 16)
  double ratio[kBackWarps][kBackHits];
  int count[kBackWarps];
};

__global__ void __launch_bounds__(kBackWarps * 32) k_up_back(TreeArgs a) {
  extern __shared__ double sm_back[];
  __shared__ BackShared sh;
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
  if (warp == 0) {
    int j = h - 1, y = s, i = a.tidx_of[y];
    while (i < 0 && j >= 0) {
      if (lane == 0) path[j] = -1 - y;
      j--;
      y = a.parent[y];
      i = y >= 0 ? a.tidx_of[y] : 0;
    }
    while (j >= 0) {
      const int4 pc = a.piece[a.piece_of[i]];
      const int cnt = i - pc.x + 1;
      if (lane < cnt) path[j - (cnt - 1) + lane] = pc.x + lane;
      j -= cnt;
      i = pc.z;
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
  for (int r0 = 0; r0 < h; r0 += kBackWarps * 32) {
    const int q0 = r0 + warp * 32;
    int done = 32;
    if (q0 < h) done = collect(warp, q0, 0);
    else if (lane == 0) sh.count[warp] = 0;
    const bool crowded = __syncthreads_or(done < 32);
    if (!crowded) {
      if (warp == 0)
        for (int w = 0; w < kBackWarps; w++) apply(w);
      __syncthreads();
      add(warp, lane, 32);
    } else if (warp == 0) {  // more entries than the lists hold: one warp, list by list
      for (int w = 0; w < kBackWarps; w++)
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

// ------------------------------------------------------------------------------- trunk down
// A CTA takes one piece (a path of at most 32 trunk vertices) for one group.  The minima over the
// separator vertices above the piece are independent, a warp per vertex (or part of its list); then
// one warp follows the path in shared memory.  Bound by the latency of those steps (5 M warp
// instructions in 18 us per 10k list entries and 64 groups at 50k): two groups per CTA, whose 114
// registers left 16 warps per SM, took 1,602 against 1,005 us for the seven wide levels.
struct PieceShared {
  int2 ine[kInPieceEdges];  // edges inside the piece: (kGroup * position, key)
  int ineC[kInPieceEdges];
  int inoff[kPieceLen + 1];
  int4 meta[kPieceLen];
  int2 sub[kPieceLen];
};

__device__ __forceinline__ void load_piece(const TreeArgs &a, int start, int len, PieceShared &p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (warp == 0) {
    const int4 m = lane < len ? a.tmeta[start + lane] : make_int4(0, 0, 0, 0);
    p.meta[lane] = m;
    if (lane < len) p.sub[lane] = a.tsub[start + lane];
    int x = m.z;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int z = __shfl_up_sync(kAll, x, o);
      if (lane >= o) x += z;
    }
    p.inoff[lane] = x - m.z;
    if (lane == 31) p.inoff[32] = x;
  }
  __syncthreads();
  for (int i = warp; i < len; i += nw) {
    const int4 m = p.meta[i];
    if (lane < m.z) {  // at most 31 edges
      const int2 v = a.ex[m.y - m.z + lane];
      p.ine[p.inoff[i] + lane] = make_int2((v.x - start) * kGroup, v.y);
      p.ineC[p.inoff[i] + lane] = a.eC[m.y - m.z + lane];
    }
  }
}

template <int GB>
__global__ void __launch_bounds__(512) k_trunk_down(TreeArgs a, int piece0, int pl) {
  extern __shared__ uint32_t sm_td[];
  __shared__ PieceShared p;
  constexpr int K = 2 * GB, E = 8 / GB;  // values per lane, edges loaded together
  if (__syncthreads_or(wrapped(a))) return;
  const int4 pc = a.piece[piece0 + blockIdx.x];
  const int start = pc.x, len = pc.y - pc.x;
  const int g0 = blockIdx.y * GB;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const unsigned mask = (1u << a.bits) - 1u;
  const int parts = max(1, min(8, nw / len));  // few vertices: several warps share a list
  const int gs = pl * kGroup;                  // a group's values in shared memory
  uint32_t *k1 = sm_td + 2 * lane, *k2 = k1 + GB * gs, *sg = k2 + GB * gs;
  if (parts > 1)
    for (int q = threadIdx.x; q < 2 * GB * gs; q += blockDim.x) sm_td[q] = kNoKey;
  int s[K];
  size_t gt[GB], gu[GB];  // this lane's place in a group's trunk and U rows (a missing group repeats the last)
#pragma unroll
  for (int w = 0; w < GB; w++) {
    const int g = min(g0 + w, a.ng - 1);
    bool live[2];
    int sw[2];
    lane_sources(a, g, lane, sw, live);
    s[2 * w] = sw[0];
    s[2 * w + 1] = sw[1];
    gt[w] = (size_t)g * a.NT * kGroup + 2 * lane;
    gu[w] = (size_t)g * a.H * kGroup + 2 * lane;
  }
  load_piece(a, start, len, p);
  __syncthreads();
  for (int task = warp; task < len * parts; task += nw) {
    const int i = task / parts, part = task - i * parts;
    const int4 m = p.meta[i];
    unsigned m1[K], m2[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const int2 sub = p.sub[i];
      m1[k] = up_key(a, part == 0 && m.w <= s[k] && s[k] < sub.x, gu[k >> 1] + (size_t)sub.y * kGroup + (k & 1));
      m2[k] = m1[k] == kNoKey ? kNoKey : m1[k] ^ mask;
    }
    const int nx = m.y - m.z - m.x, per = ((nx + parts - 1) / parts + 7) & ~7;
    const int ee = m.x + min(nx, (part + 1) * per);
    for (int e = m.x + min(nx, part * per); e < ee; e += E) {  // (the last entry may repeat)
      int2 v[E];
      uint2 d[E][GB];
#pragma unroll
      for (int q = 0; q < E; q++) v[q] = __ldg(a.ex + min(e + q, ee - 1));
#pragma unroll
      for (int q = 0; q < E; q++)
#pragma unroll
        for (int w = 0; w < GB; w++) d[q][w] = *reinterpret_cast<const uint2 *>(a.D + gt[w] + (size_t)v[q].x * kGroup);
#pragma unroll
      for (int q = 0; q < E; q += 2)
#pragma unroll
        for (int w = 0; w < GB; w++) {
          key_min2(m1[2 * w], m2[2 * w], d[q][w].x + (unsigned)v[q].y, d[q + 1][w].x + (unsigned)v[q + 1].y, mask);
          key_min2(m1[2 * w + 1], m2[2 * w + 1], d[q][w].y + (unsigned)v[q].y, d[q + 1][w].y + (unsigned)v[q + 1].y, mask);
        }
    }
#pragma unroll
    for (int w = 0; w < GB; w++) {
      const int o = w * gs + i * kGroup;
      if (parts > 1) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
          atomicMin(k1 + o + k, m1[2 * w + k]);
          atomicMin(k2 + o + k, m2[2 * w + k]);
        }
      } else {
        *reinterpret_cast<uint2 *>(k1 + o) = make_uint2(m1[2 * w], m1[2 * w + 1]);
        *reinterpret_cast<uint2 *>(k2 + o) = make_uint2(m2[2 * w], m2[2 * w + 1]);
      }
    }
  }
  __syncthreads();
  // along the piece, a warp per group: k1 becomes the distance, k2 the argument
  if (warp < GB) {
    uint32_t *r1 = k1 + warp * gs, *r2 = k2 + warp * gs;
    for (int i = 0; i < len; i++) {
      uint2 m1 = *reinterpret_cast<uint2 *>(r1 + i * kGroup), m2 = *reinterpret_cast<uint2 *>(r2 + i * kGroup);
#pragma unroll 4
      for (int k = p.inoff[i]; k < p.inoff[i + 1]; k++) {
        const int2 v = p.ine[k];
        const uint2 d = *reinterpret_cast<uint2 *>(r1 + v.x);
        key_min(m1.x, m2.x, d.x + (unsigned)v.y, mask);
        key_min(m1.y, m2.y, d.y + (unsigned)v.y, mask);
      }
      *reinterpret_cast<uint2 *>(r1 + i * kGroup) = make_uint2(m1.x & ~mask, m1.y & ~mask);
      *reinterpret_cast<uint2 *>(r2 + i * kGroup) = make_uint2((m1.x & mask) | (((m2.x & mask) ^ mask) << 16),
                                                               (m1.y & mask) | (((m2.y & mask) ^ mask) << 16));
    }
  }
  __syncthreads();
  // counts from above the piece, and how many entries reach a minimum that several do
  for (int i = warp; i < len; i += nw) {
    const int4 m = p.meta[i];
    const int nx = m.y - m.z - m.x;
    unsigned long long c[K];
    int a1[K], a2[K];
    bool tie = false;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const unsigned ar = k2[(k >> 1) * gs + i * kGroup + (k & 1)];
      a1[k] = (int)(ar & 0xffff);
      a2[k] = (int)(ar >> 16);
      tie |= a1[k] != a2[k];
      const int e = m.x + max(a1[k], 1) - 1;
      c[k] = 0;
      if (a1[k] == 0) c[k] = a.Uc[gu[k >> 1] + (size_t)p.sub[i].y * kGroup + (k & 1)];
      else if (a1[k] <= nx) c[k] = (unsigned long long)(unsigned)a.eC[e] * a.S[gt[k >> 1] + (size_t)a.ex[e].x * kGroup + (k & 1)];
    }
    if (__any_sync(kAll, tie)) {
#pragma unroll
      for (int k = 0; k < K; k++) {
        const bool tk = a1[k] != a2[k];
        if (!__any_sync(kAll, tk)) continue;
        uint32_t *r1 = k1 + (k >> 1) * gs + (k & 1);
        const unsigned dt = r1[i * kGroup];
        int hits = a1[k] == 0;
        unsigned long long cc = hits ? c[k] : 0;  // every entry above the piece that reaches the minimum
        for (int e = m.x; e < m.x + nx; e += 8) {
          int2 v[8];
          unsigned d[8];
#pragma unroll
          for (int q = 0; q < 8; q++) v[q] = __ldg(a.ex + min(e + q, m.x + nx - 1));
#pragma unroll
          for (int q = 0; q < 8; q++) d[q] = a.D[gt[k >> 1] + (size_t)v[q].x * kGroup + (k & 1)];
#pragma unroll
          for (int q = 0; q < 8; q++)
            if (tk && e + q < m.x + nx && d[q] + ((unsigned)v[q].y & ~mask) == dt) {
              hits++;
              cc = count_of(a, cc + (unsigned long long)(unsigned)a.eC[e + q] * a.S[gt[k >> 1] + (size_t)v[q].x * kGroup + (k & 1)]);
            }
        }
        for (int q = p.inoff[i]; q < p.inoff[i + 1]; q++)
          hits += tk && r1[p.ine[q].x] + ((unsigned)p.ine[q].y & ~mask) == dt;
        if (tk) {
          c[k] = cc;
          if (hits > 2) k2[(k >> 1) * gs + i * kGroup + (k & 1)] = (unsigned)a2[k] | ((unsigned)a1[k] << 16);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < K; k++) sg[(k >> 1) * gs + i * kGroup + (k & 1)] = count_of(a, c[k]);
  }
  __syncthreads();
  // counts from inside the piece, along it
  if (warp < GB) {
    uint32_t *r1 = k1 + warp * gs, *r2 = k2 + warp * gs, *rs = sg + warp * gs;
    for (int i = 1; i < len; i++) {
      const int4 m = p.meta[i];
      const int nx = m.y - m.z - m.x, in0 = p.inoff[i] - 1 - nx;
      const uint2 ar = *reinterpret_cast<uint2 *>(r2 + i * kGroup);
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int a1 = (int)((k ? ar.y : ar.x) & 0xffff), a2 = (int)((k ? ar.y : ar.x) >> 16);
        if (max(a1, a2) <= nx) continue;
        unsigned long long c = rs[i * kGroup + k];
        if (a1 <= a2) {
          if (a1 > nx) c += (unsigned long long)(unsigned)p.ineC[in0 + a1] * rs[p.ine[in0 + a1].x + k];
          if (a2 > nx && a1 != a2) c += (unsigned long long)(unsigned)p.ineC[in0 + a2] * rs[p.ine[in0 + a2].x + k];
        } else {
          const unsigned dt = r1[i * kGroup + k];
          for (int q = p.inoff[i]; q < p.inoff[i + 1]; q++)
            if (r1[p.ine[q].x + k] + ((unsigned)p.ine[q].y & ~mask) == dt)
              c = count_of(a, c + (unsigned long long)(unsigned)p.ineC[q] * rs[p.ine[q].x + k]);
        }
        rs[i * kGroup + k] = count_of(a, c);
      }
    }
  }
  __syncthreads();
  for (int task = warp; task < len * GB; task += nw) {
    const int w = task / len, i = task - w * len;
    if (g0 + w >= a.ng) break;
    const size_t o = ((size_t)(g0 + w) * a.NT + start + i) * kGroup + 2 * lane;
    const int q = w * gs + i * kGroup;
    *reinterpret_cast<uint2 *>(a.D + o) = *reinterpret_cast<uint2 *>(k1 + q);
    *reinterpret_cast<uint2 *>(a.S + o) = *reinterpret_cast<uint2 *>(sg + q);
    *reinterpret_cast<uint2 *>(a.arg + o) = *reinterpret_cast<uint2 *>(k2 + q);
    *reinterpret_cast<double2 *>(a.J + o) = make_double2(0.0, 0.0);
  }
}

// ------------------------------------------------------------------------------- trunk up
template <int GB>
__global__ void __launch_bounds__(512) k_trunk_up(TreeArgs a, int piece0, int pl) {
  extern __shared__ double sm_tu[];
  __shared__ PieceShared p;
  constexpr int K = 2 * GB;
  const unsigned mask = (1u << a.bits) - 1u;
  if (__syncthreads_or(wrapped(a))) return;
  const int4 pc = a.piece[piece0 + blockIdx.x];
  const int start = pc.x, len = pc.y - pc.x;
  const int g0 = blockIdx.y * GB;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int gs = pl * kGroup;
  double *sf = sm_tu + 2 * lane;  // flow of a vertex: delta + 1 (delta for the source itself)
  uint32_t *sa = reinterpret_cast<uint32_t *>(sm_tu + GB * gs) + 2 * lane;
  int s[K], si[K];
  bool live[K];
  size_t gt[GB], gu[GB];
#pragma unroll
  for (int w = 0; w < GB; w++) {
    const int g = min(g0 + w, a.ng - 1);
    bool lw[2];
    int sw[2];
    lane_sources(a, g, lane, sw, lw);
#pragma unroll
    for (int k = 0; k < 2; k++) {
      s[2 * w + k] = sw[k];
      live[2 * w + k] = lw[k] && g0 + w < a.ng;
      si[2 * w + k] = a.tidx_of[sw[k]];
    }
    gt[w] = (size_t)g * a.NT * kGroup + 2 * lane;
    gu[w] = (size_t)g * a.H * kGroup + 2 * lane;
  }
  load_piece(a, start, len, p);
  __syncthreads();
  for (int i = warp; i < len; i += nw) {
    const int t = p.meta[i].w;
#pragma unroll
    for (int w = 0; w < GB; w++) {
      const size_t o = gt[w] + (size_t)(start + i) * kGroup;
      const double2 j = __ldcg(reinterpret_cast<const double2 *>(a.J + o));
      const uint2 ar = *reinterpret_cast<const uint2 *>(a.arg + o);
      const bool l0 = live[2 * w], l1 = live[2 * w + 1];
      // a lane without a source has no flow and no argument
      *reinterpret_cast<double2 *>(sf + w * gs + i * kGroup) =
          make_double2(l0 ? j.x + (t != s[2 * w] ? 1.0 : 0.0) : 0.0, l1 ? j.y + (t != s[2 * w + 1] ? 1.0 : 0.0) : 0.0);
      *reinterpret_cast<uint2 *>(sa + w * gs + i * kGroup) = make_uint2(l0 ? ar.x : 0u, l1 ? ar.y : 0u);
    }
  }
  __syncthreads();
  // what is handed on inside the piece, a warp per group, deepest vertex first
  if (warp < GB) {
    double *rf = sf + warp * gs;
    const uint32_t *ra = sa + warp * gs;
    for (int i = len - 1; i > 0; i--) {
      const int4 m = p.meta[i];
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
        } else {
          const size_t gp = ((size_t)(g0 + warp) * a.NT + start) * kGroup + 2 * lane + k;
          const uint32_t st = a.S[gp + (size_t)i * kGroup];
          const unsigned dt = a.D[gp + (size_t)i * kGroup];
          for (int q = p.inoff[i]; q < p.inoff[i + 1]; q++) {
            const int x = p.ine[q].x;
            const bool hit = a1 < a2 ? q == in0 + a1 || q == in0 + a2 : a.D[gp + x] + ((unsigned)p.ine[q].y & ~mask) == dt;
            if (hit) rf[x + k] += share(p.ineC[q], a.S[gp + x], st) * f;
          }
        }
      }
    }
  }
  __syncthreads();
  // everything else of a vertex, a warp with all the CTA's sources
  for (int i = warp; i < len; i += nw) {
    const int4 m = p.meta[i];
    const int2 sub = p.sub[i];
    const int nx = m.y - m.z - m.x;
    int a1[K], a2[K], one[K];
    double f[K];
    bool tie = false;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const unsigned ar = sa[(k >> 1) * gs + i * kGroup + (k & 1)];
      a1[k] = (int)(ar & 0xffff);
      a2[k] = (int)(ar >> 16);
      f[k] = sf[(k >> 1) * gs + i * kGroup + (k & 1)];
      tie |= a1[k] != a2[k];
      one[k] = a1[k] == a2[k] ? a1[k] : 0;
    }
#pragma unroll
    for (int k = 0; k < K; k++)
      if (live[k] && m.w <= s[k] && s[k] < sub.x) {
        const size_t u = gu[k >> 1] + (size_t)sub.y * kGroup + (k & 1);
        const int lo = min(a1[k], a2[k]);
        a.seed[u] = lo != 0 ? 0.0 : a1[k] == a2[k] ? f[k] : f[k] * share(1, a.Uc[u], a.S[gt[k >> 1] + (size_t)(start + i) * kGroup + (k & 1)]);
      }
    int xi[K];
#pragma unroll
    for (int k = 0; k < K; k++) xi[k] = one[k] > 0 ? a.ex[m.x + one[k] - 1].x : INT_MIN;
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (one[k] > 0 && one[k] <= nx) atomicAdd(a.J + gt[k >> 1] + (size_t)xi[k] * kGroup + (k & 1), f[k]);
      if (xi[k] == si[k]) {  // flow into the lane's own source counts apart
        atomicAdd(a.Bs + m.x + one[k] - 1, f[k]);
        one[k] = 0;
      }
    }
    add_flows<K>(a, m.x, one, f);
    if (__any_sync(kAll, tie)) {
#pragma unroll
      for (int k = 0; k < K; k++) {
        if (a1[k] == a2[k]) continue;
        const size_t gk = gt[k >> 1] + (k & 1);
        const uint32_t st = a.S[gk + (size_t)(start + i) * kGroup];
        const unsigned dt = a.D[gk + (size_t)(start + i) * kGroup];
        auto use = [&](int idx) {
          const int e = m.x + idx - 1, x = a.ex[e].x;
          const double w = f[k] * share(a.eC[e], a.S[gk + (size_t)x * kGroup], st);
          if (idx <= nx) atomicAdd(a.J + gk + (size_t)x * kGroup, w);
          atomicAdd((x == si[k] ? a.Bs : a.Bd) + e, w);
        };
        if (a1[k] < a2[k]) {
          if (a1[k] > 0) use(a1[k]);
          use(a2[k]);
        } else {  // more than two entries
          for (int e = m.x; e < m.y; e++) {
            const int2 v = a.ex[e];
            if (a.D[gk + (size_t)v.x * kGroup] + ((unsigned)v.y & ~mask) == dt) use(e - m.x + 1);
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------- bottoms
// A whole subtree below the trunk for a group at a time in a warp's shared memory: rows
// 0..b-1 are the root's separator (trunk vertices), then the subtree in preorder.  Down then up, so
// nothing of the subtree is written to global memory.  Distances are kept shifted (a key without its
// index), and an entry's index in the keys is its row + 1 (0: U), so the row a lane's paths come from
// needs no lookup.  On the way up most vertices hand everything to one entry in all lanes (at 50k 1.1
// to 1.3 different entries per vertex and warp): that entry's flow stays in the finished row and is
// summed after the pass, eight rows at a time, instead of by a warp-wide sum per vertex.
//
// The pass is bound by instruction issue, so shared memory is addressed by 32-bit offsets (ld.shared
// / st.shared); a row's block holds delta (f64), distance, count and argument of the warp's sources.
constexpr int kTieCode = 0xff, kSkipCode = 0xfe;  // arguments that are no row: a tie, a lane without a source
constexpr int kBottomPairs = (kBottomEdges + kBottomRows) / 2 + 1;
constexpr int kBottomWarps = 2;
constexpr int kLeadFull = 1 << 16;  // deferred sum: every lane, the rows' delta + 1 each

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

__global__ void __launch_bounds__(kBottomWarps * 32) k_bottom(TreeArgs a, int first, int rows, int gpc, unsigned absent) {
  extern __shared__ int4 sm_b[];
  using R = RowLayout;
  constexpr int SPL = 2;
  __shared__ int4 ep[kBottomPairs];           // two edges: (x row offset, key) twice
  __shared__ int2 er[kBottomEdges];           // an edge: (x row + 1, count)
  __shared__ int4 vt[kBottomRows + 1];        // a vertex: (address of its first pair, end, first edge | edges << 16, depth - 1 | counts above 1 << 31)
  __shared__ int vs[kBottomRows], sep[kBottomRows];  // subtree end, trunk index
  __shared__ uint8_t emap[kBottomRows][kBottomRows + 4];  // edge of (vertex, x row)
  if (__syncthreads_or(wrapped(a))) return;
  const int4 bt = a.bot[first + blockIdx.x];
  const int r = bt.x, m = bt.y, b = bt.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int ebase = a.xoff[r];
  const uint32_t ep0 = (uint32_t)__cvta_generic_to_shared(ep), vt0 = (uint32_t)__cvta_generic_to_shared(vt);
  if (warp == 0) {
    const int e0 = lane < m ? a.xoff[r + lane] - ebase : 0, k = lane < m ? a.xoff[r + lane + 1] - ebase - e0 : 0;
    const int pairs = lane < m ? max(1, (k + 1) >> 1) : 0;  // (the tree's root has no entries: one absent pair)
    int x = pairs;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int z = __shfl_up_sync(kAll, x, o);
      if (lane >= o) x += z;
    }
    if (lane < m)
      vt[lane] = make_int4((int)ep0 + 16 * (x - pairs), (int)ep0 + 16 * x, e0 | (k << 16), a.depth[r + lane] - 1);
    if (lane == 0) vt[m] = make_int4((int)ep0, (int)ep0, 0, 0);  // read ahead, not used
  }
  for (int i = threadIdx.x; i < m; i += blockDim.x) vs[i] = a.send[r + i];
  for (int i = threadIdx.x; i < b; i += blockDim.x) sep[i] = a.etr[ebase + i];
  __syncthreads();
  for (int t = warp; t < m; t += nw) {
    const int4 v = vt[t];
    const int e0 = v.z & 0xffff, k = v.z >> 16;
    bool many = false;
    if (lane < max(2, (k + 1) & ~1)) {
      const int2 x = lane < k ? a.ex[ebase + e0 + lane] : make_int2(0, (int)absent);
      reinterpret_cast<int2 *>(ep + (((uint32_t)v.x - ep0) >> 4))[lane] = make_int2(x.x * R::size, x.y);
      if (lane < k) {
        const int c = a.eC[ebase + e0 + lane];
        many = c > 1;
        er[e0 + lane] = make_int2(x.x + 1, c);
        emap[t][x.x] = (uint8_t)(e0 + lane);
      }
    }
    if (__any_sync(kAll, many) && lane == 0) vt[t].w |= INT_MIN;
  }
  __syncthreads();
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm_b) + (uint32_t)warp * (uint32_t)rows * R::size;
  const uint32_t bJ = base + lane * 8 * SPL, bD = base + R::D + lane * 4 * SPL, bG = base + R::G + lane * SPL;
  const unsigned mask = (1u << a.bits) - 1u;
  const int gend = min(a.ng, ((int)blockIdx.y + 1) * gpc);
  for (int g = blockIdx.y * gpc + warp; g < gend; g += nw) {
    int s[SPL], srow[SPL], si[SPL];
    bool live[SPL];
    lane_sources(a, g, lane, s, live);
    const size_t gt = (size_t)g * a.NT * kGroup + 2 * lane, gu = (size_t)g * a.H * kGroup + 2 * lane;
    bool in_any = false, odd = false;
#pragma unroll
    for (int k = 0; k < SPL; k++) {
      srow[k] = r <= s[k] && s[k] < r + m ? b + s[k] - r : -1;  // the row of this lane's own source
      in_any |= srow[k] >= 0;
      si[k] = a.tidx_of[s[k]];
    }
    const double zero[SPL] = {};
    const uint32_t none[SPL] = {};
    if (b == 0) row_store(bD, none);  // the whole tree: an absent entry of its root reads this row
    for (int i = 0; i < b; i += 4) {  // the separator's rows, four loads of each in flight
      uint32_t d[4][SPL], c[4][SPL];
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
          row_store(bD + (R::S - R::D) + (i + q) * R::size, c[q]);
          row_store(bJ + (i + q) * R::size, zero);
#pragma unroll
          for (int k = 0; k < SPL; k++)
            if (sp[q] == si[k]) srow[k] = i + q;
        }
    }
#pragma unroll
    for (int k = 0; k < SPL; k++) odd |= srow[k] >= 0 || !live[k];
    // special: some lane's source lies among these rows, or lanes without a source
    const bool inside = __any_sync(kAll, in_any), special = __any_sync(kAll, odd);
    unsigned over = 0;
    uint32_t off = b * R::size;  // of the current row
    int4 v = lds128(vt0), e = lds128(v.x);
    for (int t = 0; t < m; t++, off += R::size) {
      const int4 vn = lds128(vt0 + 16 * (t + 1));
      unsigned m1[SPL], m2[SPL];
#pragma unroll
      for (int k = 0; k < SPL; k++) m1[k] = m2[k] = kNoKey;
      if (inside) {
        const int se = vs[t];
#pragma unroll
        for (int k = 0; k < SPL; k++) {
          m1[k] = up_key(a, r + t <= s[k] && s[k] < se, gu + (size_t)(v.w & INT_MAX) * kGroup + k);
          m2[k] = m1[k] == kNoKey ? kNoKey : m1[k] ^ mask;
        }
      }
      uint32_t pe = v.x;
      do {
        uint32_t d1[SPL], d2[SPL];
        row_load(bD + e.x, d1);
        row_load(bD + e.z, d2);
        const int4 ec = e;
        pe += 16;
        if (pe < (uint32_t)v.y) e = lds128(pe);
#pragma unroll
        for (int k = 0; k < SPL; k++) {
          const unsigned v1 = d1[k] + (unsigned)ec.y, v2 = d2[k] + (unsigned)ec.w;
          m1[k] = __vimin3_u32(m1[k], v1, v2);
          m2[k] = __vimin3_u32(m2[k], v1 ^ mask, v2 ^ mask);
        }
      } while (pe < (uint32_t)v.y);
      e = lds128(vn.x);
      unsigned x1[SPL];
      uint32_t c[SPL], dt[SPL];
      unsigned again = 0;  // several entries reach the minimum
#pragma unroll
      for (int k = 0; k < SPL; k++) {
        x1[k] = m1[k] & mask;
        dt[k] = m1[k] & ~mask;
        again |= m1[k] ^ m2[k] ^ mask;
        c[k] = (uint32_t)lds32(bD + (R::S - R::D) + 4 * k + (max(x1[k], 1u) - 1) * R::size);
      }
      if (inside)
#pragma unroll
        for (int k = 0; k < SPL; k++)
          if (x1[k] == 0) c[k] = a.Uc[gu + (size_t)(v.w & INT_MAX) * kGroup + k];
      if (__any_sync(kAll, (again != 0) | (v.w < 0))) {  // or counts above 1: the edges once more
#pragma unroll
        for (int k = 0; k < SPL; k++) {
          const bool tk = (m1[k] ^ m2[k]) != mask;
          unsigned long long cc = x1[k] == 0 ? c[k] : 0;
          for (int q = 0; q < v.z >> 16; q++) {
            const int2 z = er[(v.z & 0xffff) + q];
            const uint32_t xo = (uint32_t)(z.x - 1) * R::size + 4 * k, key = (uint32_t)lds32(v.x + 8 * q + 4);
            const bool hit = tk ? (uint32_t)lds32(bD + xo) + (key & ~mask) == dt[k] : (unsigned)z.x == x1[k];
            if (hit) cc += (unsigned long long)(unsigned)z.y * (uint32_t)lds32(bD + (R::S - R::D) + xo);
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
        for (int k = 0; k < SPL; k++)
          if (!live[k]) x1[k] = kSkipCode;
      row_store(bD + off, dt);
      row_store(bD + (R::S - R::D) + off, c);
      row_store(bJ + off, zero);
      code_store(bG + off, x1[0] | (x1[1] << 8));
      v = vn;
    }
    if (over) *a.wrap = 1;
    for (int t = m - 1; t >= 0; t--) {
      off -= R::size;
      const unsigned code = code_load(bG + off);
      double f[SPL];
      row_load(bJ + off, f);
      const unsigned x0 = code & 0xff;
      int all = 0;
      __match_all_sync(kAll, code, &all);
#pragma unroll
      for (int k = 0; k < SPL; k++) f[k] += 1.0;
      if (all && !special && code == x0 * 0x101 && x0 <= kBottomRows) {  // (no U without special)
        double j[SPL];
        const uint32_t xo = (x0 - 1) * R::size;
        row_load(bJ + xo, j);
#pragma unroll
        for (int k = 0; k < SPL; k++) j[k] += f[k];
        row_store(bJ + xo, j);
        sts32(base + off + R::lead, x0 | kLeadFull);
        continue;
      }
      unsigned x1[SPL];
#pragma unroll
      for (int k = 0; k < SPL; k++) x1[k] = (code >> (8 * k)) & 0xff;
      bool own[SPL] = {};
      if (special) {
        const int4 w = vt[t];
        const int se = vs[t], dep = w.w & INT_MAX;
#pragma unroll
        for (int k = 0; k < SPL; k++) {
          if (b + t == srow[k]) f[k] = lds64(bJ + off + 8 * k);  // the source itself is no target
          if (live[k] && r + t <= s[k] && s[k] < se) {
            const size_t u = gu + (size_t)dep * kGroup + k;
            double sd = x1[k] == 0 ? f[k] : 0.0;
            if (x1[k] == kTieCode && (unsigned)a.Ud[u] == (uint32_t)lds32(bD + off + 4 * k) >> a.bits)
              sd = f[k] * share(1, a.Uc[u], (uint32_t)lds32(bD + (R::S - R::D) + off + 4 * k));
            a.seed[u] = sd;
          }
          own[k] = x1[k] <= (unsigned)kBottomRows && x1[k] > 0 && (int)x1[k] - 1 == srow[k];  // counts apart
        }
      }
#pragma unroll
      for (int k = 0; k < SPL; k++)
        if (x1[k] - 1 < (unsigned)kBottomRows) {
          const uint32_t xo = bJ + (x1[k] - 1) * R::size + 8 * k;
          sts64(xo, lds64(xo) + f[k]);
          if (own[k]) {
            atomicAdd(a.Bs + ebase + emap[t][x1[k] - 1], f[k]);
            x1[k] = 0;
          }
        } else if (x1[k] == kTieCode) {
          const int4 w = vt[t];
          const uint32_t st = (uint32_t)lds32(bD + (R::S - R::D) + off + 4 * k), dk = (uint32_t)lds32(bD + off + 4 * k);
          for (int q = 0; q < w.z >> 16; q++) {
            const int eq = (w.z & 0xffff) + q, xr = er[eq].x - 1;
            const uint32_t xo = (uint32_t)xr * R::size, key = (uint32_t)lds32(w.x + 8 * q + 4);
            if ((uint32_t)lds32(bD + xo + 4 * k) + (key & ~mask) == dk) {
              const double fl = f[k] * share(er[eq].y, (uint32_t)lds32(bD + (R::S - R::D) + xo + 4 * k), st);
              sts64(bJ + xo + 8 * k, lds64(bJ + xo + 8 * k) + fl);
              atomicAdd((xr == srow[k] ? a.Bs : a.Bd) + ebase + eq, fl);
            }
          }
          x1[k] = 0;
        } else {
          x1[k] = 0;
        }
      // up to SPL entries wait for the end, a value per lane each; any others now, one after another
      unsigned leads = 0;
      double w[SPL];
#pragma unroll
      for (int j = 0; j < SPL; j++) {
        unsigned mine = 0;
#pragma unroll
        for (int k = 0; k < SPL; k++) mine = mine ? mine : x1[k];
        const unsigned any = __ballot_sync(kAll, mine != 0);
        w[j] = 0.0;
        if (any) {
          const unsigned xl = __shfl_sync(kAll, mine, __ffs(any) - 1);
          leads |= xl << (8 * j);
#pragma unroll
          for (int k = 0; k < SPL; k++)
            if (x1[k] == xl) {
              w[j] += f[k];
              x1[k] = 0;
            }
        }
      }
      row_store(bJ + off, w);
      sts32(base + off + R::lead, leads);
      for (;;) {
        unsigned mine = 0;
#pragma unroll
        for (int k = 0; k < SPL; k++) mine = mine ? mine : x1[k];
        const unsigned any = __ballot_sync(kAll, mine != 0);
        if (!any) break;
        const unsigned xl = __shfl_sync(kAll, mine, __ffs(any) - 1);
        double z = 0.0;
#pragma unroll
        for (int k = 0; k < SPL; k++)
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
    for (int t0 = 0; t0 < m; t0 += 8) {
      const int t = t0 + (lane >> 2);
      const uint32_t ro = base + (b + min(t, m - 1)) * R::size;
      const unsigned leads = t < m ? (unsigned)lds32(ro + R::lead) : 0;
      double z[SPL] = {};
      if (leads) {
#pragma unroll
        for (int c = 0; c < 8; c++) {
          double x[SPL];
          row_load(ro + ((lane & 3) * 8 + c) * 8 * SPL, x);
#pragma unroll
          for (int k = 0; k < SPL; k++) z[k] += x[k];
        }
      }
      if (leads & kLeadFull) z[0] += z[1];  // one entry: both values of a lane are its
#pragma unroll
      for (int j = 0; j < SPL; j++) {
        z[j] += __shfl_xor_sync(kAll, z[j], 1);
        z[j] += __shfl_xor_sync(kAll, z[j], 2);
        const unsigned x = (leads >> (8 * j)) & 0xff;
        if (x && (lane & 3) == j)
          atomicAdd(a.Bd + ebase + emap[t][x - 1], leads & kLeadFull ? z[j] + (double)kGroup : z[j]);
      }
    }
    for (int i = 0; i < b; i++) {
      double z[SPL];
      row_load(bJ + i * R::size, z);
#pragma unroll
      for (int k = 0; k < SPL; k++)
        if (z[k] != 0.0) atomicAdd(a.J + gt + (size_t)sep[i] * kGroup + k, z[k]);
    }
    __syncwarp();
  }
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
// the small ones at the end (a few thousand triangles each) by one CTA with barriers between them
// instead of a launch each.
__global__ void k_unpack(const int4 *__restrict__ tri, int64_t count, const int32_t *__restrict__ eC, double *B, double *F,
                         const int32_t *wrap) {
  if (__ldcg(wrap) != 0) return;
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < count) unpack_one(tri[k], eC, B, F);
}

constexpr int64_t kTailLevel = 8192;  // triangles of a level that the one-CTA form takes
__global__ void __launch_bounds__(1024) k_unpack_tail(const int4 *__restrict__ tri, const int64_t *__restrict__ at, int l0,
                                                      int l1, const int32_t *__restrict__ eC, double *B, double *F,
                                                      const int32_t *wrap) {
  if (__ldcg(wrap) != 0) return;  // (not written while this kernel runs)
  for (int l = l0; l < l1; l++) {
    const int64_t e = at[l + 1];
    for (int64_t k = at[l] + threadIdx.x; k < e; k += blockDim.x) unpack_one(tri[k], eC, B, F);
    __threadfence();
    __syncthreads();
  }
}

__global__ void k_finish(const double *__restrict__ F, double *__restrict__ bc_tid, int n, const int32_t *wrap) {
  if (__ldcg(wrap) != 0) return;
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
                            const int32_t *__restrict__ depth, const int32_t *__restrict__ tidx_of, const int4 *__restrict__ bot,
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
      if (x >= bt.x) ref = bt.z + (x - bt.x);
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

// triangles (y; t, x): shortcut (t, x) of least length through y.  A warp per (y, deeper vertex t).
__global__ void k_triangles(const int32_t *__restrict__ xoff, const int32_t *__restrict__ xtid, const int32_t *__restrict__ eL,
                            const int32_t *__restrict__ owner, int64_t E, int4 *tri, unsigned long long *count,
                            unsigned long long cap) {
  const int64_t e2 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
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

}  // namespace

// Host part and device arrays of the plan.
struct TreePlan {
  TreeArgs args{};  // without the per-launch fields
  int nbot = 0, up_warps = 0;
  std::vector<int32_t> level_first;  // first piece of each trunk level, end
  std::vector<int32_t> level_len;    // longest piece of each trunk level
  struct BotClass {
    int first, end, rows;
  };
  std::vector<BotClass> bot_class;
  std::vector<int64_t> tri_first;    // first triangle of each unpack level, end
  int4 *tri = nullptr;
  unsigned absent = 0;               // key of a missing entry: above every distance
  int64_t *tri_at = nullptr;         // tri_first on the device
  int32_t *owner = nullptr;          // per edge its lower end
  int tail_level = 0;                // levels from here on hold at most kTailLevel triangles each
  int64_t E = 0, bytes = 0;
  bool off = false;  // a count wrapped: the label kernels answer from now on
  std::vector<void *> owned;

  template <class T>
  T *alloc(size_t count) {
    void *p = nullptr;
    CK(cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T)));
    owned.push_back(p);
    bytes += (int64_t)(std::max<size_t>(count, 1) * sizeof(T));
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
  std::vector<int32_t> piece_of, level_first, trunk_tid;
};

static TreeShape tree_shape(const Index &ix, const std::vector<int64_t> &soff) {
  const int32_t n = ix.n;
  TreeShape s;
  s.tidx_of.assign((size_t)n, 0);
  std::vector<int32_t> heavy((size_t)n, -1), piece((size_t)n, -1);
  // bottoms: maximal subtrees whose separator and vertices fit the rows
  std::vector<char> is_bot((size_t)n, 0);
  for (int32_t t = 0; t < n;) {
    const int32_t size = ix.send[t] - t, k = (int32_t)(soff[t + 1] - soff[t]);
    if (size + k <= kBottomRows && soff[ix.send[t]] - soff[t] <= kBottomEdges) {
      s.bot.push_back(make_int4(t, size, k, 0));
      std::fill(is_bot.begin() + t, is_bot.begin() + ix.send[t], 1);
      t = ix.send[t];
    } else {
      t++;
    }
  }
  std::stable_sort(s.bot.begin(), s.bot.end(), [](const int4 &x, const int4 &y) { return x.y + x.z > y.y + y.z; });
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
  std::vector<int32_t> at(s.level_first.begin(), s.level_first.end()), by_level(ps.size());
  for (size_t i = 0; i < ps.size(); i++) by_level[at[ps[i].level]++] = (int32_t)i;
  for (int32_t id : by_level) {
    const int32_t first = (int32_t)s.trunk_tid.size(), np = (int32_t)s.piece.size();
    for (int32_t t : ps[id].v) {
      s.tidx_of[t] = (int32_t)s.trunk_tid.size();
      s.trunk_tid.push_back(t);
      s.piece_of.push_back(np);
    }
    const int32_t par = ix.parent[ps[id].v[0]];
    s.piece.push_back(make_int4(first, (int32_t)s.trunk_tid.size(), par < 0 ? -1 : s.tidx_of[par], 0));
  }
  return s;
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
  if (!up_warps || (size_t)H * 20 + sizeof(BackShared) > (size_t)d->smem_optin - 2048) return;
  cudaStream_t st = d->s_label;
  auto p = new TreePlan();
  d->tree = p;
  std::vector<void *> tmp;
  auto talloc = [&](size_t bytes) {
    void *q = nullptr;
    CK(cudaMalloc(&q, std::max<size_t>(bytes, 16)));
    tmp.push_back(q);
    return q;
  };
  bool keep = false;
  try {
    TreeArgs &a = p->args;
    p->E = E;
    p->up_warps = up_warps;
    const int32_t n = ix.n;
    const TreeShape s = tree_shape(ix, soff);
    p->nbot = (int)s.bot.size();
    p->level_first = s.level_first;
    for (size_t l = 0; l + 1 < s.level_first.size(); l++) {
      int32_t len = 0;
      for (int32_t q = s.level_first[l]; q < s.level_first[l + 1]; q++) len = std::max(len, s.piece[q].y - s.piece[q].x);
      p->level_len.push_back(len);
    }
    for (int i = 0; i < p->nbot;) {  // bottoms come largest first: launches of 32, 24, 16 and 8 rows
      const int rows = (s.bot[i].y + s.bot[i].z + 7) & ~7;
      int e = i;
      while (e < p->nbot && ((s.bot[e].y + s.bot[e].z + 7) & ~7) == rows) e++;
      p->bot_class.push_back({i, e, rows});
      i = e;
    }
    a.n = n;
    a.H = H;
    a.NT = (int)s.trunk_tid.size();
    a.bits = bits;
    a.dist_lim = (unsigned)(dmax + 1);
    p->absent = ((unsigned)(lim - 2 - dmax) << bits) | ((1u << bits) - 2u);
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
    a.tidx_of = p->upload(s.tidx_of, st);
    a.bot = p->upload(s.bot, st);
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
    int32_t *lvl = (int32_t *)talloc((size_t)E * 4);
    double *cd = a.Bd;  // the edge accumulators are free until the first call
    unsigned long long *cnt = (unsigned long long *)talloc(8 * (kMaxUnpackLevels + 2));
    int32_t *flag = (int32_t *)talloc(16);
    if (E > 0) {
      k_sort_edges<<<blocks_for((int64_t)n * 32, 256), 256, 0, st>>>(d_soff, d_sep, n, xtid, eL, eC);
      CK(cudaGetLastError());
      k_owner<<<blocks_for((int64_t)n * 32, 256), 256, 0, st>>>(a.xoff, n, owner);
      CK(cudaGetLastError());
      const int32_t lcap = (int32_t)(lim - 2 - dmax);
      k_edge_refs<<<blocks_for((int64_t)n * 32, 256), 256, 0, st>>>(a.xoff, xtid, eL, d->depth, a.tidx_of, a.bot, n, bits, lcap, eC,
                                                                  ex, eup, etr);
      CK(cudaGetLastError());
      if (a.NT > 0) {
        k_piece_edges<<<blocks_for((int64_t)a.NT * 32, 256), 256, 0, st>>>(a, tm);
        CK(cudaGetLastError());
      }
      // triangles
      unsigned long long cap = (unsigned long long)E + 1024, found = 0;
      int4 *raw = nullptr;
      for (int round = 0; round < 2; round++) {
        raw = (int4 *)talloc((size_t)cap * 16);
        CK(cudaMemsetAsync(cnt, 0, 8, st));
        k_triangles<<<blocks_for(E * 32, 256), 256, 0, st>>>(a.xoff, xtid, eL, owner, E, raw, cnt, cap);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(&found, cnt, 8, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        if (found <= cap) break;
        cap = found;
      }
      const int64_t T = (int64_t)found;
      CK(cudaMemsetAsync(lvl, 0, (size_t)E * 4, st));
      int32_t top = 0;
      bool settled = T == 0;
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
      if (settled) {
        std::vector<unsigned long long> hist((size_t)kMaxUnpackLevels + 2, 0), first;
        CK(cudaMemsetAsync(cnt, 0, 8 * (kMaxUnpackLevels + 2), st));
        if (T > 0) {
          k_level_hist<<<blocks_for(T, 256), 256, 0, st>>>(raw, T, lvl, cnt);
          CK(cudaGetLastError());
        }
        CK(cudaMemcpyAsync(hist.data(), cnt, hist.size() * 8, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        while (top < kMaxUnpackLevels && hist[top]) top++;
        p->tri_first.assign(1, 0);
        first.push_back(0);
        for (int l = 0; l < top; l++) {
          p->tri_first.push_back(p->tri_first.back() + (int64_t)hist[l]);
          first.push_back((unsigned long long)p->tri_first.back());
        }
        p->tri = p->alloc<int4>((size_t)T);
        p->tri_at = p->upload(p->tri_first, st);
        p->tail_level = top;
        while (p->tail_level > 0 && hist[p->tail_level - 1] <= (unsigned long long)kTailLevel) p->tail_level--;
        CK(cudaMemcpyAsync(cnt, first.data(), first.size() * 8, cudaMemcpyHostToDevice, st));
        if (T > 0) {
          k_level_scatter<<<blocks_for(T, 256), 256, 0, st>>>(raw, T, lvl, cnt, p->tri);
          CK(cudaGetLastError());
        }
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
        keep = bad == 0 && p->tri_first.back() == T;
      }
    } else {
      p->tri_first.assign(1, 0);
      keep = true;
    }
    CK(cudaStreamSynchronize(st));  // the staging vectors die here
  } catch (...) {
    for (void *q : tmp) cudaFree(q);
    p->bytes = 0;  // not yet part of the index's
    tree_free(d);
    try {
      throw;
    } catch (const Error &e) {
      if (e.code != QBC_ENOMEM) throw;
      cudaGetLastError();  // no room for the plan: the label kernels answer
    }
    return;
  }
  for (void *q : tmp) cudaFree(q);
  if (keep) {
    d->bytes += p->bytes;
  } else {
    p->bytes = 0;
    tree_free(d);
  }
}

// ------------------------------------------------------------------------------- launch
// device bytes of one group of sources
static size_t group_bytes(const TreeArgs &a) { return ((size_t)a.NT * (4 + 4 + 4 + 8) + (size_t)a.H * (4 + 4 + 8)) * kGroup; }

// Groups of sources that the per-source scratch holds, at most kMaxGroups.
constexpr int kMaxGroups = 128;
static int groups_fit(const DeviceState *d) {
  const size_t room = (size_t)d->chunk * d->n_pad * sizeof(int4);
  return (int)std::min<size_t>(kMaxGroups, room / group_bytes(d->tree->args));
}

// (source, vertex) pairs from which the tree is the faster path: its launches follow the trunk level by
// level, about 1.1 ms at 50k vertices however few the sources, where the label kernels answer 16
// sources in 1.07 ms and 64 in 1.38 ms, and 256 take 2.40 against 1.87 ms; 2,024 sources of 2,024
// vertices 0.57 against 0.56 ms.  An H2H index's label path counts paths by Kahn waves (1.40 against
// 0.60 ms there).  QBC_TREE_MIN_PAIRS overrides it for tests.
static int64_t min_pairs(const Handle &h) {
  const char *e = std::getenv("QBC_TREE_MIN_PAIRS");
  if (e && *e) return std::strtoll(e, nullptr, 10);
  return h.host.kind == IndexKind::H2H ? (int64_t)1 << 20 : (int64_t)5 << 20;
}

bool use_tree(const Handle &h, const DeviceState *d, int32_t ns) {
  const Tuning &t = h.tuning;
  if (!d->tree || d->tree->off || ns < 1) return false;
  // a tuning that picks a label or dependency kernel, or the test hook of the label rows' copies, gets it
  if (t.lanes_per_source || t.split || t.dep_form || t.queue_depth || t.label_warps || t.label_tile || t.label_passes ||
      t.label_sources || t.label_stream)
    return false;
  const char *hook = std::getenv("QBC_TEST_ROW_WAIT_SPINS");
  if (hook && *hook) return false;
  return (int64_t)ns * d->n >= min_pairs(h) && groups_fit(d) >= 1;
}

const int32_t *tree_guard(const DeviceState *d) { return d->tree ? d->tree->args.wrap : nullptr; }

bool tree_disable(DeviceState *d) {
  if (!d->tree || d->tree->off) return false;
  d->tree->off = true;
  return true;
}

template <int GB>
static void launch_down(const TreeArgs &a, int piece0, int pieces, int pl, int threads, cudaStream_t st) {
  const size_t smem = (size_t)GB * pl * kGroup * 12;
  CK(cudaFuncSetAttribute(k_trunk_down<GB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_trunk_down<GB><<<dim3(pieces, (a.ng + GB - 1) / GB), threads, smem, st>>>(a, piece0, pl);
}
template <int GB>
static void launch_up(const TreeArgs &a, int piece0, int pieces, int pl, int threads, cudaStream_t st) {
  const size_t smem = (size_t)GB * pl * kGroup * 12;
  CK(cudaFuncSetAttribute(k_trunk_up<GB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_trunk_up<GB><<<dim3(pieces, (a.ng + GB - 1) / GB), threads, smem, st>>>(a, piece0, pl);
}

// The bottoms [first, end) of at most `rows` rows: the warps of a CTA share a bottom's edges, and a
// CTA takes more groups one after another while there are CTAs enough.
static void launch_bottom(const TreeArgs &a, int first, int end, int rows, unsigned absent, cudaStream_t st) {
  const int warps = std::min(kBottomWarps, a.ng);
  int gpc = warps;
  while (gpc < 64 && (int64_t)(end - first) * ((a.ng + 2 * gpc - 1) / (2 * gpc)) >= 148 * 24) gpc *= 2;
  const size_t smem = (size_t)warps * rows * RowLayout::size;
  CK(cudaFuncSetAttribute(k_bottom, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_bottom<<<dim3(end - first, (a.ng + gpc - 1) / gpc), warps * 32, smem, st>>>(a, first, rows, gpc, absent);
}

void launch_tree(const Handle &h, DeviceState *d, const int32_t *d_src_tid, int32_t ns, cudaStream_t st) {
  TreePlan &p = *d->tree;
  CK(cudaMemsetAsync(p.args.Bd, 0, ((size_t)p.E * 3 + (size_t)p.args.n) * 8, st));
  auto launched = [&] {
    CK(cudaGetLastError());
    d->launches++;
  };
  const int fit = groups_fit(d);
  const int levels = (int)p.level_len.size();
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
      CK(cudaFuncSetAttribute(k_up_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      k_up_rows<<<(a.ng * kGroup + p.up_warps - 1) / p.up_warps, p.up_warps * 32, smem, st>>>(a);
      launched();
    }
    // a CTA takes one piece, for two groups when there are CTAs enough
    auto pair_of = [&](int pieces) { return a.ng > 1 && (int64_t)pieces * a.ng >= 148 * 8; };
    for (int l = 0; l < levels; l++) {
      const int pieces = p.level_first[l + 1] - p.level_first[l], pl = p.level_len[l];
      launch_down<1>(a, p.level_first[l], pieces, pl, pair_of(pieces) ? 256 : 512, st);
      launched();
    }
    if (a.ng > 4) {
      for (const TreePlan::BotClass &c : p.bot_class) {
        launch_bottom(a, c.first, c.end, c.rows, p.absent, st);
        launched();
      }
    } else if (p.nbot) {
      launch_bottom(a, 0, p.nbot, p.bot_class[0].rows, p.absent, st);
      launched();
    }
    if (d->profiling) {
      CK(cudaEventRecord(ev.second, st));
      ev = take_events(d->ev_dp, d->ev_dp_used);
      CK(cudaEventRecord(ev.first, st));
    }
    for (int l = levels - 1; l >= 0; l--) {
      const int pieces = p.level_first[l + 1] - p.level_first[l], pl = p.level_len[l];
      launch_up<1>(a, p.level_first[l], pieces, pl, pair_of(pieces) ? 256 : 512, st);
      launched();
    }
    {
      const size_t smem = (size_t)a.H * 20;
      CK(cudaFuncSetAttribute(k_up_back, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      k_up_back<<<a.ns, kBackWarps * 32, smem, st>>>(a);
      launched();
    }
    if (d->profiling) CK(cudaEventRecord(ev.second, st));
    d->label_launches++;
    d->dep_launches++;
  }
  const TreeArgs &a = p.args;
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
    k_unpack_tail<<<1, 1024, 0, st>>>(p.tri, p.tri_at, p.tail_level, top, a.eC, a.Bd, a.F, a.wrap);
    launched();
  }
  k_finish<<<std::min(148 * 4, (p.args.n + 255) / 256), 256, 0, st>>>(p.args.F, d->bc_tid, p.args.n, p.args.wrap);
  launched();
}

}  // namespace qbc
