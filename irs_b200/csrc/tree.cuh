// Quadtree over the star field, built level by level on the device.
//
// Semantics follow the reference tree (include/tree_node.cuh, driven from
// include/ipm.cuh:740-842):
//   * the root is centred at 0 with half length root_half_length;
//   * a node is split into 4 children when its own stars plus its neighbours'
//     stars exceed 32 (get_node_star_info_kernel / create_children_kernel,
//     tree_node.cuh:321-381), empty nodes included;
//   * child q has centre parent + hl/2 * {(1,1),(-1,1),(-1,-1),(1,-1)}[q]
//     (make_child, tree_node.cuh:151-168) and owns the stars with
//     x >= cx && y >= cy (q=0), x < cx && y >= cy (1), x < cx && y < cy (2),
//     otherwise (3); children's star ranges are contiguous in child order
//     (sort_stars_kernel, tree_node.cuh:392-501);
//   * neighbours / interaction lists as set_neighbors (tree_node.cuh:183-267).
// Differences by design: node slots are assigned by an exclusive scan over the
// split flags and stars are partitioned stably, so the tree and the star order
// are deterministic (the reference uses atomics for both). The structure
// (levels, centres, per-node star sets, neighbour sets) is the same.
//
// Layout: structure-of-arrays over a global node index; nodes of level l are
// [level_off[l], level_off[l+1]). Each node also records the half-open box
// [lox, hix) x [loy, hiy) that the descent of get_nearest_node
// (tree_node.cuh:529-561) maps to it; a ray lattice is partitioned by leaf
// with those boxes.
#pragma once
#include "common.cuh"
#include "devutil.cuh"
#include "params.hpp"

#include <algorithm>
#include <cstdio>
#include <vector>

namespace irsb {

template <typename T>
struct TreeDev {
  int cap = 0;
  int num_nodes = 0;
  int levels = 0;  // number of levels - 1 (the reference's tree_levels)
  int num_leaves = 0;
  std::vector<int> level_off;  // host copy, size levels + 2
  DevVec<T> cx, cy, hl;
  DevVec<int> level, parent, child0, sbeg, scnt;
  DevVec<int> rid;         // realization of the node (0 for a single star field)
  DevVec<int> nbr, n_nbr;  // [cap][kMaxNeighbors]
  DevVec<int> sil, n_sil;  // [cap][kMaxSameLevelIL]
  DevVec<int> dil, n_dil;  // [cap][kMaxDiffLevelIL]
  DevVec<double> lox, hix, loy, hiy;
  // scratch
  DevVec<int> split, rank;
  DevVec<int> cta;          // per-CTA counts of the build
  DevVec<int> status;       // TreeStatus, then the level offsets (the FMM reads them there)
  DevVec<unsigned long long> words;  // grid barriers of the build and of the expansions
  DevVec<StarRec<T>> tmp_stars, star_backup;
  HostBuf<int> h_status;      // copy of `status`
  long long launches = 0;   // kernels the last build launched
};

template <typename T>
bool tree_reserve(TreeDev<T>& t, int want, cudaStream_t s) {
  if (want <= t.cap) return true;
  int nc = t.cap ? t.cap : 1024;
  while (nc < want) nc *= 2;
  bool ok = t.cx.reserve(nc, s) && t.cy.reserve(nc, s) && t.hl.reserve(nc, s) && t.level.reserve(nc, s) &&
            t.parent.reserve(nc, s) && t.child0.reserve(nc, s) && t.sbeg.reserve(nc, s) && t.scnt.reserve(nc, s) && t.rid.reserve(nc, s) &&
            t.nbr.reserve(size_t(nc) * kMaxNeighbors, s) && t.n_nbr.reserve(nc, s) &&
            t.sil.reserve(size_t(nc) * kMaxSameLevelIL, s) && t.n_sil.reserve(nc, s) &&
            t.dil.reserve(size_t(nc) * kMaxDiffLevelIL, s) && t.n_dil.reserve(nc, s) && t.lox.reserve(nc, s) &&
            t.hix.reserve(nc, s) && t.loy.reserve(nc, s) && t.hiy.reserve(nc, s);
  if (!ok) return false;
  // keep the logical sizes in step so that growth copies every live node
  for (auto* v : {&t.cx.n, &t.cy.n, &t.hl.n}) *v = nc;
  t.level.n = t.parent.n = t.child0.n = t.sbeg.n = t.scnt.n = t.n_nbr.n = t.n_sil.n = t.n_dil.n = t.rid.n = nc;
  t.lox.n = t.hix.n = t.loy.n = t.hiy.n = nc;
  t.nbr.n = size_t(nc) * kMaxNeighbors;
  t.sil.n = size_t(nc) * kMaxSameLevelIL;
  t.dil.n = size_t(nc) * kMaxDiffLevelIL;
  t.cap = nc;
  return true;
}

// Words of TreeDev::status: the build's outcome, then off[0 .. kMaxLevels + 1]
// (nodes of level l are [off[l], off[l + 1]); the offsets past the last level
// all hold the number of nodes).
enum TreeStatus : int {
  kTreeErr = 0,        // DeviceError bits
  kTreeBarrier = 1,    // a grid barrier gave up
  kTreeLevels = 2,     // the deepest level
  kTreeLeaves = 3,     // leaves
  kTreeNear = 4,       // a leaf's near field overflowed (leaf_build, build_leaves)
  kTreeTable = 5,      // the tile table overflowed (leaf_tile_table)
  kTreeLattice = 6,    // LatticeStat: 64-bit words (lattice_rects)
  kTreeOff = kTreeLattice + 2 * 3,
  kTreeStatusWords = kTreeOff + kMaxLevels + 2,
};
// Grid barriers of a build: at most four per level, one for the leaves; then
// those of the expansions (fmm.cuh).
constexpr int kTreeBarriers = 4 * kMaxLevels + 8;
constexpr int kFmmBarriers = 2 * kMaxLevels + 4;

template <typename T>
struct TreeBuild {
  T *cx, *cy, *hl;
  int *level, *parent, *child0, *sbeg, *scnt, *rid, *nbr, *n_nbr, *sil, *n_sil, *dil, *n_dil;
  double *lox, *hix, *loy, *hiy;
  int *split, *rank;  // per node of the level: split flag; rank among the CTA's split nodes
  int* cta;           // [3 + 4 * kShareNodes][grid] counts per CTA
  int* status;
  unsigned long long* words;
  long long* leaf_pos;  // per node: leaves before it
  int* leaf_node;       // per leaf: its node
  StarRec<T>*stars, *tmp;
  int nroots, nstars, cap, nlev;
  T root_hl;                  // one root over all stars, or
  const T* root_hls;          // per root: half length
  const long long* star_off;  // per root: first star (nroots + 1 values)
};

template <typename T>
__device__ __forceinline__ int star_quadrant(T x, T y, T cx, T cy) {
  if (x >= cx && y >= cy) return 0;
  if (x < cx && y >= cy) return 1;
  if (x < cx && y < cy) return 2;
  return 3;
}

// set_neighbors (tree_node.cuh:183-267) for node k (of a level >= 1) by one
// warp: lane q examines candidate q in the order of the reference's loops (the
// 4 siblings, then for each of the parent's neighbours either the neighbour
// itself, a leaf, or its 4 children), and each list takes its candidates in
// that order through a ballot prefix, so the lists are those of one thread
// walking the loops. Returns the stars of the node and its neighbours.
template <typename T>
__device__ __forceinline__ int tree_node_lists(const TreeBuild<T>& b, int k, int lane, int& err) {
  const unsigned below = (1u << lane) - 1u;
  const int p = b.parent[k];
  const T h = b.hl[k], x = b.cx[k], y = b.cy[k];
  const int pc0 = b.child0[p];
  const int nq = 4 + 4 * b.n_nbr[p];
  int nn = 0, ns = 0, nd = 0, near = 0;
  for (int q0 = 0; q0 < nq; q0 += 32) {
    const int q = q0 + lane;
    int cat = 0, c = -1, cnt = 0;  // 1 neighbour, 2 same-level interaction, 3 different-level interaction
    if (q < 4) {
      c = pc0 + q;
      cnt = b.scnt[c];
      if (cnt != 0 && c != k) cat = 1;
    } else if (q < nq) {
      const int i = (q - 4) >> 2, j = (q - 4) & 3;
      const int nb = b.nbr[p * kMaxNeighbors + i];
      cnt = b.scnt[nb];
      if (cnt != 0) {
        const int nc0 = b.child0[nb];
        if (nc0 < 0) {
          if (j == 0) {
            c = nb;
            cat = (double(xfabs(T(b.cx[nb] - x))) < 3.5 * double(h) && double(xfabs(T(b.cy[nb] - y))) < 3.5 * double(h))
                      ? 1
                      : 3;
          }
        } else {
          c = nc0 + j;
          cnt = b.scnt[c];
          if (cnt != 0) cat = (xfabs(T(b.cx[c] - x)) < 3 * h && xfabs(T(b.cy[c] - y)) < 3 * h) ? 1 : 2;
        }
      }
    }
    const unsigned m1 = __ballot_sync(0xffffffffu, cat == 1);
    const unsigned m2 = __ballot_sync(0xffffffffu, cat == 2);
    const unsigned m3 = __ballot_sync(0xffffffffu, cat == 3);
    if (cat == 1) {
      const int pos = nn + __popc(m1 & below);
      if (pos < kMaxNeighbors) {
        b.nbr[k * kMaxNeighbors + pos] = c;
        near += cnt;
      } else {
        err |= kErrNeighborOverflow;
      }
    } else if (cat == 2) {
      const int pos = ns + __popc(m2 & below);
      if (pos < kMaxSameLevelIL) b.sil[k * kMaxSameLevelIL + pos] = c;
      else err |= kErrSameLevelOverflow;
    } else if (cat == 3) {
      const int pos = nd + __popc(m3 & below);
      if (pos < kMaxDiffLevelIL) b.dil[k * kMaxDiffLevelIL + pos] = c;
      else err |= kErrDiffLevelOverflow;
    }
    nn += __popc(m1);
    ns += __popc(m2);
    nd += __popc(m3);
  }
  if (lane == 0) {
    b.n_nbr[k] = min(nn, kMaxNeighbors);
    b.n_sil[k] = min(ns, kMaxSameLevelIL);
    b.n_dil[k] = min(nd, kMaxDiffLevelIL);
  }
  return int(__reduce_add_sync(0xffffffffu, unsigned(near))) + b.scnt[k];
}

// The 4 children of node k from c0 on; their star ranges follow from the
// partition of k's stars.
template <typename T>
__device__ __forceinline__ void tree_node_children(const TreeBuild<T>& b, int k, int c0) {
  b.child0[k] = c0;
  const T h = b.hl[k] / 2;
  const T pcx = b.cx[k], pcy = b.cy[k];
  const T ox[4] = {T(1), T(-1), T(-1), T(1)};
  const T oy[4] = {T(1), T(1), T(-1), T(-1)};
  const double plox = b.lox[k], phix = b.hix[k], ploy = b.loy[k], phiy = b.hiy[k];
  const int lev = b.level[k] + 1, r = b.rid[k];
  for (int q = 0; q < 4; q++) {
    const int c = c0 + q;
    b.cx[c] = pcx + h * ox[q];
    b.cy[c] = pcy + h * oy[q];
    b.hl[c] = h;
    b.level[c] = lev;
    b.parent[c] = k;
    b.rid[c] = r;
    b.child0[c] = -1;
    b.n_nbr[c] = b.n_sil[c] = b.n_dil[c] = 0;
    // x >= pcx for q = 0, 3; y >= pcy for q = 0, 1
    const bool right = (q == 0 || q == 3), top = (q == 0 || q == 1);
    b.lox[c] = right ? double(pcx) : plox;
    b.hix[c] = right ? phix : double(pcx);
    b.loy[c] = top ? double(pcy) : ploy;
    b.hiy[c] = top ? phiy : double(pcy);
  }
}

// Stars [s0, s0 + n) of a node with centre (x, y) into its 4 children's ranges
// from child c0 on, keeping their relative order: by one warp.
template <typename T>
__device__ __forceinline__ void tree_partition_warp(const TreeBuild<T>& b, int s0, int n, int c0, T x, T y, int lane) {
  int cnt[4] = {0, 0, 0, 0};
  for (int i0 = 0; i0 < n; i0 += 32) {
    int q = -1;
    if (i0 + lane < n) q = star_quadrant(b.stars[s0 + i0 + lane].x, b.stars[s0 + i0 + lane].y, x, y);
#pragma unroll
    for (int qq = 0; qq < 4; qq++) cnt[qq] += __popc(__ballot_sync(0xffffffffu, q == qq));
  }
  int base[4];
  base[0] = s0;
#pragma unroll
  for (int q = 1; q < 4; q++) base[q] = base[q - 1] + cnt[q - 1];
#pragma unroll
  for (int q = 0; q < 4; q++)
    if (lane == q) {
      b.sbeg[c0 + q] = base[q];
      b.scnt[c0 + q] = cnt[q];
    }
  for (int i0 = 0; i0 < n; i0 += 32) {
    int q = -1;
    StarRec<T> st;
    if (i0 + lane < n) {
      st = b.stars[s0 + i0 + lane];
      q = star_quadrant(st.x, st.y, x, y);
    }
#pragma unroll
    for (int qq = 0; qq < 4; qq++) {
      const unsigned m = __ballot_sync(0xffffffffu, q == qq);
      if (q == qq) b.tmp[base[qq] + __popc(m & ((1u << lane) - 1u))] = st;
      base[qq] += __popc(m);
    }
  }
  __syncwarp();
  for (int i = lane; i < n; i += 32) b.stars[s0 + i] = b.tmp[s0 + i];
}

constexpr int kTreeThreads = 512;
constexpr int kTreeWarps = kTreeThreads / 32;
// A node of up to this many stars is partitioned by one warp, up to
// tree_big_node by its CTA, beyond that by all CTAs.
constexpr int kPartWarpStars = 512;

// The same by the whole CTA.
template <typename T>
__device__ __forceinline__ void tree_partition_block(const TreeBuild<T>& b, int s0, int n, int c0, T x, T y) {
  __shared__ int cnt[4], base[4], warp_cnt[kTreeWarps][4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x < 4) cnt[threadIdx.x] = 0;
  __syncthreads();
  int lc[4] = {0, 0, 0, 0};
  for (int i = threadIdx.x; i < n; i += kTreeThreads) {
    const int q = star_quadrant(b.stars[s0 + i].x, b.stars[s0 + i].y, x, y);
#pragma unroll
    for (int qq = 0; qq < 4; qq++) lc[qq] += q == qq;
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int v = int(__reduce_add_sync(0xffffffffu, unsigned(lc[q])));
    if (lane == 0 && v) atomicAdd(&cnt[q], v);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = s0;
    for (int q = 0; q < 4; q++) {
      base[q] = acc;
      b.sbeg[c0 + q] = acc;
      b.scnt[c0 + q] = cnt[q];
      acc += cnt[q];
    }
  }
  __syncthreads();
  for (int start = 0; start < n; start += kTreeThreads) {
    const int i = start + int(threadIdx.x);
    int q = -1;
    StarRec<T> st;
    if (i < n) {
      st = b.stars[s0 + i];
      q = star_quadrant(st.x, st.y, x, y);
    }
    unsigned mine = 0;
#pragma unroll
    for (int qq = 0; qq < 4; qq++) {
      const unsigned m = __ballot_sync(0xffffffffu, q == qq);
      if (lane == 0) warp_cnt[w][qq] = __popc(m);
      if (q == qq) mine = m;
    }
    __syncthreads();
    if (q >= 0) {
      int off = base[q];
      for (int ww = 0; ww < w; ww++) off += warp_cnt[ww][q];
      b.tmp[off + __popc(mine & ((1u << lane) - 1u))] = st;
    }
    __syncthreads();
    if (threadIdx.x < 4) {
      int add = 0;
      for (int ww = 0; ww < kTreeWarps; ww++) add += warp_cnt[ww][threadIdx.x];
      base[threadIdx.x] += add;
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < n; i += kTreeThreads) b.stars[s0 + i] = b.tmp[s0 + i];
  __syncthreads();
}

// The same by all CTAs, for every split node of the level [beg, end) that holds
// more than `big` stars: CTA c takes the c-th share [s0, s1) of the whole star
// array (the level's nodes are star ranges in node order, so a share meets a
// few of them, all but the first and last inside it), counts its stars per node
// and quadrant, and after a grid barrier places them in `tmp` behind those of
// the CTAs before it; after another one it copies its share back. At most
// kShareNodes such nodes meet a share (tree_big_node). Returns false when a
// grid barrier gave up.
constexpr int kShareNodes = 10;
__host__ __device__ __forceinline__ int tree_big_node(int per) { return per / 8 > 2048 ? per / 8 : 2048; }

template <typename T>
__device__ __forceinline__ bool tree_partition_shared(const TreeBuild<T>& b, int beg, int end, int per, int big,
                                                      unsigned long long*& word, long long spins) {
  __shared__ int s_node[kShareNodes], s_n, run[kShareNodes][4], warp_cnt[kTreeWarps][4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, grid = gridDim.x, me = blockIdx.x;
  const int s0 = min(b.nstars, me * per), s1 = min(b.nstars, s0 + per);
  int* seg_n = b.cta + 2 * grid;   // [grid] big nodes that meet the share
  int* counts = b.cta + 3 * grid;  // [grid][kShareNodes][4]
  if (threadIdx.x == 0) {
    int lo = beg, hi = end - 1;  // last node that starts at or before s0
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (b.sbeg[mid] <= s0) lo = mid;
      else hi = mid - 1;
    }
    int n = 0;
    for (int k = lo; s0 < s1 && k < end && b.sbeg[k] < s1; k++)
      if (b.split[k - beg] && b.scnt[k] > big && b.sbeg[k] + b.scnt[k] > s0 && n < kShareNodes) s_node[n++] = k;
    s_n = n;
    seg_n[me] = n;
  }
  if (threadIdx.x < kShareNodes * 4) run[threadIdx.x / 4][threadIdx.x % 4] = 0;
  __syncthreads();
  const int n = s_n;
  for (int g = 0; g < n; g++) {
    const int k = s_node[g], i0 = max(s0, b.sbeg[k]), i1 = min(s1, b.sbeg[k] + b.scnt[k]);
    const T x = b.cx[k], y = b.cy[k];
    int lc[4] = {0, 0, 0, 0};
    for (int i = i0 + int(threadIdx.x); i < i1; i += kTreeThreads) {
      const int q = star_quadrant(b.stars[i].x, b.stars[i].y, x, y);
#pragma unroll
      for (int qq = 0; qq < 4; qq++) lc[qq] += q == qq;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int v = int(__reduce_add_sync(0xffffffffu, unsigned(lc[q])));
      if (lane == 0 && v) atomicAdd(&run[g][q], v);
    }
  }
  __syncthreads();
  if (threadIdx.x < n * 4) counts[me * kShareNodes * 4 + threadIdx.x] = run[threadIdx.x / 4][threadIdx.x % 4];
  if (grid_barrier_sum(word++, 0, b.status + kTreeBarrier, spins) < 0) return false;
  // warp g: node g's counts before this CTA and in all. The node is the last
  // big one of the CTA it starts in and the first of every CTA after that.
  for (int g = w; g < n; g += kTreeWarps) {
    const int k = s_node[g], c0 = b.sbeg[k] / per, c1 = (b.sbeg[k] + b.scnt[k] - 1) / per;
    int before[4] = {0, 0, 0, 0}, all[4] = {0, 0, 0, 0};
    for (int c = c0 + lane; c <= c1; c += 32) {
      const int gg = c == me ? g : (c == c0 ? seg_n[c] - 1 : 0);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int v = counts[(c * kShareNodes + gg) * 4 + q];
        all[q] += v;
        before[q] += c < me ? v : 0;
      }
    }
    int acc = b.sbeg[k];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      all[q] = int(__reduce_add_sync(0xffffffffu, unsigned(all[q])));
      before[q] = int(__reduce_add_sync(0xffffffffu, unsigned(before[q])));
      if (lane == 0) {
        run[g][q] = acc + before[q];
        if (c0 == me) {
          b.sbeg[b.child0[k] + q] = acc;
          b.scnt[b.child0[k] + q] = all[q];
        }
      }
      acc += all[q];
    }
  }
  __syncthreads();
  for (int g = 0; g < n; g++) {
    const int k = s_node[g], i0 = max(s0, b.sbeg[k]), i1 = min(s1, b.sbeg[k] + b.scnt[k]);
    const T x = b.cx[k], y = b.cy[k];
    for (int r = i0; r < i1; r += kTreeThreads) {  // rounds in star order
      const int i = r + int(threadIdx.x);
      int q = -1;
      StarRec<T> st;
      if (i < i1) {
        st = b.stars[i];
        q = star_quadrant(st.x, st.y, x, y);
      }
      unsigned mine = 0;
#pragma unroll
      for (int qq = 0; qq < 4; qq++) {
        const unsigned m = __ballot_sync(0xffffffffu, q == qq);
        if (lane == 0) warp_cnt[w][qq] = __popc(m);
        if (q == qq) mine = m;
      }
      __syncthreads();
      if (q >= 0) {
        int pos = run[g][q];
        for (int ww = 0; ww < w; ww++) pos += warp_cnt[ww][q];
        b.tmp[pos + __popc(mine & ((1u << lane) - 1u))] = st;
      }
      __syncthreads();
      if (threadIdx.x < 4) {
        int add = 0;
        for (int ww = 0; ww < kTreeWarps; ww++) add += warp_cnt[ww][threadIdx.x];
        run[g][threadIdx.x] += add;
      }
      __syncthreads();
    }
  }
  if (grid_barrier_sum(word++, 0, b.status + kTreeBarrier, spins) < 0) return false;
  for (int g = 0; g < n; g++) {
    const int k = s_node[g], i0 = max(s0, b.sbeg[k]), i1 = min(s1, b.sbeg[k] + b.scnt[k]);
    for (int i = i0 + int(threadIdx.x); i < i1; i += kTreeThreads) b.stars[i] = b.tmp[i];
  }
  return true;
}

// Exclusive scan of a flag (0 or 1) over the CTA's threads; *total their sum.
__device__ __forceinline__ int block_scan_flag(int flag, int* total) {
  __shared__ int s_w[kTreeWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned m = __ballot_sync(0xffffffffu, flag != 0);
  if (lane == 0) s_w[w] = __popc(m);
  __syncthreads();
  int before = __popc(m & ((1u << lane) - 1u)), all = 0;
#pragma unroll
  for (int ww = 0; ww < kTreeWarps; ww++) {
    const int v = s_w[ww];
    before += ww < w ? v : 0;
    all += v;
  }
  __syncthreads();
  *total = all;
  return before;
}

// Sums of an array over the CTAs before this one and over all of them.
__device__ __forceinline__ void cta_prefix(const int* v, int* before, int* all) {
  __shared__ int s_r[2];
  if (threadIdx.x < 32) {
    int p = 0, a = 0;
    for (int c = threadIdx.x; c < int(gridDim.x); c += 32) {
      const int x = v[c];
      a += x;
      p += c < int(blockIdx.x) ? x : 0;
    }
    p = int(__reduce_add_sync(0xffffffffu, unsigned(p)));
    a = int(__reduce_add_sync(0xffffffffu, unsigned(a)));
    if (threadIdx.x == 0) {
      s_r[0] = p;
      s_r[1] = a;
    }
  }
  __syncthreads();
  *before = s_r[0];
  *all = s_r[1];
  __syncthreads();
}

// The whole tree in one cooperative launch: per level, the nodes' lists and
// split flags (a warp per node), a grid barrier, the children of the split
// nodes and the stable partition of their stars (by a warp, the CTA or, for the
// few nodes of the top levels, all CTAs), a grid barrier; finally the leaves are numbered in node order. CTA c owns the
// c-th contiguous share of a level's nodes, so node slots and leaf numbers are
// those of an exclusive scan.
//
// Bound by latency: a handful of dependent loads per level and phase. As eight
// to eleven launches per level with three scan passes among them, a field of
// 2.2e3 stars (7 levels) took 0.35 ms (B200); now 0.09.
template <typename T>
__global__ void __launch_bounds__(kTreeThreads, 1) tree_build_kernel(TreeBuild<T> b) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int grid = gridDim.x, me = blockIdx.x;
  const long long spins = (1LL << 23) + b.nstars;
  unsigned long long* word = b.words;
  int* off = b.status + kTreeOff;
  int* berr = b.status + kTreeBarrier;
  {  // roots
    const int per = (b.nroots + grid - 1) / grid;
    for (int r = me * per + int(threadIdx.x); r < min(b.nroots, (me + 1) * per); r += kTreeThreads) {
      b.cx[r] = b.cy[r] = T(0);
      b.hl[r] = b.root_hls ? b.root_hls[r] : b.root_hl;
      b.level[r] = 0;
      b.parent[r] = -1;
      b.child0[r] = -1;
      b.sbeg[r] = b.star_off ? int(b.star_off[r]) : 0;
      b.scnt[r] = b.star_off ? int(b.star_off[r + 1] - b.star_off[r]) : b.nstars;
      b.rid[r] = r;
      b.n_nbr[r] = b.n_sil[r] = b.n_dil[r] = 0;
      b.lox[r] = b.loy[r] = -INFINITY;
      b.hix[r] = b.hiy[r] = INFINITY;
    }
    __syncthreads();
  }
  const int share = (b.nstars + grid - 1) / grid, big = tree_big_node(share);
  int beg = 0, end = b.nroots, l = 0;
  for (;; l++) {
    const int n = end - beg, per = (n + grid - 1) / grid;
    const int k0 = min(end, beg + me * per), k1 = min(end, k0 + per);
    // ---- lists, split flags and their ranks within the CTA
    int err = 0;
    for (int k = k0 + w; k < k1; k += kTreeWarps) {
      const int near = l > 0 ? tree_node_lists(b, k, lane, err) : b.scnt[k];
      if (lane == 0) b.split[k - beg] = near > kMaxStarsDirect ? 1 : 0;
    }
    if (err) atomicOr(b.status + kTreeErr, err);
    __syncthreads();
    int mine = 0, bigs = 0;
    for (int base = k0; base < k1; base += kTreeThreads) {
      const int k = base + int(threadIdx.x);
      const int f = k < k1 ? b.split[k - beg] : 0;
      bigs |= f && b.scnt[k] > big;
      int total;
      const int before = block_scan_flag(f, &total);
      if (k < k1) b.rank[k - beg] = mine + before;
      mine += total;
    }
    if (threadIdx.x == 0) b.cta[(l & 1) * grid + me] = mine;
    bigs = __any_sync(0xffffffffu, bigs) ? 1 : 0;
    bigs = grid_barrier_sum(word++, bigs, berr, spins);  // > 0: some node is partitioned by all CTAs
    if (bigs < 0) return;
    // ---- children
    int before, nsplit;
    cta_prefix(b.cta + (l & 1) * grid, &before, &nsplit);
    if (me == 0 && threadIdx.x == 0) off[l] = beg;
    int stop = 0;  // running out of levels or of node capacity ends the build with this level's nodes as leaves
    if (nsplit > 0 && l == b.nlev - 1) stop = kErrLevelOverflow;
    else if ((long long)end + 4LL * nsplit > b.cap) stop = kErrNodeOverflow;
    if (stop && me == 0 && threadIdx.x == 0) atomicOr(b.status + kTreeErr, stop);
    if (stop || nsplit == 0) break;
    int mid = 0;  // nodes of the CTA's share that the whole CTA partitions
    for (int k = k0 + int(threadIdx.x); k < k1; k += kTreeThreads)
      if (b.split[k - beg]) {
        tree_node_children(b, k, end + 4 * (before + b.rank[k - beg]));
        mid |= b.scnt[k] > kPartWarpStars && b.scnt[k] <= big;
      }
    mid = __syncthreads_or(mid);
    for (int k = k0 + w; k < k1; k += kTreeWarps)
      if (b.split[k - beg] && b.scnt[k] <= kPartWarpStars)
        tree_partition_warp(b, b.sbeg[k], b.scnt[k], b.child0[k], b.cx[k], b.cy[k], lane);
    for (int k = k0; mid && k < k1; k++)
      if (b.split[k - beg] && b.scnt[k] > kPartWarpStars && b.scnt[k] <= big)  // CTA-uniform
        tree_partition_block(b, b.sbeg[k], b.scnt[k], b.child0[k], b.cx[k], b.cy[k]);
    if (bigs > 0 && !tree_partition_shared(b, beg, end, share, big, word, spins)) return;
    if (grid_barrier_sum(word++, 0, berr, spins) < 0) return;
    beg = end;
    end += 4 * nsplit;
  }
  // ---- leaves in node order
  const int per = (end + grid - 1) / grid, k0 = min(end, me * per), k1 = min(end, k0 + per);
  int mine = 0;
  for (int base = k0; base < k1; base += kTreeThreads) {
    const int k = base + int(threadIdx.x);
    int total;
    const int pos = block_scan_flag(k < k1 && b.child0[k] < 0, &total);
    if (k < k1) b.leaf_pos[k] = mine + pos;
    mine += total;
  }
  int* counts = b.cta + 2 * grid;
  if (threadIdx.x == 0) counts[me] = mine;
  if (grid_barrier_sum(word++, 0, berr, spins) < 0) return;
  int before, leaves;
  cta_prefix(counts, &before, &leaves);
  for (int k = k0 + int(threadIdx.x); k < k1; k += kTreeThreads) {
    const long long pos = b.leaf_pos[k] + before;
    b.leaf_pos[k] = pos;
    if (b.child0[k] < 0) b.leaf_node[pos] = k;
  }
  if (me == 0 && threadIdx.x == 0) {
    b.status[kTreeLevels] = l;
    b.status[kTreeLeaves] = leaves;
    for (int i = l + 1; i <= kMaxLevels + 1; i++) off[i] = end;
  }
}

// Launches the build of nroots trees over `stars` (device, permuted in place
// into tree order) on stream s: no synchronisation. t's node arrays hold cap
// nodes. leaf_pos / leaf_node: DevVecs of at least cap entries.
template <typename T>
bool launch_tree_build(TreeDev<T>& t, StarRec<T>* stars, int nstars, int nroots, T root_hl, const T* root_hls,
                       const long long* star_off, int cap, int nlev, long long* leaf_pos, int* leaf_node,
                       cudaStream_t s) {
  int grid = 0;
  // a CTA per 64 stars: fewer arrivals per barrier where a field has less work
  // than the whole chip
  if (!cooperative_grid(tree_build_kernel<T>, kTreeThreads, std::max(nroots, ceil_div(nstars, 64)), &grid)) return false;
  TreeBuild<T> b{t.cx.p, t.cy.p, t.hl.p, t.level.p, t.parent.p, t.child0.p, t.sbeg.p, t.scnt.p, t.rid.p, t.nbr.p,
                 t.n_nbr.p, t.sil.p, t.n_sil.p, t.dil.p, t.n_dil.p, t.lox.p, t.hix.p, t.loy.p, t.hiy.p, t.split.p,
                 t.rank.p, t.cta.p, t.status.p, t.words.p, leaf_pos, leaf_node, stars, t.tmp_stars.p, nroots, nstars,
                 cap, nlev, root_hl, root_hls, star_off};
  IRSB_CKR(cudaMemsetAsync(t.words.p, 0, (kTreeBarriers + kFmmBarriers) * sizeof(unsigned long long), s));
  IRSB_CKR(cudaMemsetAsync(t.status.p, 0, kTreeStatusWords * sizeof(int), s));
  void* args[] = {&b};
  IRSB_CKR(cudaLaunchCooperativeKernel((const void*)tree_build_kernel<T>, dim3(grid), dim3(kTreeThreads), args, 0, s));
  return true;
}

// Buffers of a build over nstars stars with room for cap nodes.
template <typename T>
bool tree_build_reserve(TreeDev<T>& t, int nstars, int cap, cudaStream_t s) {
  return tree_reserve(t, cap, s) && t.split.reserve(cap, s) && t.rank.reserve(cap, s) &&
         t.cta.reserve((3 + 4 * kShareNodes) * 1024, s) && t.status.reserve(kTreeStatusWords, s) &&
         t.words.reserve(kTreeBarriers + kFmmBarriers, s) && t.tmp_stars.reserve(nstars, s);
}

// The first n status words to the host, once the work queued on s is done. Pinning
// these words took 0.5 - 1 ms of every new object's first run; it gains 2 us of each
// of a run's two copies (HostBuf).
constexpr long long kStatusPinAfter = 128;
template <typename T>
bool tree_status(TreeDev<T>& t, int n, cudaStream_t s) {
  if (!t.h_status.prepare(kTreeStatusWords, kStatusPinAfter)) return false;
  IRSB_CKR(cudaMemcpyAsync(t.h_status.p, t.status.p, n * sizeof(int), cudaMemcpyDeviceToHost, s));
  return IRSB_CK(cudaStreamSynchronize(s));
}

// Builds the tree over `stars` (device, permuted in place into tree order) and
// numbers its leaves (leaf_pos, leaf_node: grown as needed). Returns false on a
// CUDA error or a list overflow. Node storage is reserved up front; a field
// that needs more restores its star order and builds again with twice the
// capacity. `before_sync(cap)` enqueues work that needs only the device's
// tree ahead of the one synchronisation.
template <typename T, typename F>
bool build_tree(TreeDev<T>& t, StarRec<T>* stars, int nstars, T root_hl, DevVec<long long>& leaf_pos,
                DevVec<int>& leaf_node, cudaStream_t s, F before_sync) {
  if (!t.star_backup.reserve(nstars, s)) return false;
  IRSB_CKR(cudaMemcpyAsync(t.star_backup.p, stars, size_t(nstars) * sizeof(StarRec<T>), cudaMemcpyDeviceToDevice, s));
  long long cap = std::max<long long>(t.cap, nstars + nstars / 2 + 1024);
  t.launches = 0;
  for (int attempt = 0;; attempt++) {
    if (cap > (1LL << 28)) {
      std::fprintf(stderr, "Error. Tree needs more than %lld nodes.\n", 1LL << 28);
      return false;
    }
    if (!tree_build_reserve(t, nstars, int(cap), s) || !leaf_pos.alloc_exact(cap) || !leaf_node.alloc_exact(cap))
      return false;
    if (attempt > 0)
      IRSB_CKR(cudaMemcpyAsync(stars, t.star_backup.p, size_t(nstars) * sizeof(StarRec<T>), cudaMemcpyDeviceToDevice,
                               s));
    if (!launch_tree_build<T>(t, stars, nstars, 1, root_hl, nullptr, nullptr, int(cap), kMaxLevels, leaf_pos.p,
                              leaf_node.p, s))
      return false;
    t.launches++;
    if (!before_sync(cap)) return false;
    if (!tree_status(t, kTreeStatusWords, s)) return false;
    const int* st = t.h_status.p;
    const int err = st[kTreeErr];
    if (st[kTreeBarrier]) {
      std::fprintf(stderr, "Error. The tree build did not finish.\n");
      return false;
    }
    if (err & kErrNodeOverflow) {
      cap *= 2;
      continue;
    }
    if (err & kErrLevelOverflow) {
      std::fprintf(stderr, "Error. Tree exceeded %d levels.\n", kMaxLevels);
      return false;
    }
    if (err) {
      std::fprintf(stderr, "Error. Tree neighbour/interaction list overflow (code %d).\n", err);
      return false;
    }
    t.levels = st[kTreeLevels];
    t.level_off.assign(st + kTreeOff, st + kTreeOff + t.levels + 2);
    t.num_nodes = t.level_off.back();
    t.num_leaves = st[kTreeLeaves];
    return true;
  }
}

}  // namespace irsb
