// Row-list growth: the batched fit's level step without per-feature lists.
//
// A tree keeps one list, its rows in row order.  A node splits on one of the
// m features it selects, so keeping every feature's list sorted per node
// (list growth, ct_level.cu + ct_partition.cu) moves F lists per level for m
// that are scanned.  Here a node's sorted order of a feature is made when the
// node selects it, from the row's rank in the feature's presort (View::pair,
// built once per fit), and only the row list is partitioned.
//
//   k_row_pairs    (rank, value) of every (feature, row)
//   k_row_roots    in-bag rows of each tree, its row list and root node
//                  (reference bootstrap_fill.cu + bootstrap_reshuffle.cu)
//   k_row_select   feature subset of each node: constancy from the node's rows
//   k_row_select_big  the same for large nodes with features that look constant
//   k_row_warp     nodes of at most WARP_ROWS rows: one warp sorts one
//                  (node, feature) in registers and scans it
//   k_row_group    nodes of at most GROUP_ROWS rows: the same by one CTA
//   k_row_bits     larger nodes, by a bitmap over the feature's ranks, which
//                  stands for the sorted list of a node with one row in 64
//   k_row_order    larger nodes that are sparser: their list, from such a bitmap
//   k_row_hist, k_row_carry, k_row_bound, k_row_limit, k_row_scan  the Gini scan
//                  of those lists and bitmaps in pieces (reference compute_2d,
//                  dfs_module.cu:310-443)
//   k_row_reduce   best candidate of each node; node record, children, work list
//   k_row_mark     left flags and class counts; moves the rows of small splits
//   k_row_move     stable split of the row lists of larger ones
//   k_row_children child records for the next step
//   k_row_subtree  subtrees of at most 32 rows, one warp each
//
// Measured on one B200 (ct_fit): 581,012 x 54 covtype-shaped rows, 100 trees
// 62.5 -> 30.6 ms; 10,000 x 3,000 rows, 100 classes, 200 trees 202 -> 30.6 ms
// (the lists of 3,000 features were partitioned per level for 55 scanned); 200,003 x
// 28 continuous columns, 50 trees 14.2 -> 5.3 ms; 1,797 x 64, 50 trees 1.44 ->
// 0.63 ms.  What bounds each kernel stands at it.
//
// Rows of equal value may come in any order in a sorted list: no candidate
// lies between them, and a candidate's class counts depend only on the set of
// rows up to it, so the splits are those of the presorted lists.
#include <algorithm>
#include <cfloat>

#include "ct_items.cuh"

namespace ct {

namespace {

constexpr uint32_t WARP_ROWS = 512;      // nodes up to this size: one warp per (node, feature)
constexpr uint32_t WARP_ROWS_BITS = 9;
constexpr uint32_t GROUP_ROWS = 9216;    // nodes up to this size: one CTA per (node, feature)
constexpr uint32_t GROUP_SMALL_ROWS = 2048;  // the smaller of these nodes take a smaller CTA
constexpr int GROUP_SMALL_WARPS = 8;
constexpr int GROUP_WARPS = 16;
constexpr uint32_t SELECT_ROWS = 2048;   // a selecting warp checks at most this many rows of a larger node
constexpr int ORDER_THREADS = 512;
constexpr uint32_t ORDER_SMEM_MAX = 224u * 1024u;

// Shared memory of k_row_order: the rank bitmap, then a prefix count per word
// (16 bits) or per four words (32 bits) in as many bytes.
__host__ __device__ __forceinline__ uint32_t order_words(uint32_t n_rows) { return ((n_rows + 127) / 128) * 4; }
__host__ __device__ __forceinline__ size_t order_smem(uint32_t n_rows) { return (size_t)order_words(n_rows) * 6; }

// Nodes whose rank bitmap (over all ranks) stands for their sorted list: those
// with at least about one row in 64, so that the bitmap takes no more room
// than the list would (it is kept in the list's place) and a scan meets a row
// in every other word.  Their pieces are runs of ranks.
__host__ __device__ __forceinline__ bool row_dense(uint32_t n, uint32_t n_rows) {
  return n > GROUP_ROWS && 8u * (size_t)n >= (size_t)order_words(n_rows) * 4 + 16;
}
// Ranks of one piece of a bitmap: a power of two of about as many rows as a
// list's piece, at least a 1,024-rank window, at most what 16 bits can list.
__device__ __forceinline__ uint32_t dense_chunk(uint32_t n, uint32_t n_rows, uint32_t scan_piece) {
  const uint64_t ranks = (uint64_t)scan_piece * n_rows / n;
  return ranks >= 32768u ? 32768u : ranks <= 1024u ? 1024u : 1u << (31 - __clz((int)ranks));
}
// Bytes per (node, selected feature, row) that the two cannot do without: a
// row's entry and its rank; its entry, its (rank, value) and its place in the list.
constexpr uint32_t ORDER_BYTES_BITS = 8;
constexpr uint32_t ORDER_BYTES_LIST = 20;
constexpr uint32_t BITS_SLICE = 32768;   // rows per k_row_bits unit
constexpr int BITS_THREADS = 512;
constexpr uint32_t BITS_COUNTS = 4096;   // pieces x classes that k_row_bits counts itself (else k_row_hist does)

__device__ __forceinline__ uint32_t* rank_bits(const View& v, const ct_node& nd, uint32_t slot) {
  return reinterpret_cast<uint32_t*>((reinterpret_cast<uintptr_t>(sorted_list(v, nd.slot, slot) + nd.start) + 15) &
                                     ~uintptr_t(15));
}

constexpr uint32_t SEQ_CLASSES = 8;  // most classes of the lane-sequential scan (seq_scan)

// A candidate's gain n / (nl nr) sum_c (L_c - nl T_c / n)^2 is what its split
// takes off n times the node's Gini impurity: the score is (const - gain) / n,
// so the order of the gains is that of the scores.  Kept as 1 + gain in a
// positive float (whose bits order as it does).  An estimate is off by less
// than 6e-7 of itself (conversions and approximate reciprocals in fp32) plus
// 4e-15 n^2 (fp64 rounding of sums of up to n^2 that cancel).
__device__ __forceinline__ float gain_bound(float known, uint32_t n) {
  return known * (1.0f - 2e-6f) - 8e-15f * (float)n * (float)n;
}
__device__ __forceinline__ float gain_of(double d, float nl, float nr, float n) {
  return 1.0f + (float)d * __fdividef(n, nl * nr);
}
// At a position with `left` class counts, nl rows in all.
__device__ __forceinline__ float gain_at(const uint32_t* left, const uint32_t* total, uint32_t C, uint32_t nl,
                                         uint32_t n) {
  const double t = (double)nl / (double)n;
  double d = 0.0;
  for (uint32_t c = 0; c < C; ++c) {
    const double u = (double)left[c] - t * (double)total[c];
    d += u * u;
  }
  return gain_of(d, (float)nl, (float)(n - nl), (float)n);
}

// Lane holding the warp's lowest (score, pos): two 32-bit minima over the
// score's bits (scores are >= 0 or +inf, so their bits order as they do), one
// over the positions.  All lanes get the lane id; NONE when no lane has a
// finite score.
__device__ __forceinline__ uint32_t warp_best_lane(double score, uint32_t pos) {
  const uint64_t b = (uint64_t)__double_as_longlong(score);
  const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b;
  const uint32_t mhi = __reduce_min_sync(FULL, hi);
  if (mhi >= 0x7ff00000u) return NONE;
  const uint32_t mlo = __reduce_min_sync(FULL, hi == mhi ? lo : 0xffffffffu);
  const bool tie = hi == mhi && lo == mlo;
  const uint32_t mp = __reduce_min_sync(FULL, tie ? pos : 0xffffffffu);
  return (uint32_t)__ffs(__ballot_sync(FULL, tie && pos == mp)) - 1;
}

// Exact score of a candidate (the scan's arithmetic, ct_level.cu).
struct Scored {
  double score;
  uint32_t pure;
};
__device__ __forceinline__ Scored score_at(int64_t sl, int64_t sr, uint32_t nl, double nn) {
  const double l = (double)nl;
  const double gl = gini_part(sl, l, nn);
  const double gr = gini_part(sr, __dsub_rn(nn, l), nn);
  return Scored{__dadd_rn(gl, gr), (gl == 0.0 ? 1u : 0u) | (gr == 0.0 ? 2u : 0u)};
}

// ------------------------------------------------------------------------
// (rank, value bits) by row and (value bits, label) by rank, of the features
// that keep a presort order.
template <typename IdxT, typename LabT>
__global__ void k_row_pairs(const IdxT* __restrict__ presort, const float* __restrict__ x_fm,
                            const LabT* __restrict__ labels, uint32_t n, uint64_t vmask, uint2* __restrict__ pair,
                            uint2* __restrict__ ranked, uint32_t* __restrict__ rank) {
  const uint32_t f = blockIdx.y;
  if (f < 64 && ((vmask >> f) & 1ull)) return;
  const size_t off = (size_t)f * n;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const uint32_t row = presort[off + p];
    const uint32_t x = __float_as_uint(__ldg(x_fm + off + row));
    pair[off + row] = make_uint2(p, x);
    if (rank) rank[off + row] = p;
    if (ranked) ranked[off + p] = make_uint2(x, (uint32_t)__ldg(labels + row));
  }
}

// Class of the first row, in feature 0's order, of `n` listed rows: the leaf
// rule.  Warp-collective.
__device__ __forceinline__ uint32_t first_row_class(const View& v, const uint32_t* rows, uint32_t n) {
  uint64_t best = ~0ull;
  for (uint32_t i0 = 0; i0 < n; i0 += 32 * 8) {
    uint32_t e[8], k[8];
#pragma unroll
    for (uint32_t r = 0; r < 8; ++r) {
      const uint32_t i = i0 + r * 32 + lane_id();
      e[r] = i < n ? rows[i] : NONE;
    }
#pragma unroll
    for (uint32_t r = 0; r < 8; ++r) k[r] = i0 + r * 32 + lane_id() < n ? v.pair[entry_row(v, e[r])].x : NONE;
#pragma unroll
    for (uint32_t r = 0; r < 8; ++r)
      if (i0 + r * 32 + lane_id() < n) best = min(best, ((uint64_t)k[r] << 32) | (e[r] >> v.lab_shift));
  }
  const uint32_t hi = (uint32_t)(best >> 32);
  const uint32_t m = __reduce_min_sync(FULL, hi);
  return __reduce_min_sync(FULL, hi == m ? (uint32_t)best : NONE);
}

__device__ __forceinline__ void write_leaf(const TreeView& tv, size_t at, uint32_t value) {
  tv.left[at] = 0;
  tv.right[at] = 0;
  tv.feature[at] = 0;
  tv.threshold[at] = 0.f;
  tv.value[at] = value;
}

// One CTA per tree: the in-bag rows as a bitmap in shared memory (a draw is
// one atomic there), then the row list in row order, the root's class counts
// and its record (a leaf if it holds fewer than min_samples_split rows).
template <typename LabT>
__global__ void __launch_bounds__(1024) k_row_roots(View v, uint64_t seed, uint32_t bootstrap, uint32_t slot_lo,
                                                    uint32_t tree_lo, uint32_t* n_in, TreeView tv, ct_node* out,
                                                    uint32_t* out_tot, uint32_t cap, Counters* ctr,
                                                    uint64_t* out_mask, const float2* vals) {
  extern __shared__ __align__(16) uint32_t root_smem[];
  __shared__ uint32_t s_wcnt[32];
  __shared__ uint32_t s_idx, s_min;
  const uint32_t slot = slot_lo + blockIdx.x, N = v.n_rows, C = v.n_classes;
  const uint32_t words = (N + 31) / 32;
  uint32_t* bm = root_smem;
  uint32_t* hist = root_smem + words;
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const LabT* labels = reinterpret_cast<const LabT*>(v.labels);
  for (uint32_t w = threadIdx.x; w < words; w += blockDim.x)
    bm[w] = bootstrap ? 0u : (w * 32 + 32 <= N ? FULL : (1u << (N & 31)) - 1u);
  for (uint32_t c = threadIdx.x; c < C; c += blockDim.x) hist[c] = 0;
  __syncthreads();
  const uint64_t tkey = tree_key(seed, tree_lo + blockIdx.x);
  if (bootstrap) {
    const uint64_t bk = boot_key(tkey);
    for (uint32_t i = threadIdx.x; i < N; i += blockDim.x) {
      const uint32_t r = boot_draw(bk, i, N);
      atomicOr(&bm[r >> 5], 1u << (r & 31));
    }
    __syncthreads();
  }
  const uint32_t per = ceil_div(words, nwarps);
  const uint32_t wlo = min(warp * per, words), whi = min(wlo + per, words);
  uint32_t c = 0;
  for (uint32_t w = wlo + lane; w < whi; w += 32) c += __popc(bm[w]);
  c = __reduce_add_sync(FULL, c);
  if (lane == 0) s_wcnt[warp] = c;
  __syncthreads();
  uint32_t pos = 0, n = 0;
  for (uint32_t k = 0; k < nwarps; ++k) {
    pos += k < warp ? s_wcnt[k] : 0u;
    n += s_wcnt[k];
  }
  uint32_t* rows = row_list(v, 0, slot);
  const unsigned lt = lanemask_lt();
  for (uint32_t w0 = wlo; w0 < whi; w0 += 4) {
    uint32_t lab[4], bits[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      bits[k] = w0 + k < whi ? bm[w0 + k] : 0u;
      lab[k] = (bits[k] >> lane) & 1u ? (uint32_t)labels[(w0 + k) * 32 + lane] : NONE;
    }
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      const unsigned grp = __match_any_sync(FULL, lab[k]);
      if (lab[k] != NONE) {
        rows[pos + __popc(bits[k] & lt)] = ((w0 + k) * 32 + lane) | (lab[k] << v.lab_shift);
        if ((grp & lt) == 0u) atomicAdd(&hist[lab[k]], (uint32_t)__popc(grp));
      }
      pos += __popc(bits[k]);
    }
  }
  if (threadIdx.x == 0) {
    s_idx = NONE;
    s_min = NONE;
    n_in[slot] = n;
    tv.n_nodes[slot + tv.slot_base] = 1;
    if (n >= v.mss && n > 0) {
      const uint32_t idx = atomicAdd(&ctr->n_next, 1u);
      if (idx < cap) {
        ct_node nd;
        nd.slot = slot;
        nd.start = 0;
        nd.n = n;
        nd.raw_id = 0;
        nd.key = root_key(tkey);
        nd.impurity = 1.0f;
        nd.buf = 0;
        out[idx] = nd;
        atomicAdd(&ctr->next_total, (unsigned long long)n);
        s_idx = idx;
      } else {
        atomicOr(&ctr->error, DEV_ERR_CAPACITY);
      }
    }
  }
  __syncthreads();
  if (s_idx != NONE) {
    for (uint32_t k = threadIdx.x; k < C; k += blockDim.x) out_tot[(size_t)s_idx * C + k] = hist[k];
    if (out_mask)  // features constant over the whole data
      for (uint32_t k = threadIdx.x; k < mask_words(v.n_features); k += blockDim.x) {
        uint64_t m = 0;
        for (uint32_t f = k * 64; f < min(k * 64 + 64, v.n_features); ++f)
          m |= (uint64_t)(vals[f].x == vals[f].y) << (f & 63);
        out_mask[(size_t)s_idx * v.mask_stride + k] = m;
      }
  } else if (n < v.mss || n == 0) {  // a leaf: the class of its first row in feature 0's order
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) atomicMin(&s_min, v.pair[entry_row(v, rows[i])].x);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
      if (v.pair[entry_row(v, rows[i])].x == s_min)
        write_leaf(tv, (size_t)(slot + tv.slot_base) * tv.capacity, rows[i] >> v.lab_shift);
    if (n == 0 && threadIdx.x == 0) write_leaf(tv, (size_t)(slot + tv.slot_base) * tv.capacity, 0u);
  }
}

// ------------------------------------------------------------------------
// Selection.  The first m non-constant features of the node's permutation
// (the rule of k_select); a feature varies in a node when two of its rows
// differ in it.  A lane takes one feature and compares four of the node's
// rows, which settles nearly every feature that varies; the others are read
// row by row (CTA: by the whole block) until two values differ.  Features
// found constant go into the node's mask, which its descendants inherit.
template <bool CTA>
__device__ __forceinline__ bool rows_vary(const View& v, const uint32_t* rows, const float* xf, uint32_t n, float x0) {
  const uint32_t tid = CTA ? threadIdx.x : lane_id(), nt = CTA ? blockDim.x : 32u;
  for (uint32_t i0 = 0; i0 < n; i0 += nt * 4) {
    bool d = false;
    uint32_t r[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      const uint32_t i = i0 + k * nt + tid;
      r[k] = i < n ? entry_row(v, rows[i]) : NONE;
    }
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) d |= r[k] != NONE && __ldg(xf + (r[k] != NONE ? r[k] : 0u)) != x0;
    if (CTA ? __syncthreads_or(d) : __any_sync(FULL, d)) return true;
  }
  return false;
}

// Zeroes a bitmap that several slices fill, and its pieces' class counts.
__device__ __forceinline__ void zero_bits(const View& v, const ct_node& nd, uint32_t slot, uint32_t* counts, uint32_t nc,
                                          uint32_t tid, uint32_t nt) {
  uint4* b4 = reinterpret_cast<uint4*>(rank_bits(v, nd, slot));
  for (uint32_t g = tid; g < order_words(v.n_rows) / 4; g += nt) b4[g] = make_uint4(0u, 0u, 0u, 0u);
  if (nc <= BITS_COUNTS)
    for (uint32_t i = tid; i < nc; i += nt) counts[i] = 0;
}

// CTA: every warp of the block selects alike, warp 0 writes.
template <bool Q, bool CTA>
__device__ __forceinline__ void row_select_item(const View& vb, const StepLists& lists, const LevelScratch& s,
                                                uint32_t w) {
  const uint32_t lane = lane_id();
  const ct_node nd = lists.nodes[w];
  CT_JOB_REF(v, vb, nd.slot);
  const uint32_t m = v.max_features, n = nd.n;
  const bool writer = !CTA || threadIdx.x < 32;
  uint64_t* cmask = lists.node_mask ? const_cast<uint64_t*>(lists.node_mask) + (size_t)w * v.mask_stride : nullptr;
  const uint32_t* rows = row_list(v, nd.buf, nd.slot) + nd.start;
  const uint32_t limit = CTA || n <= SELECT_ROWS ? n : SELECT_ROWS;
  uint32_t taken = 0;
  uint64_t vsel = 0;  // selected slots that hold virtual features (m <= 64 when there are any)
  if (n >= 2) {
    uint32_t r[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) r[j] = entry_row(v, rows[(uint64_t)j * (n - 1) / 3]);
    for (uint32_t i0 = 0; i0 < v.n_features && taken < m; i0 += 32) {
      const uint32_t i = i0 + lane;
      bool usable = false, virt = false, unknown = false;
      uint32_t f = 0;
      if (i < v.n_features) {
        f = feature_perm(i, v.n_features, nd.key, v.feistel_h);
        virt = is_virtual(v, f);
        if (virt) {  // some but not all rows take the high value
          const uint32_t nb = s.vcnt[(size_t)w * 64 + f];
          usable = nb > 0 && nb < n;
        } else if (!mask_bit(cmask, f)) {
          const float* xf = v.x_fm + (size_t)f * v.n_rows;
          const float x0 = xf[r[0]];
          usable = xf[r[1]] != x0 || xf[r[2]] != x0 || xf[r[3]] != x0;
          unknown = !usable && n > 4;
        }
      }
      unsigned ok = __ballot_sync(FULL, usable);
      for (unsigned um = __ballot_sync(FULL, unknown); um; um &= um - 1) {
        const uint32_t u = (uint32_t)__ffs(um) - 1;
        if (taken + __popc(ok & ((1u << u) - 1u)) >= m) break;
        const uint32_t fu = __shfl_sync(FULL, f, u);
        const float* xf = v.x_fm + (size_t)fu * v.n_rows;
        if (rows_vary<CTA>(v, rows, xf, limit, xf[r[0]])) {
          ok |= 1u << u;
        } else if (limit < n) {  // undecided: the block form selects for this node
          if (lane == 0) {
            const uint32_t b = atomicAdd(&s.ctr->n_big_segs, 1u);
            if (b < s.cap_big) s.big_nodes[b] = w;
            else atomicOr(&s.ctr->error, DEV_ERR_CAPACITY);
          }
          return;
        } else if (cmask && writer && lane == 0) {
          cmask[fu >> 6] |= 1ull << (fu & 63);
        }
      }
      usable = (ok >> lane) & 1u;
      const uint32_t rank = __popc(ok & lanemask_lt());
      const bool keep = usable && taken + rank < m;
      if (keep && writer) s.sel[(size_t)w * v.sel_stride + taken + rank] = f;
      const uint64_t b = (keep && virt) ? 1ull << ((taken + rank) & 63) : 0ull;
      vsel |= ((uint64_t)__reduce_or_sync(FULL, (uint32_t)(b >> 32)) << 32) | __reduce_or_sync(FULL, (uint32_t)b);
      taken += min((uint32_t)__popc(ok), m - taken);
    }
  }
  if (!writer) return;
  // work items of the slots that need a sorted order (virtual ones are scored from counts)
  const uint32_t tmat = taken - (uint32_t)__popcll(vsel);
  const bool small = n <= WARP_ROWS, group = !small && n <= GROUP_ROWS, dense = row_dense(n, v.n_rows);
  const bool narrow = n <= GROUP_SMALL_ROWS;
  const uint32_t pps = small || group ? 1u : dense ? ceil_div(v.n_rows, dense_chunk(n, v.n_rows, lists.scan_piece)) : ceil_div(n, lists.scan_piece);
  const uint32_t slices = dense ? ceil_div(n, BITS_SLICE) : 0u;
  // the largest gain of the node's virtual candidates: a start for its scans' bound
  uint32_t q0 = 0;
  if (vsel && !small && vb.n_classes <= SEQ_CLASSES) {
    __syncwarp();  // the slots' features, written by other lanes
    for (uint32_t q = lane; q < taken; q += 32) {
      if (!((vsel >> q) & 1ull)) continue;
      const uint32_t f = s.sel[(size_t)w * v.sel_stride + q];
      if (!is_candidate_sorted(v.vval[f].x, v.vval[f].y)) continue;
      // from the high-value rows' counts: the gain is the same from either side
      const float e = gain_at(s.vcls + ((size_t)w * v.n_features + f) * v.n_classes,
                                 lists.tot + (size_t)w * v.n_classes, v.n_classes, s.vcnt[(size_t)w * 64 + f], n);
      q0 = max(q0, __float_as_uint(e));
    }
    q0 = __reduce_max_sync(FULL, q0);
  }
  uint32_t base = 0, obase = 0, zbase = 0, cbase = 0, ok = 1;
  if (lane == 0) {
    if (tmat) {
      atomicAdd(&s.ctr->scan_elems, (unsigned long long)tmat * n);
      if (small) {
        base = atomicAdd(&s.ctr->n_small_segs, tmat);
        ok = base + (uint64_t)tmat <= s.cap_w;
      } else if (group) {
        base = atomicAdd(narrow ? &s.ctr->n_huge_segs : &s.ctr->n_hchains, tmat);
        ok = base + (uint64_t)tmat <= s.cap_order;
      } else {
        base = atomicAdd(&s.ctr->n_scan_pieces, tmat * pps);
        ok = base + (uint64_t)tmat * pps <= s.cap_scan;
        atomicAdd(&s.ctr->order_bytes, (unsigned long long)tmat * n * (dense ? ORDER_BYTES_BITS : ORDER_BYTES_LIST));
        if (pps > 1) {
          cbase = atomicAdd(&s.ctr->n_bchains, tmat);
          ok = ok && cbase + (uint64_t)tmat <= s.cap_order;
        }
        if (dense) {
          obase = atomicAdd(&s.ctr->n_tv, tmat * slices);
          if (!CTA && slices > 1) zbase = atomicAdd(&s.ctr->n_tiles, tmat);
          ok = ok && obase + (uint64_t)tmat * slices <= s.cap_units && zbase + (uint64_t)tmat <= s.cap_order;
        } else {
          obase = atomicAdd(&s.ctr->n_carry, tmat);
          ok = ok && obase + (uint64_t)tmat <= s.cap_order;
        }
      }
      if (!ok) atomicOr(&s.ctr->error, DEV_ERR_CAPACITY);
    }
    s.nsel[w] = taken;
    s.node_q[w] = q0;
    s.piece_base[w] = base;
    s.piece_cnt[w] = small || group || !ok ? 0u : tmat * pps;
  }
  base = __shfl_sync(FULL, base, 0);
  obase = __shfl_sync(FULL, obase, 0);
  zbase = __shfl_sync(FULL, zbase, 0);
  cbase = __shfl_sync(FULL, cbase, 0);
  ok = __shfl_sync(FULL, ok, 0);
  if (!ok) return;
  for (uint32_t k = 0; k < tmat; ++k) {  // k-th slot with a list
    uint32_t slot = k;
    if (vsel) {
      slot = 0;
      for (uint32_t left = k;; ++slot)
        if (!((vsel >> slot) & 1ull) && left-- == 0) break;
    }
    if (small) {
      if (lane == (k & 31u)) s.witems[base + k] = make_uint2(w, slot);
      continue;
    }
    if (group) {
      if (lane == (k & 31u)) (narrow ? s.gsmall : s.glarge)[base + k] = make_uint2(w, slot);
      continue;
    }
    const uint32_t pb = base + k * pps;  // its first piece
    for (uint32_t j = lane; j < pps; j += 32) s.rpieces[pb + j] = RowPiece{w, slot, j, pps};
    if (pps > 1 && lane == 0) s.citems[cbase + k] = make_uint2(pb, pps);
    if (dense) {
      for (uint32_t j = lane; j < slices; j += 32)
        s.bunits[obase + k * slices + j] = make_uint4(w, slot, j | (slices << 16), pb);
      if (slices > 1 && lane == 0 && !CTA) s.bzero[zbase + k] = make_uint4(w, slot, pb, pps);
      if (slices > 1 && CTA)  // a node the block form selects for: zeroed here
        zero_bits(v, nd, slot, s.carry + (size_t)pb * vb.n_classes, pps * vb.n_classes, lane, 32);
    } else if (lane == 0) {
      s.oitems[obase + k] = make_uint2(w, slot);
    }
  }
}

template <bool Q>
__global__ void __launch_bounds__(THREADS_PER_BLOCK) k_row_select(View v, LevelScratch s) {
  const uint32_t count = min(s.ctr->n_nodes, s.cap_nodes);
  const StepLists sl = *s.step;
  for_items(count, &s.ctr->claim[ITEM_SELECT], [&](uint32_t w) { row_select_item<Q, false>(v, sl, s, w); });
}

template <bool Q>
__global__ void __launch_bounds__(512) k_row_select_big(View v, LevelScratch s) {
  const uint32_t count = live_count(s, s.ctr->n_big_segs, s.cap_big);
  const StepLists sl = *s.step;
  for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
    row_select_item<Q, true>(v, sl, s, s.big_nodes[i]);
    __syncthreads();
  }
  // bitmaps that several slices fill
  const uint32_t zeros = live_count(s, s.ctr->n_tiles, s.cap_order);
  for (uint32_t i = blockIdx.x; i < zeros; i += gridDim.x) {
    const uint4 z = s.bzero[i];
    const ct_node nd = sl.nodes[z.x];
    CT_JOB_REF(vj, v, nd.slot);
    zero_bits(vj, nd, z.y, s.carry + (size_t)z.z * v.n_classes, z.w * v.n_classes, threadIdx.x, blockDim.x);
  }
}

// ------------------------------------------------------------------------
// Rank bitmap of a dense (node, feature): one CTA per slice of the node's rows
// sets their rank's bits in shared memory, and counts the classes of each
// piece's rows there.  A node of one slice stores its words and counts; the
// slices of a larger one merge theirs into the zeroed bitmap and counts with
// one coalesced atomic per non-empty word.  Bound by the gather of the ranks: a
// 32-byte sector serves 8 rows in row order, 1 to 5 of them in the node.  The
// classes counted here replace a pass over the sorted rows: covtype-shaped, 100
// trees, 9.0 ms with ranks gathered from the (rank, value) pairs plus 5.8 ms of
// counting -> 4.9 ms.
__host__ __device__ __forceinline__ uint32_t bits_words(uint32_t n_rows) { return order_words(n_rows) + BITS_COUNTS; }

template <bool Q>
__global__ void __launch_bounds__(BITS_THREADS, 2) k_row_bits(View vb, LevelScratch s, uint32_t n_max) {
  extern __shared__ __align__(16) uint32_t bits_sm[];
  __shared__ uint32_t s_item;
  const uint32_t count = live_count(s, s.ctr->n_tv, s.cap_units);
  const StepLists lists = *s.step;
  constexpr uint32_t T = BITS_THREADS, U = 8;
  const uint32_t C = vb.n_classes;
  uint4* bm4 = reinterpret_cast<uint4*>(bits_sm);
  uint32_t* hist = bits_sm + order_words(n_max);
  while (true) {
    __syncthreads();  // the previous unit is done with the bitmap and s_item
    if (threadIdx.x == 0) s_item = atomicAdd(&s.ctr->claim[ITEM_BITS], 1u);
    __syncthreads();
    if (s_item >= count) break;
    const uint4 unit = s.bunits[s_item];
    const uint32_t slice = unit.z & 0xffffu, slices = unit.z >> 16;
    const ct_node nd = lists.nodes[unit.x];
    CT_JOB_REF(v, vb, nd.slot);
    const uint32_t f = s.sel[(size_t)unit.x * v.sel_stride + unit.y];
    const uint32_t* rows = row_list(v, nd.buf, nd.slot) + nd.start;
    const uint32_t* rf = v.rank + (size_t)f * v.n_rows;
    const uint32_t groups = order_words(v.n_rows) / 4;
    const uint32_t chunk = dense_chunk(nd.n, v.n_rows, lists.scan_piece), csh = 31 - __clz((int)chunk);
    const uint32_t nc = ceil_div(v.n_rows, chunk) * C;
    const bool counts = nc <= BITS_COUNTS;
    const uint32_t lo = slice * BITS_SLICE, hi = min(lo + BITS_SLICE, nd.n);
    for (uint32_t g = threadIdx.x; g < groups; g += T) bm4[g] = make_uint4(0u, 0u, 0u, 0u);
    if (counts)
      for (uint32_t i = threadIdx.x; i < nc; i += T) hist[i] = 0;
    __syncthreads();
    for (uint32_t i0 = lo + threadIdx.x; i0 < hi; i0 += T * U) {
      uint32_t e[U], r[U];
#pragma unroll
      for (uint32_t k = 0; k < U; ++k) e[k] = i0 + k * T < hi ? rows[i0 + k * T] : 0u;
#pragma unroll
      for (uint32_t k = 0; k < U; ++k) r[k] = i0 + k * T < hi ? __ldg(rf + entry_row(v, e[k])) : 0u;
#pragma unroll
      for (uint32_t k = 0; k < U; ++k)
        if (i0 + k * T < hi) {
          atomicOr(&bits_sm[r[k] >> 5], 1u << (r[k] & 31));
          if (counts) atomicAdd(&hist[(r[k] >> csh) * C + (e[k] >> v.lab_shift)], 1u);
        }
    }
    __syncthreads();
    uint4* out = reinterpret_cast<uint4*>(rank_bits(v, nd, unit.y));
    uint32_t* oc = s.carry + (size_t)unit.w * C;
    if (slices == 1) {
      for (uint32_t g = threadIdx.x; g < groups; g += T) out[g] = bm4[g];
      if (counts)
        for (uint32_t i = threadIdx.x; i < nc; i += T) oc[i] = hist[i];
    } else {
      uint32_t* ow = reinterpret_cast<uint32_t*>(out);
      for (uint32_t w = threadIdx.x; w < groups * 4; w += T)
        if (const uint32_t b = bits_sm[w]) atomicOr(ow + w, b);
      if (counts)
        for (uint32_t i = threadIdx.x; i < nc; i += T)
          if (const uint32_t t = hist[i]) atomicAdd(oc + i, t);
    }
  }
}

// ------------------------------------------------------------------------
// Scan of a run of at most SEQ_ROWS sorted rows with at most SEQ_CLASSES
// classes: the rows lie in shared memory so that lane l walks the l-th piece
// of 2^k consecutive ones.  First every lane counts its rows' classes in 8-bit
// fields of two registers; a prefix over the lanes gives each its left class
// counts and sums at its first row; then each updates them row by row, with no
// exchange between lanes.  The exact score costs more than the rest of a step,
// so a step only estimates the candidate's gain (gain_of) and the walk keeps
// the largest.  Only a lane whose largest gain reaches the best known for the
// node within the estimate's error walks again, and there the candidates
// within that error are scored exactly: one further below can neither win nor
// tie.
constexpr uint32_t SEQ_ROWS = 512;

// A run of `count` rows, 2^sh per lane: row i sits at (i >> sh) lanes of
// 2^sh + 1 entries (no bank conflicts between lanes).
__device__ __forceinline__ uint32_t seq_shift(uint32_t count) {  // count <= SEQ_ROWS
  return count <= 32 ? 0u : 27u - (uint32_t)__clz((int)(count - 1));
}
__device__ __forceinline__ uint32_t seq_at(uint32_t i, uint32_t sh) { return i + (i >> sh); }
constexpr uint32_t SEQ_SLOTS = SEQ_ROWS + 32;    // entries of a run, at the most
// Shared memory of one warp, in words: 2 L + 1 per (class, lane), the class
// totals as doubles, the class counts before the run, the class totals.
constexpr uint32_t SEQ_TAB = SEQ_CLASSES * 32;
constexpr uint32_t SEQ_BEFORE = SEQ_TAB + 2 * SEQ_CLASSES;
constexpr uint32_t SEQ_WORDS = SEQ_BEFORE + 2 * SEQ_CLASSES;

struct SeqBest {
  double score;
  uint32_t pos;
  uint32_t pure;
  float xl;
  float xr;
};

// An entry: (value bits, 8 x label).
__device__ __forceinline__ uint2 seq_entry(uint32_t x, uint32_t label) { return make_uint2(x, label << 3); }

// 1 << s, 0 for s >= 32 (also when s wrapped below 0).
__device__ __forceinline__ uint32_t shl_clamp(uint32_t s) {
  uint32_t r;
  asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(s));
  return r;
}

// This lane's class counts as 8-bit fields, spread over pairs of 16-bit
// fields: word h of class c is (c >> 2) * 2 + (c & 1), its half (c >> 1) & 1.
__device__ __forceinline__ void seq_count(const uint2* run, uint32_t m, uint32_t (&w)[4]) {
  uint32_t lo = 0, hi = 0;
#pragma unroll 4
  for (uint32_t j = 0; j < m; ++j) {
    const uint32_t c8 = run[j].y;
    lo += shl_clamp(c8);
    hi += shl_clamp(c8 - 32);
  }
  w[0] = lo & 0x00ff00ffu;
  w[1] = (lo >> 8) & 0x00ff00ffu;
  w[2] = hi & 0x00ff00ffu;
  w[3] = (hi >> 8) & 0x00ff00ffu;
}
__device__ __forceinline__ uint32_t seq_field(const uint32_t (&w)[4], uint32_t c) {
  return (w[(c >> 2) * 2 + (c & 1u)] >> (((c >> 1) & 1u) * 16)) & 0xffffu;
}

// The class totals of the node, for seq_scan; before[] is the caller's.
__device__ __forceinline__ void seq_totals(uint32_t* sq, const uint32_t* tot, uint32_t C) {
  const uint32_t lane = lane_id();
  if (lane < SEQ_CLASSES) {
    const uint32_t t = lane < C ? tot[lane] : 0u;
    reinterpret_cast<double*>(sq + SEQ_TAB)[lane] = (double)t;
    sq[SEQ_BEFORE + SEQ_CLASSES + lane] = t;
  }
}

// The scan of a run at positions p0.. of the node's order.  run: this lane's
// m rows; w: their counts (seq_count); sq: the warp's tables, with the totals
// and the class counts before the run set; the latter are advanced past the
// run here.  xp: the value before the lane's first row (its own value when
// there is none).  node_q: the largest gain known for the node, kept by all of
// its scans.
__device__ __forceinline__ void seq_scan(const uint2* run, uint32_t m, uint32_t sh, const uint32_t (&w)[4], uint32_t* sq,
                                         uint32_t C, float xp, uint32_t p0, uint32_t n, uint32_t* node_q, SeqBest& bb) {
  const uint32_t lane = lane_id();
  uint32_t* tab = sq + lane;
  const double* tt = reinterpret_cast<const double*>(sq + SEQ_TAB);
  uint32_t* before = sq + SEQ_BEFORE;
  const uint32_t* total = before + SEQ_CLASSES;
  uint32_t ex[4], tot[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) {  // words 0 and 1 hold classes 0-3, 2 and 3 classes 4-7
    ex[h] = tot[h] = 0;
    if (h < 2 || C > 4) {
      const uint32_t incl = (uint32_t)warp_incl_scan_i32((int32_t)w[h]);
      ex[h] = incl - w[h];
      tot[h] = __shfl_sync(FULL, incl, 31);
    }
  }
  int64_t sl = 0, a = 0, st2 = 0;  // sums of L^2, L T, T^2
#pragma unroll
  for (uint32_t c = 0; c < SEQ_CLASSES; ++c) {
    if (c >= C) break;
    const uint32_t l = before[c] + seq_field(ex, c), t = total[c];
    tab[c * 32] = 2 * l + 1;
    sl += (int64_t)l * l;
    a += (int64_t)l * t;
    st2 += (int64_t)t * t;
  }
  __syncwarp();
  if (lane < C) before[lane] += seq_field(tot, lane);
  const uint32_t k0 = p0 + (lane << sh);
  const double inv = 1.0 / (double)n, std2 = (double)st2;
  const float nf = (float)n;
  float gmax = 0.f;
  {
    double s = (double)sl, a2 = -2.0 * (double)a, nl = (double)k0;
    float nlf = (float)k0, nrf = nf - nlf, x0 = xp;  // exact: n < 2^24
#pragma unroll 2
    for (uint32_t j = 0; j < m; ++j) {
      const uint2 e = run[j];
      const float x = __uint_as_float(e.x);
      uint32_t* t = tab + (e.y << 2);
      const uint32_t d = *t;
      const double r = nl * inv;
      const float g = gain_of(fma(r, fma(r, std2, a2), s), nlf, nrf, nf);
      if (is_candidate_sorted(x0, x)) gmax = fmaxf(gmax, g);
      *t = d + 2;
      s += (double)d;
      a2 = fma(-2.0, tt[e.y >> 3], a2);
      nl += 1.0;
      nlf += 1.f;
      nrf -= 1.f;
      x0 = x;
    }
  }
  const uint32_t gw = __reduce_max_sync(FULL, __float_as_uint(gmax));
  uint32_t known = 0;
  if (lane == 0 && gw) known = atomicMax(node_q, gw);
  known = max(__shfl_sync(FULL, known, 0), gw);
  const float bound = gain_bound(__uint_as_float(known), n);
  if (gmax > 0.f && gmax >= bound) {  // this lane holds such a candidate
    for (uint32_t j = m; j > 0; --j) tab[run[j - 1].y << 2] -= 2;  // the counts at the lane's first row again
    const double nn = (double)n;
    for (uint32_t j = 0; j < m; ++j) {
      const uint2 e = run[j];
      const float x = __uint_as_float(e.x);
      uint32_t* t = tab + (e.y << 2);
      const uint32_t d = *t, k = k0 + j;
      if (is_candidate_sorted(xp, x)) {
        const double r = (double)k * inv;
        const float g = gain_of(fma(r, fma(r, std2, -2.0 * (double)a), (double)sl), (float)k, nf - (float)k, nf);
        if (g >= bound) {
          const Scored sc = score_at(sl, st2 - 2 * a + sl, k, nn);
          if (sc.score < bb.score) bb = SeqBest{sc.score, k - 1, sc.pure, xp, x};
        }
      }
      *t = d + 2;
      sl += d;
      a += total[e.y >> 3];
      xp = x;
    }
  }
  __syncwarp();
}

// ------------------------------------------------------------------------
// Small nodes: one warp per (node, feature).  Sort keys are the row's rank in
// the feature's presort above its index in the node (ranks are distinct), in
// 32 bits.  Lane l ends up with the K consecutive sorted positions from l K
// on, so a bitonic sort exchanges between lanes in 15 steps only, whatever K.
// The steps are loops: the unrolled networks of all sizes (and their scans)
// overflowed the instruction cache (16 of 25 stall cycles per instruction).
template <int K>
__device__ __forceinline__ void lane_sort(uint32_t (&v)[K]) {  // ascending, within the lane
#pragma unroll
  for (int size = 2; size <= K; size <<= 1)
#pragma unroll
    for (int j = size >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (k & j) continue;
        const bool up = (k & size) == 0;
        const uint32_t x = v[k], y = v[k | j];
        v[k] = up ? min(x, y) : max(x, y);
        v[k | j] = up ? max(x, y) : min(x, y);
      }
}
template <int K>
__device__ __forceinline__ void lane_merge(uint32_t (&v)[K]) {  // bitonic -> ascending, within the lane
#pragma unroll
  for (int j = K >> 1; j > 0; j >>= 1)
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (k & j) continue;
      const uint32_t x = v[k], y = v[k | j];
      v[k] = min(x, y);
      v[k | j] = max(x, y);
    }
}
template <int K>
__device__ __forceinline__ void warp_sort_keys(uint32_t (&v)[K], uint32_t lane) {
  uint32_t flip = 0u - (lane & 1u);  // lanes sorting downwards hold complements
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] ^= flip;
  lane_sort<K>(v);
#pragma unroll 1
  for (uint32_t g = 2; g <= 32; g <<= 1) {
    const uint32_t next = lane & g ? FULL : 0u;  // (g = 32: ascending everywhere)
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] ^= flip ^ next;
    flip = next;
#pragma unroll 1
    for (uint32_t j = g >> 1; j > 0; j >>= 1) {
      const bool lower = (lane & j) == 0u;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const uint32_t o = __shfl_xor_sync(FULL, v[k], j);
        v[k] = lower ? min(v[k], o) : max(v[k], o);
      }
    }
    lane_merge<K>(v);
  }
}

// Shared memory of one warp: the node's rows as seq entries, sorted in place,
// then the scan's tables.
__host__ __device__ __forceinline__ uint32_t warp_item_words(uint32_t n_classes) {
  return 2 * SEQ_SLOTS + (n_classes <= SEQ_CLASSES ? SEQ_WORDS : ((n_classes + 1) / 2 + 3u) & ~3u);
}

// Loads the node's rows and leaves them sorted in ent (seq_at addressing, K
// rows per lane); second word 8 x label, or label | class total << 16.
template <int K>
__device__ __forceinline__ void row_warp_sort(const View& v, const uint32_t* tot, const uint32_t* rows, uint32_t n,
                                              const uint2* pf, bool seq, uint2* ent) {
  const uint32_t lane = lane_id();
  uint32_t key[K];
  {
    uint32_t e[K];
    uint2 pr[K];
#pragma unroll
    for (int k = 0; k < K; ++k) e[k] = 32 * k + lane < n ? rows[32 * k + lane] : 0u;
#pragma unroll
    for (int k = 0; k < K; ++k) pr[k] = 32 * k + lane < n ? __ldg(pf + entry_row(v, e[k])) : make_uint2(0u, 0u);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const uint32_t i = 32 * k + lane;
      key[k] = NONE;
      if (i < n) {
        const uint32_t lab = e[k] >> v.lab_shift;
        key[k] = (pr[k].x << WARP_ROWS_BITS) | i;
        ent[i] = seq ? seq_entry(pr[k].y, lab) : make_uint2(pr[k].y, lab | (__ldg(tot + lab) << 16));
      }
    }
  }
  warp_sort_keys<K>(key, lane);
  __syncwarp();
  uint2 r[K];
#pragma unroll
  for (int k = 0; k < K; ++k) r[k] = ent[key[k] & (WARP_ROWS - 1)];
  __syncwarp();
#pragma unroll
  for (int k = 0; k < K; ++k) ent[lane * (K + 1) + k] = r[k];
  __syncwarp();
}

template <bool Q>
__device__ __forceinline__ void row_warp_item(const View& vb, const StepLists& lists, const LevelScratch& s,
                                              uint32_t* smem, uint32_t i) {
  const uint2 it = s.witems[i];
  const ct_node nd = lists.nodes[it.x];
  CT_JOB_REF(v, vb, nd.slot);
  const uint32_t lane = lane_id(), C = vb.n_classes, n = nd.n;
  const uint32_t f = s.sel[(size_t)it.x * v.sel_stride + it.y];
  const uint32_t* rows = row_list(v, nd.buf, nd.slot) + nd.start;
  const uint2* pf = v.pair + (size_t)f * v.n_rows;
  const uint32_t* tot = lists.tot + (size_t)it.x * C;
  RowBest* out = s.rbest + (size_t)it.x * v.sel_stride + it.y;
  uint2* ent = reinterpret_cast<uint2*>(smem);
  const bool seq = C <= SEQ_CLASSES;
  uint32_t sh = 0;
  if (n <= 32) {
    row_warp_sort<1>(v, tot, rows, n, pf, seq, ent);
  } else if (n <= 64) {
    row_warp_sort<2>(v, tot, rows, n, pf, seq, ent);
    sh = 1;
  } else if (n <= 128) {
    row_warp_sort<4>(v, tot, rows, n, pf, seq, ent);
    sh = 2;
  } else if (n <= 256) {
    row_warp_sort<8>(v, tot, rows, n, pf, seq, ent);
    sh = 3;
  } else {
    row_warp_sort<16>(v, tot, rows, n, pf, seq, ent);
    sh = 4;
  }
  if (seq) {
    uint32_t* sq = smem + 2 * SEQ_SLOTS;
    if (lane < SEQ_CLASSES) sq[SEQ_BEFORE + lane] = 0;
    seq_totals(sq, tot, C);
    __syncwarp();
    const uint32_t i0 = min(lane << sh, n), m = min(n - i0, 1u << sh);
    const uint2* run = ent + seq_at(i0, sh);
    uint32_t w[4];
    seq_count(run, m, w);
    const float xp = __uint_as_float(ent[i0 > 0 ? seq_at(i0 - 1, sh) : 0u].x);
    SeqBest bb{dinf(), NONE, 0u, 0.f, 0.f};
    seq_scan(run, m, sh, w, sq, C, xp, 0, n, s.node_q + it.x, bb);
    const uint32_t win = warp_best_lane(bb.score, bb.pos);
    if (win == NONE ? lane == 0 : lane == win) *out = RowBest{bb.score, bb.pos, bb.pure, bb.xl, bb.xr};
    return;
  }
  uint16_t* cnt = reinterpret_cast<uint16_t*>(smem + 2 * SEQ_SLOTS);
  for (uint32_t c = lane; c < C; c += 32) cnt[c] = 0;
  int32_t st2 = 0;  // sum of squared class totals, as a sum over the rows of their class's total
  for (uint32_t p = lane; p < n; p += 32) st2 += (int32_t)(ent[seq_at(p, sh)].y >> 16);
  st2 = (int32_t)__reduce_add_sync(FULL, (uint32_t)st2);
  __syncwarp();
  const double nn = (double)n;
  const unsigned lt = lanemask_lt();
  int32_t sl = 0, a = 0;  // sum of squared left counts; sum of left count x total
  RowBest rb{dinf(), NONE, 0u, 0.f, 0.f};
  float x_last = __uint_as_float(ent[0].x);
#pragma unroll 1
  for (uint32_t p0 = 0; p0 < n; p0 += 32) {
    const uint32_t p = p0 + lane;
    const bool valid = p < n;
    const uint2 en = valid ? ent[seq_at(p, sh)] : make_uint2(0u, 0u);
    const float x = __uint_as_float(en.x);
    float xp = __shfl_up_sync(FULL, x, 1);
    if (lane == 0) xp = x_last;
    x_last = __shfl_sync(FULL, x, 31);
    const uint32_t c = valid ? en.y & 0xffffu : NONE;
    const unsigned grp = __match_any_sync(FULL, c);
    uint32_t packed = 0;
    if (valid) packed = (2u * (cnt[c] + (uint32_t)__popc(grp & lt)) + 1u) | (en.y & 0xffff0000u);
    __syncwarp();
    if (valid && (grp >> lane) == 1u) cnt[c] += (uint16_t)__popc(grp);
    __syncwarp();
    // 32 x (2 x 512 + 1) and 32 x 512 both stay below 2^16
    const uint32_t incl = (uint32_t)warp_incl_scan_i32((int32_t)packed), excl = incl - packed;
    const uint32_t total = __shfl_sync(FULL, incl, 31);
    const int32_t SL = sl + (int32_t)(excl & 0xffffu);  // of the rows before this one
    const int32_t SR = st2 - 2 * (a + (int32_t)(excl >> 16)) + SL;
    sl += (int32_t)(total & 0xffffu);
    a += (int32_t)(total >> 16);
    if (valid && is_candidate_sorted(xp, x)) {
      const Scored sc = score_at(SL, SR, p, nn);
      if (sc.score < rb.score) rb = RowBest{sc.score, p - 1, sc.pure, xp, x};
    }
  }
  const uint32_t win = warp_best_lane(rb.score, rb.pos);
  if (win == NONE ? lane == 0 : lane == win) *out = rb;
}

template <bool Q>
__global__ void __launch_bounds__(THREADS_PER_BLOCK, 8) k_row_warp(View v, LevelScratch s) {
  extern __shared__ __align__(16) uint32_t smem[];
  uint32_t* ws = smem + (threadIdx.x >> 5) * warp_item_words(v.n_classes);
  const uint32_t count = live_count(s, s.ctr->n_small_segs, s.cap_w);
  const StepLists sl = *s.step;
  for_items(count, &s.ctr->claim[ITEM_PLAN], [&](uint32_t i) { row_warp_item<Q>(v, sl, s, ws, i); });
}

// ------------------------------------------------------------------------
// Nodes of WARP_ROWS + 1 .. GROUP_ROWS rows: one CTA per (node, feature) finds
// its rows' sorted positions, stores their values and labels there, and each
// warp scans a run of them from the class counts of the warps before it.
//
// By bitmap: the rows set their rank's bit in a bitmap over all ranks and count
// themselves in their group of 128 ranks; a prefix over the groups and the set
// bits below a row's own give its position.  Only the words a node touched are
// cleared after it, so an item costs its rows and the groups, not the ranks.
// By buckets: the rows count themselves in their bucket of 32 ranks (a byte
// each); a prefix over the buckets gives every bucket's first position, where a
// word, in the place of the sorted rows, holds the bits of its ranks.  One
// phase more, but a third of the bitmap's memory, which the scan's tables then
// share.  Both are bound by latency, so by the CTAs that an SM holds: at 581,012
// ranks the bitmap leaves two CTAs of 8 warps, the buckets four (the smaller
// nodes of 100 covtype-shaped trees: 3.7 -> 2.6 ms); the larger nodes' rows
// themselves leave one CTA or two of 16, and there the bitmap is faster (5.1
// against 5.8 ms) up to about 640,000 ranks (700,000 x 20 rows, 4 classes: 20.6
// against 19.8 ms; from 930,000 on it does not fit), as it is for both while it
// leaves four CTAs (10,000 x 3,000 rows, ct_fit: 29.9 against 31.6 ms).  A
// bitonic sort of the ranks in registers took 13.7 ms against 8.5 of the
// bitmaps.
constexpr uint32_t BUCKET_RANKS = 200000;  // more ranks: less than four CTAs of 8 warps by bitmap
constexpr uint32_t BUCKET_RANKS_LARGE = 640000;
__host__ __device__ __forceinline__ uint32_t group_count_words(uint32_t n_rows) {  // two 16-bit counts per word
  return ((order_words(n_rows) / 4 + 7) / 8) * 4;
}
__host__ __device__ __forceinline__ uint32_t bucket_words(uint32_t n_rows) {  // a word per 4 buckets
  return ((order_words(n_rows) / 4 + 3) / 4) * 4;
}
// The bytes of a word added up (at most 4 x 32).
__device__ __forceinline__ uint32_t byte_sum(uint32_t w) {
  const uint32_t t = (w & 0x00ff00ffu) + ((w >> 8) & 0x00ff00ffu);
  return (t & 0xffffu) + (t >> 16);
}
// Shared memory, in words: (value bits, 8 x label or label | class total << 16)
// by position; the bitmap, group counts and the warps' class counts or seq
// tables; or the buckets' bytes and the prefix of every word of them (16 bits),
// in whose place the tables come.
// With up to SEQ_CLASSES classes a warp's run is padded for seq_scan.
template <int W>
__host__ __device__ __forceinline__ uint32_t group_rows_words() {
  return 2 * ((W == GROUP_SMALL_WARPS ? GROUP_SMALL_ROWS : GROUP_ROWS) + W * 34);
}
__host__ __device__ __forceinline__ uint32_t group_class_words(uint32_t n_classes) {
  return n_classes <= SEQ_CLASSES ? SEQ_WORDS : (n_classes + 3u) & ~3u;
}
template <int W>
__host__ __device__ __forceinline__ bool group_by_buckets(uint32_t n_rows) {
  return n_rows > (W == GROUP_SMALL_WARPS ? BUCKET_RANKS : BUCKET_RANKS_LARGE);
}
template <int W>
__host__ __device__ __forceinline__ uint32_t group_words(uint32_t n_classes, uint32_t n_rows) {
  const uint32_t tables = W * group_class_words(n_classes);
  if (!group_by_buckets<W>(n_rows)) return group_rows_words<W>() + order_words(n_rows) + group_count_words(n_rows) + tables;
  const uint32_t buckets = bucket_words(n_rows) / 2 * 3;
  return group_rows_words<W>() + (buckets > tables ? buckets : tables);
}

template <bool Q, int W, bool BUCKETS>
__device__ __forceinline__ void row_group_item(const View& vb, const StepLists& lists, const LevelScratch& s,
                                               uint32_t* smem, uint32_t n_max, RowBest* s_best, uint32_t* s_wsum,
                                               uint2 item) {
  constexpr uint32_t T = W * 32, K = (W == GROUP_SMALL_WARPS ? GROUP_SMALL_ROWS : GROUP_ROWS) / T;
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, C = vb.n_classes;
  const ct_node nd = lists.nodes[item.x];
  CT_JOB_REF(v, vb, nd.slot);
  const uint32_t n = nd.n;
  const uint32_t f = s.sel[(size_t)item.x * v.sel_stride + item.y];
  const uint32_t* rows = row_list(v, nd.buf, nd.slot) + nd.start;
  const uint2* pf = v.pair + (size_t)f * v.n_rows;
  const uint32_t* tot = lists.tot + (size_t)item.x * C;
  uint2* ent = reinterpret_cast<uint2*>(smem);
  uint32_t* bits = smem;  // by buckets: of a bucket's ranks, at its first position
  uint32_t* bm = smem + group_rows_words<W>();  // the bitmap or the buckets
  uint32_t* gc = bm + order_words(n_max);
  uint32_t* cls = BUCKETS ? bm : gc + group_count_words(n_max);
  uint32_t* cnt = cls + warp * group_class_words(C);
  const bool seq = C <= SEQ_CLASSES;
  // 16-byte units: of 16 buckets, or of 8 groups
  const uint32_t units = (BUCKETS ? bucket_words(v.n_rows) : group_count_words(v.n_rows)) / 4;
  uint4* unit = reinterpret_cast<uint4*>(BUCKETS ? bm : gc);
  uint16_t* prefix = reinterpret_cast<uint16_t*>(bm + bucket_words(v.n_rows));
  // rows of one warp's run, and where position p is kept: runs of 32 << sh
  // rows padded for seq_scan, else runs without padding
  const uint32_t sh = seq_shift(ceil_div(n, (uint32_t)W));
  const uint32_t len = seq ? 32u << sh : ceil_div(ceil_div(n, 32u), (uint32_t)W) * 32;
  auto at = [&](uint32_t p) { return seq ? p + (p >> sh) : p; };
  uint32_t rk[K], lb[K];
  float xv[K];
#pragma unroll
  for (uint32_t k = 0; k < K; ++k) lb[k] = k * T + threadIdx.x < n ? rows[k * T + threadIdx.x] : 0u;
  for (uint32_t g = threadIdx.x; g < units; g += T) unit[g] = make_uint4(0u, 0u, 0u, 0u);
  if (BUCKETS)
    for (uint32_t i = threadIdx.x; i < n; i += T) bits[i] = 0u;
#pragma unroll
  for (uint32_t k = 0; k < K; ++k) {
    rk[k] = 0;
    xv[k] = 0.f;
    if (k * T + threadIdx.x < n) {
      const uint2 pr = __ldg(pf + entry_row(v, lb[k]));
      rk[k] = pr.x;
      xv[k] = __uint_as_float(pr.y);
    }
  }
  if (!BUCKETS && !seq)
    for (uint32_t c = lane; c < C; c += 32) cnt[c] = 0;
  __syncthreads();
#pragma unroll
  for (uint32_t k = 0; k < K; ++k)
    if (k * T + threadIdx.x < n) {
      if (BUCKETS) {
        atomicAdd(&bm[rk[k] >> 7], 1u << ((rk[k] >> 2) & 24));
      } else {
        atomicOr(&bm[rk[k] >> 5], 1u << (rk[k] & 31));
        atomicAdd(&gc[rk[k] >> 8], 1u << ((rk[k] >> 3) & 16));
      }
    }
  __syncthreads();
  // exclusive prefix of the counts by 128 ranks (at most 9,216: 16 bits)
  const uint32_t per_w = ceil_div(ceil_div(units, 32u), (uint32_t)W) * 32;
  const uint32_t ulo = min(warp * per_w, units), uhi = min(ulo + per_w, units);
  uint32_t sum = 0;
  for (uint32_t u = ulo + lane; u < uhi; u += 32) {
    const uint4 q = unit[u];
    if (BUCKETS) {
      sum += byte_sum(q.x) + byte_sum(q.y) + byte_sum(q.z) + byte_sum(q.w);
    } else {
      const uint32_t t = q.x + q.y + q.z + q.w;  // 16-bit fields: at most 512 each
      sum += (t & 0xffffu) + (t >> 16);
    }
  }
  sum = __reduce_add_sync(FULL, sum);
  if (lane == 0) s_wsum[warp] = sum;
  __syncthreads();
  uint32_t run = __reduce_add_sync(FULL, lane < warp ? s_wsum[lane & (W - 1)] : 0u);
  for (uint32_t u0 = ulo; u0 < uhi; u0 += 32) {
    const uint32_t u = u0 + lane;
    const uint4 q = u < uhi ? unit[u] : make_uint4(0u, 0u, 0u, 0u);
    uint32_t tx, ty, tz, tw;  // by word
    if (BUCKETS) {
      tx = byte_sum(q.x), ty = byte_sum(q.y), tz = byte_sum(q.z), tw = byte_sum(q.w);
    } else {
      tx = (q.x & 0xffffu) + (q.x >> 16), ty = (q.y & 0xffffu) + (q.y >> 16);
      tz = (q.z & 0xffffu) + (q.z >> 16), tw = (q.w & 0xffffu) + (q.w >> 16);
    }
    const uint32_t t = tx + ty + tz + tw, incl = (uint32_t)warp_incl_scan_i32((int32_t)t);
    const uint32_t b0 = run + incl - t, b1 = b0 + tx, b2 = b1 + ty, b3 = b2 + tz;
    if (u < uhi) {
      if (BUCKETS)
        reinterpret_cast<uint2*>(prefix)[u] = make_uint2(b0 | (b1 << 16), b2 | (b3 << 16));
      else  // each word holds the groups 2 i (low half) and 2 i + 1
        unit[u] = make_uint4(b0 | ((b0 + (q.x & 0xffffu)) << 16), b1 | ((b1 + (q.y & 0xffffu)) << 16),
                             b2 | ((b2 + (q.z & 0xffffu)) << 16), b3 | ((b3 + (q.w & 0xffffu)) << 16));
    }
    run += __shfl_sync(FULL, incl, 31);
  }
  __syncthreads();
  if (BUCKETS) {
#pragma unroll
    for (uint32_t k = 0; k < K; ++k)
      if (k * T + threadIdx.x < n) {
        const uint32_t r = rk[k], first = prefix[r >> 7] + byte_sum(bm[r >> 7] & ((1u << ((r >> 2) & 24)) - 1u));
        atomicOr(&bits[first], 1u << (r & 31));
        rk[k] = (first << 5) | (r & 31);
      }
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < K; ++k)
      if (k * T + threadIdx.x < n) rk[k] = (rk[k] >> 5) + __popc(bits[rk[k] >> 5] & ((1u << (rk[k] & 31)) - 1u));
    if (!seq)  // every row is done with the buckets
      for (uint32_t c = lane; c < C; c += 32) cnt[c] = 0;
    __syncthreads();
  }
#pragma unroll
  for (uint32_t k = 0; k < K; ++k)
    if (k * T + threadIdx.x < n) {
      uint32_t pos = rk[k];
      if (!BUCKETS) {
        const uint32_t r = rk[k], in = (r >> 5) & 3u, below = (1u << (r & 31)) - 1u;
        const uint4 q = reinterpret_cast<const uint4*>(bm)[r >> 7];
        pos = reinterpret_cast<const uint16_t*>(gc)[r >> 7] + __popc(q.x & (in > 0 ? FULL : below)) +
              __popc(q.y & (in > 1 ? FULL : in == 1 ? below : 0u)) +
              __popc(q.z & (in > 2 ? FULL : in == 2 ? below : 0u)) + __popc(q.w & (in == 3 ? below : 0u));
      }
      const uint32_t lab = lb[k] >> v.lab_shift;
      ent[at(pos)] = seq ? seq_entry(__float_as_uint(xv[k]), lab)
                         : make_uint2(__float_as_uint(xv[k]), lab | (__ldg(tot + lab) << 16));
    }
  __syncthreads();
  if (!BUCKETS) {
#pragma unroll
    for (uint32_t k = 0; k < K; ++k)  // every row is placed: clear the words it touched
      if (k * T + threadIdx.x < n) bm[rk[k] >> 5] = 0u;
  }
  // this warp's run of sorted rows
  const uint32_t w0 = min(warp * len, n), w1 = min(w0 + len, n);
  RowBest rb{dinf(), NONE, 0u, 0.f, 0.f};
  if (seq) {
    uint32_t* before = cnt + SEQ_BEFORE;
    const uint32_t i0 = min(w0 + (lane << sh), w1), m = min(w1 - i0, 1u << sh);
    const uint2* run = ent + at(i0);
    uint32_t w[4], t[4];
    seq_count(run, m, w);
#pragma unroll
    for (int h = 0; h < 4; ++h) t[h] = __reduce_add_sync(FULL, w[h]);
    if (lane < SEQ_CLASSES) before[lane] = seq_field(t, lane);
    seq_totals(cnt, tot, C);
    __syncthreads();
    uint32_t mine = 0;
    if (lane < SEQ_CLASSES)
      for (uint32_t k = 0; k < warp; ++k) mine += cls[k * SEQ_WORDS + SEQ_BEFORE + lane];
    __syncthreads();
    if (lane < SEQ_CLASSES) before[lane] = mine;
    __syncwarp();
    if (w0 < w1) {
      SeqBest bb{dinf(), NONE, 0u, 0.f, 0.f};
      const float xp = __uint_as_float(ent[at(i0 < w1 ? (i0 ? i0 - 1 : 0u) : w0)].x);
      seq_scan(run, m, sh, w, cnt, C, xp, w0, n, s.node_q + item.x, bb);
      rb = RowBest{bb.score, bb.pos, bb.pure, bb.xl, bb.xr};
    }
  } else {
    for (uint32_t i = w0 + lane; i < w1; i += 32) atomicAdd(&cnt[ent[i].y & 0xffffu], 1u);
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < C; c += T) {
      uint32_t before = 0;
#pragma unroll
      for (uint32_t k = 0; k < W; ++k) {
        const uint32_t t = cls[k * group_class_words(C) + c];
        cls[k * group_class_words(C) + c] = before;
        before += t;
      }
    }
    __syncthreads();
    // sums of squares stay below 2^27 (at most 9,216 rows)
    uint32_t sl = 0, a = 0, st2 = 0;
    for (uint32_t c = lane; c < C; c += 32) {
      const uint32_t k = cnt[c], t = __ldg(tot + c);
      sl += k * k;
      a += k * t;
      st2 += t * t;
    }
    sl = __reduce_add_sync(FULL, sl);
    a = __reduce_add_sync(FULL, a);
    st2 = __reduce_add_sync(FULL, st2);
    __syncwarp();
    const double nn = (double)n;
    const unsigned lt = lanemask_lt();
    float x_last = __uint_as_float(ent[w0 ? w0 - 1 : 0u].x);
    for (uint32_t p0 = w0; p0 < w1; p0 += 32) {
      const uint32_t p = p0 + lane;
      const bool valid = p < w1;
      const uint2 en = valid ? ent[p] : make_uint2(0u, 0u);
      const uint32_t ltv = en.y;
      const float x = __uint_as_float(en.x);
      float xp = __shfl_up_sync(FULL, x, 1);
      if (lane == 0) xp = x_last;
      x_last = __shfl_sync(FULL, x, 31);
      const uint32_t c = valid ? ltv & 0xffffu : NONE;
      const unsigned grp = __match_any_sync(FULL, c);
      uint32_t dl = 0, dt = 0;
      if (valid) {
        dl = 2 * (cnt[c] + (uint32_t)__popc(grp & lt)) + 1;
        dt = ltv >> 16;
      }
      __syncwarp();
      if (valid && (grp >> lane) == 1u) cnt[c] += __popc(grp);
      __syncwarp();
      const uint32_t il = (uint32_t)warp_incl_scan_i32((int32_t)dl), it = (uint32_t)warp_incl_scan_i32((int32_t)dt);
      const uint32_t SL = sl + (il - dl);  // of the rows before this one
      const uint32_t SR = st2 - 2 * (a + (it - dt)) + SL;
      sl += __shfl_sync(FULL, il, 31);
      a += __shfl_sync(FULL, it, 31);
      if (valid && p > 0 && is_candidate_sorted(xp, x)) {
        const Scored sc = score_at((int64_t)SL, (int64_t)SR, p, nn);
        if (sc.score < rb.score) rb = RowBest{sc.score, p - 1, sc.pure, xp, x};
      }
    }
  }
  const uint32_t win = warp_best_lane(rb.score, rb.pos);
  if (win == NONE ? lane == 0 : lane == win) s_best[warp] = rb;
  __syncthreads();
  if (warp == 0) {
    rb = lane < W ? s_best[lane] : RowBest{dinf(), NONE, 0u, 0.f, 0.f};
    const uint32_t wl = warp_best_lane(rb.score, rb.pos);
    if (wl == NONE ? lane == 0 : lane == wl) s.rbest[(size_t)item.x * v.sel_stride + item.y] = rb;
  }
}

template <bool Q, int W, bool BUCKETS>
__global__ void __launch_bounds__(W * 32, W == GROUP_SMALL_WARPS ? 4 : 2) k_row_group(View v, LevelScratch s, uint32_t n_max) {
  extern __shared__ __align__(16) uint32_t group_sm[];
  __shared__ RowBest s_best[W];
  __shared__ uint32_t s_wsum[W];
  __shared__ uint32_t s_item;
  const uint32_t count = live_count(s, W == GROUP_SMALL_WARPS ? s.ctr->n_huge_segs : s.ctr->n_hchains, s.cap_order);
  const uint2* list = W == GROUP_SMALL_WARPS ? s.gsmall : s.glarge;
  uint32_t* claim = W == GROUP_SMALL_WARPS ? &s.ctr->ticket : &s.ctr->ticket_huge;
  const StepLists sl = *s.step;
  uint32_t i = blockIdx.x;
  if (i >= count) return;
  if (!BUCKETS) {
    uint4* bm4 = reinterpret_cast<uint4*>(group_sm + group_rows_words<W>());
    for (uint32_t g = threadIdx.x; g < order_words(n_max) / 4; g += W * 32) bm4[g] = make_uint4(0u, 0u, 0u, 0u);
  }
  while (i < count) {
    if (threadIdx.x == 0) s_item = gridDim.x + atomicAdd(claim, 1u);  // the next item, claimed ahead
    row_group_item<Q, W, BUCKETS>(v, sl, s, group_sm, n_max, s_best, s_wsum, list[i]);
    __syncthreads();
    i = s_item;
    __syncthreads();
  }
}

// ------------------------------------------------------------------------
// Larger nodes: one CTA per (node, feature).  The node's rows set their rank's
// bit in a bitmap over all ranks; a row's sorted position is then the count
// of set bits before its own (a prefix per word, or per four words when the
// node has more than 65,535 rows), where its value and label are stored.
template <bool Q>
__global__ void __launch_bounds__(ORDER_THREADS, 2) k_row_order(View vb, LevelScratch s) {
  extern __shared__ __align__(16) uint32_t order_sm[];
  __shared__ uint32_t s_wsum[ORDER_THREADS / 32];
  __shared__ uint32_t s_item;
  const uint32_t count = live_count(s, s.ctr->n_carry, s.cap_order);
  const StepLists lists = *s.step;
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  constexpr uint32_t T = ORDER_THREADS, NW = T / 32;
  while (true) {
    __syncthreads();  // the previous item is done with the bitmap and s_item
    if (threadIdx.x == 0) s_item = atomicAdd(&s.ctr->claim[ITEM_TWO_VALUED], 1u);
    __syncthreads();
    const uint32_t it = s_item;
    if (it >= count) break;
    const uint2 item = s.oitems[it];
    const ct_node nd = lists.nodes[item.x];
    CT_JOB_REF(v, vb, nd.slot);
    const uint32_t n = nd.n;
    const uint32_t f = s.sel[(size_t)item.x * v.sel_stride + item.y];
    const uint32_t* rows = row_list(v, nd.buf, nd.slot) + nd.start;
    const uint2* pf = v.pair + (size_t)f * v.n_rows;
    uint2* out = sorted_list(v, nd.slot, item.y) + nd.start;
    const uint32_t words = order_words(v.n_rows), groups = words / 4;
    uint32_t* bm = order_sm;
    uint4* bm4 = reinterpret_cast<uint4*>(order_sm);
    uint16_t* pre16 = reinterpret_cast<uint16_t*>(order_sm + words);
    uint32_t* pre32 = order_sm + words;
    for (uint32_t g = threadIdx.x; g < groups; g += T) bm4[g] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    for (uint32_t i0 = threadIdx.x; i0 < n; i0 += T * 4) {
      uint32_t r[4];
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) r[k] = i0 + k * T < n ? rows[i0 + k * T] : NONE;
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k)
        if (i0 + k * T < n) r[k] = __ldg(&pf[entry_row(v, r[k])].x);
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k)
        if (i0 + k * T < n) atomicOr(&bm[r[k] >> 5], 1u << (r[k] & 31));
    }
    __syncthreads();
    // exclusive prefix: each warp sums, then scans, a run of groups
    const uint32_t per = ceil_div(ceil_div(groups, 32u), NW) * 32;
    const uint32_t glo = min(warp * per, groups), ghi = min(glo + per, groups);
    uint32_t sum = 0;
    for (uint32_t g = glo + lane; g < ghi; g += 32) {
      const uint4 q = bm4[g];
      sum += __popc(q.x) + __popc(q.y) + __popc(q.z) + __popc(q.w);
    }
    sum = __reduce_add_sync(FULL, sum);
    if (lane == 0) s_wsum[warp] = sum;
    __syncthreads();
    uint32_t run = 0;
#pragma unroll
    for (uint32_t k = 0; k < NW; ++k) run += k < warp ? s_wsum[k] : 0u;
    const bool wide = n > 0xffffu;
    for (uint32_t g0 = glo; g0 < ghi; g0 += 32) {
      const uint32_t g = g0 + lane;
      const uint4 q = g < ghi ? bm4[g] : make_uint4(0u, 0u, 0u, 0u);
      const uint32_t c0 = __popc(q.x), c1 = __popc(q.y), c2 = __popc(q.z), c3 = __popc(q.w);
      const uint32_t t = c0 + c1 + c2 + c3;
      const uint32_t incl = (uint32_t)warp_incl_scan_i32((int32_t)t);
      const uint32_t b = run + incl - t;
      if (g < ghi) {
        if (wide) {
          pre32[g] = b;
        } else {
          reinterpret_cast<uint2*>(pre16)[g] =
              make_uint2(b | ((b + c0) << 16), (b + c0 + c1) | ((b + c0 + c1 + c2) << 16));
        }
      }
      run += __shfl_sync(FULL, incl, 31);
    }
    __syncthreads();
    for (uint32_t i0 = threadIdx.x; i0 < n; i0 += T * 4) {
      uint32_t e[4];
      uint2 pr[4];
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) e[k] = i0 + k * T < n ? __ldcs(rows + i0 + k * T) : 0u;
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k)
        if (i0 + k * T < n) pr[k] = __ldg(pf + entry_row(v, e[k]));
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
        if (i0 + k * T >= n) continue;
        const uint32_t wd = pr[k].x >> 5, below = (1u << (pr[k].x & 31)) - 1u;
        uint32_t pos;
        if (wide) {
          const uint4 q = bm4[wd >> 2];
          const uint32_t in = wd & 3u;
          pos = pre32[wd >> 2] + __popc(q.x & (in > 0 ? FULL : below)) + (in > 0 ? __popc(q.y & (in > 1 ? FULL : below)) : 0) +
                (in > 1 ? __popc(q.z & (in > 2 ? FULL : below)) : 0) + (in > 2 ? __popc(q.w & below) : 0);
        } else {
          pos = pre16[wd] + __popc(bm[wd] & below);
        }
        if (pos < n) out[pos] = make_uint2(pr[k].y, e[k] >> v.lab_shift);
      }
    }
  }
}

// ------------------------------------------------------------------------
// The elements of a piece, in sorted order, as (value bits, label).  A sorted
// list's piece is its positions [lo, hi); a bitmap's is a run of ranks, whose
// set bits are listed in shared memory a batch at a time (each lane takes a
// word of a 1,024-rank window and writes its bits behind the lower lanes').
constexpr uint32_t ROW_BATCH = 4;
constexpr uint32_t LIST_FILL = 512;              // a batch ends with the window that reaches this
constexpr uint32_t LIST_CAP = LIST_FILL + 1024;

struct PieceStream {
  const uint2* base;      // element i of the batch: base[dense ? list[i] : i]
  const uint32_t* words;  // dense: bitmap words of the piece
  uint16_t* list;
  uint32_t n_words;
  uint32_t next;          // first word (dense) or batch (list) not listed yet
  uint32_t count;         // elements of the batch
  bool dense;
  __device__ __forceinline__ bool more() const { return dense && next < n_words; }
  __device__ __forceinline__ uint2 load(uint32_t i) const { return dense ? __ldg(base + list[i]) : __ldcs(base + i); }
  // Lists the next batch behind the last `keep` elements of this one, which
  // are still to be read; false at the end of the piece.  Warp-collective.
  __device__ __forceinline__ bool fill(uint32_t keep = 0) {
    if (!dense) return next++ == 0 && count > 0;
    const uint32_t lane = lane_id();
    __syncwarp();
    if (keep) {
      for (uint32_t i0 = 0; i0 < keep; i0 += 32) {
        const uint16_t e = i0 + lane < keep ? list[count - keep + i0 + lane] : (uint16_t)0;
        __syncwarp();
        if (i0 + lane < keep) list[i0 + lane] = e;
        __syncwarp();
      }
    }
    count = keep;
    while (next < n_words && count < LIST_FILL) {
      uint32_t b = next + lane < n_words ? __ldg(words + next + lane) : 0u;
      const uint32_t c = __popc(b);
      const uint32_t incl = (uint32_t)warp_incl_scan_i32((int32_t)c);
      uint32_t pos = count + incl - c;
      const uint32_t r0 = (next + lane) * 32 - 1;
      for (; b; b &= b - 1) list[pos++] = (uint16_t)(r0 + __ffs(b));
      count += __shfl_sync(FULL, incl, 31);
      next += 32;
    }
    __syncwarp();
    return count > 0;
  }
};

// Shared memory of one warp of k_row_hist and k_row_scan, in words.
__host__ __device__ __forceinline__ uint32_t hist_words(uint32_t n_classes) { return LIST_CAP / 2 + n_classes; }
__host__ __device__ __forceinline__ uint32_t scan_words(uint32_t n_classes) {
  return LIST_CAP / 2 + 2 * n_classes;
}

__device__ __forceinline__ PieceStream piece_stream(const View& v, const ct_node& nd, const RowPiece& pc, uint32_t f,
                                                    uint32_t scan_piece, uint32_t* smem) {
  PieceStream ps;
  ps.list = reinterpret_cast<uint16_t*>(smem);
  ps.next = 0;
  ps.dense = row_dense(nd.n, v.n_rows);
  if (ps.dense) {
    const uint32_t chunk = dense_chunk(nd.n, v.n_rows, scan_piece), r0 = pc.j * chunk;
    ps.base = v.ranked + (size_t)f * v.n_rows + r0;
    ps.words = rank_bits(v, nd, pc.slot) + r0 / 32;
    ps.n_words = min(chunk / 32, order_words(v.n_rows) - r0 / 32);
    ps.count = 0;
  } else {
    const uint32_t lo = pc.j * scan_piece;
    ps.base = sorted_list(v, nd.slot, pc.slot) + nd.start + lo;
    ps.words = nullptr;
    ps.n_words = 0;
    ps.count = min(scan_piece, nd.n - lo);
  }
  return ps;
}

// Class counts of all but the last piece of a multi-piece list (carry rows
// are indexed by piece).
template <bool Q>
__device__ __forceinline__ void row_hist_item(const View& vb, const StepLists& lists, const LevelScratch& s,
                                              uint32_t* smem, uint32_t pi) {
  const uint32_t C = vb.n_classes, lane = lane_id();
  const RowPiece pc = s.rpieces[pi];
  if (pc.j + 1 >= pc.npieces) return;
  const ct_node nd = lists.nodes[pc.node];
  CT_JOB_REF(v, vb, nd.slot);
  if (row_dense(nd.n, v.n_rows) && pc.npieces * C <= BITS_COUNTS) return;  // k_row_bits counted them
  const uint32_t f = s.sel[(size_t)pc.node * v.sel_stride + pc.slot];
  PieceStream ps = piece_stream(v, nd, pc, f, lists.scan_piece, smem);
  uint32_t* cnt = smem + LIST_CAP / 2;
  uint32_t* out = s.carry + (size_t)pi * C;
  for (uint32_t c = lane; c < C; c += 32) cnt[c] = 0;
  __syncwarp();
  while (ps.fill()) {
    for (uint32_t b0 = 0; b0 < ps.count; b0 += 32 * 128) {  // at most 128 entries per lane
      const uint32_t b1 = min(b0 + 32 * 128, ps.count);
      uint64_t pk = 0;  // up to 8 classes: 8-bit field per class
      for (uint32_t b = b0; b < b1; b += 32 * ROW_BATCH) {
        uint32_t c[ROW_BATCH];
#pragma unroll
        for (uint32_t r = 0; r < ROW_BATCH; ++r) c[r] = b + r * 32 + lane < b1 ? ps.load(b + r * 32 + lane).y : NONE;
#pragma unroll
        for (uint32_t r = 0; r < ROW_BATCH; ++r) {
          if (c[r] == NONE) continue;
          if (C <= 8) pk += 1ull << (8 * c[r]);
          else atomicAdd(&cnt[c[r]], 1u);
        }
      }
      if (C <= 8) {
        const uint32_t fh[2] = {(uint32_t)pk, (uint32_t)(pk >> 32)};
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
          const uint32_t ev = __reduce_add_sync(FULL, fh[h] & 0x00ff00ffu);
          const uint32_t od = __reduce_add_sync(FULL, (fh[h] >> 8) & 0x00ff00ffu);
          const uint32_t val = (lane & 1u ? od : ev) >> ((lane & 2u) * 8) & 0xffffu;
          if (lane < 4 && 4 * h + lane < C) cnt[4 * h + lane] += val;
        }
      }
    }
  }
  __syncwarp();
  for (uint32_t c = lane; c < C; c += 32) out[c] = cnt[c];
}

template <bool Q>
__global__ void __launch_bounds__(THREADS_PER_BLOCK) k_row_hist(View v, LevelScratch s) {
  extern __shared__ uint32_t smem[];
  uint32_t* ws = smem + (threadIdx.x >> 5) * hist_words(v.n_classes);
  const uint32_t count = live_count(s, s.ctr->n_scan_pieces, s.cap_scan);
  const StepLists sl = *s.step;
  for_items(count, &s.ctr->claim[ITEM_HIST], [&](uint32_t i) { row_hist_item<Q>(v, sl, s, ws, i); });
}

// Exclusive prefix of the class counts over a list's pieces: one warp per
// (list, class), 128 pieces per round.
__global__ void __launch_bounds__(THREADS_PER_BLOCK) k_row_carry(LevelScratch s, uint32_t C) {
  const uint32_t count = live_count(s, s.ctr->n_bchains, s.cap_order);
  const uint32_t lane = lane_id();
  for_items(count * C, &s.ctr->claim[ITEM_CARRY], [&](uint32_t i) {
    const uint2 ci = s.citems[i / C];
    uint32_t* h = s.carry + (size_t)ci.x * C + i % C;
    uint32_t run = 0;
    for (uint32_t j0 = 0; j0 < ci.y; j0 += 128) {
      uint32_t t[4];
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {  // the last piece's count is not needed, and not always there
        const uint32_t j = j0 + k * 32 + lane;
        t[k] = j + 1 < ci.y ? h[(size_t)j * C] : 0u;
      }
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t j = j0 + k * 32 + lane;
        const uint32_t incl = (uint32_t)warp_incl_scan_i32((int32_t)t[k]);
        if (j < ci.y) h[(size_t)j * C] = run + incl - t[k];
        run += __shfl_sync(FULL, incl, 31);
      }
    }
  });
}

// A start for the bound of the nodes' scans (seq_scan): the estimated gain at
// every piece's first position that is a candidate.  One thread per piece.
template <bool Q>
__global__ void __launch_bounds__(256) k_row_bound(View vb, LevelScratch s) {
  const uint32_t count = live_count(s, s.ctr->n_scan_pieces, s.cap_scan), C = vb.n_classes;
  const StepLists lists = *s.step;
  for (uint32_t pi = blockIdx.x * blockDim.x + threadIdx.x; pi < count; pi += gridDim.x * blockDim.x) {
    const RowPiece pc = s.rpieces[pi];
    if (pc.j == 0) continue;
    const ct_node nd = lists.nodes[pc.node];
    CT_JOB_REF(v, vb, nd.slot);
    const uint32_t* left = s.carry + (size_t)pi * C;
    uint32_t nl = 0;
    for (uint32_t c = 0; c < C; ++c) nl += left[c];
    if (nl == 0 || nl >= nd.n) continue;
    float xa, xb;
    if (row_dense(nd.n, v.n_rows)) {
      const uint32_t f = s.sel[(size_t)pc.node * v.sel_stride + pc.slot];
      const uint32_t w0 = pc.j * dense_chunk(nd.n, v.n_rows, lists.scan_piece) / 32;
      const uint32_t* bits = rank_bits(v, nd, pc.slot);
      uint32_t wa = w0, wb = w0, ba = 0, bb = 0;  // the nearest set bits on both sides, if near
      for (uint32_t k = 0; k < 64 && wa > 0 && !ba; ++k) ba = __ldg(bits + --wa);
      for (uint32_t k = 0; k < 64 && wb < order_words(v.n_rows) && !bb; ++k) bb = __ldg(bits + wb++);
      if (!ba || !bb) continue;
      const uint2* rk = v.ranked + (size_t)f * v.n_rows;
      xa = __uint_as_float(__ldg(&rk[wa * 32 + 31 - __clz((int)ba)].x));
      xb = __uint_as_float(__ldg(&rk[(wb - 1) * 32 + __ffs((int)bb) - 1].x));
    } else {
      const uint2* lst = sorted_list(v, nd.slot, pc.slot) + nd.start + pc.j * lists.scan_piece;
      xa = __uint_as_float(lst[-1].x);
      xb = __uint_as_float(lst[0].x);
    }
    if (!is_candidate_sorted(xa, xb)) continue;
    atomicMax(s.node_q + pc.node, __float_as_uint(gain_at(left, lists.tot + (size_t)pc.node * C, C, nl, nd.n)));
  }
}

// Which pieces to scan, with up to SEQ_CLASSES classes.  The gain is a convex
// function of the left class counts, so no order of a piece's rows has a
// candidate with a larger gain than the corners have at which every class's
// rows lie all left or all right of it; a piece whose best corner is below the
// best gain known for the node holds no split (98 pieces in 100 on
// covtype-shaped data).  The counts' sums of squares and of products with the
// totals that a gain takes (seq_scan) are sums over the classes, so a lane
// adds up its five lowest classes' once and then only the others', corner by
// corner.  A warp takes LIMIT_PIECES pieces together, whose records and counts
// come in with one round of loads: checked by the scanning warp, one piece at
// a time, the loads' latency was most of the scan (9.2 ms of 100
// covtype-shaped trees, 0.7 here).
constexpr uint32_t LIMIT_PIECES = 8;
constexpr uint32_t LIMIT_BASE = 5;  // classes of a lane's own corner

struct PieceLimit {
  double2 add[SEQ_CLASSES];    // what a class's rows of the piece add to s and a when they lie left
  uint32_t rows[SEQ_CLASSES];  // those rows
  double s, a, t;              // sums of A^2, A T, T^2 over the classes, A the counts before the piece
  uint32_t nl;                 // sum of A
  uint32_t n_rows;             // rows of the piece
};
// From the class counts a before the piece, b after it, t of the node: one
// class per lane of a group of SEQ_CLASSES lanes.  Warp-collective.
__device__ __forceinline__ void limit_set(PieceLimit& pl, bool write, uint32_t a, uint32_t b, uint32_t t) {
  const uint32_t c = lane_id() % SEQ_CLASSES;
  double qs = (double)((uint64_t)a * a), qa = (double)((uint64_t)a * t), qt = (double)((uint64_t)t * t);
  uint32_t nl = a, rows = b - a;
  if (write) {
    pl.add[c] = make_double2((double)((uint64_t)b * b - (uint64_t)a * a), (double)((uint64_t)(b - a) * t));
    pl.rows[c] = b - a;
  }
#pragma unroll
  for (uint32_t k = 1; k < SEQ_CLASSES; k <<= 1) {
    qs += __shfl_xor_sync(FULL, qs, k);
    qa += __shfl_xor_sync(FULL, qa, k);
    qt += __shfl_xor_sync(FULL, qt, k);
    nl += __shfl_xor_sync(FULL, nl, k);
    rows += __shfl_xor_sync(FULL, rows, k);
  }
  if (write && c == 0) {
    pl.s = qs;
    pl.a = qa;
    pl.t = qt;
    pl.nl = nl;
    pl.n_rows = rows;
  }
}
// The largest estimated gain of the piece's corners (0: no rows, so no
// candidate).  Warp-collective.
__device__ __forceinline__ float limit_of(const PieceLimit& pl, uint32_t C, uint32_t n) {
  const uint32_t lane = lane_id();
  if (pl.n_rows == 0) return 0.f;
  const double inv = 1.0 / (double)n, st2 = pl.t;
  const float nf = (float)n;
  double ls = pl.s, la = pl.a;
  uint32_t nl = pl.nl;
#pragma unroll
  for (uint32_t c = 0; c < LIMIT_BASE; ++c)
    if ((lane >> c) & 1u) {
      const double2 d = pl.add[c];
      ls += d.x;
      la += d.y;
      nl += pl.rows[c];
    }
  float best = 1.f;  // no gain: a piece that holds all rows of a node of one class has no corner with rows on both sides
  for (uint32_t m = 0; m < (C > LIMIT_BASE ? 1u << (C - LIMIT_BASE) : 1u); ++m) {
    double ms = ls, ma = la;
    uint32_t k = nl;
#pragma unroll
    for (uint32_t c = 0; c < SEQ_CLASSES - LIMIT_BASE; ++c)
      if ((m >> c) & 1u) {
        const double2 d = pl.add[LIMIT_BASE + c];
        ms += d.x;
        ma += d.y;
        k += pl.rows[LIMIT_BASE + c];
      }
    const double t = (double)k * inv;
    const float g = gain_of(fma(t, fma(t, st2, -2.0 * ma), ms), (float)k, (float)(n - k), nf);
    if (k > 0 && k < n) best = fmaxf(best, g);
  }
  return __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(best)));
}

__global__ void __launch_bounds__(THREADS_PER_BLOCK) k_row_limit(LevelScratch s, uint32_t C) {
  __shared__ PieceLimit limits_all[WARPS_PER_BLOCK][LIMIT_PIECES];
  const uint32_t lane = lane_id();
  PieceLimit* limits = limits_all[threadIdx.x >> 5];
  const uint32_t count = live_count(s, s.ctr->n_scan_pieces, s.cap_scan);
  const StepLists lists = *s.step;
  for_items(ceil_div(count, LIMIT_PIECES), &s.ctr->claim[ITEM_LIMIT], [&](uint32_t i) {
    const uint32_t p0 = i * LIMIT_PIECES, np = min(LIMIT_PIECES, count - p0);
    RowPiece pc{0u, 0u, 0u, 1u};
    uint32_t n = 1;
    float known = 0.f;
    if (lane < np) {
      pc = s.rpieces[p0 + lane];
      n = lists.nodes[pc.node].n;
      known = __uint_as_float(*reinterpret_cast<volatile uint32_t*>(s.node_q + pc.node));
    }
#pragma unroll
    for (uint32_t r = 0; r < LIMIT_PIECES * SEQ_CLASSES / 32; ++r) {
      const uint32_t p = r * (32 / SEQ_CLASSES) + lane / SEQ_CLASSES, c = lane % SEQ_CLASSES;
      const uint32_t node = __shfl_sync(FULL, pc.node, p), j = __shfl_sync(FULL, pc.j, p);
      const uint32_t npieces = __shfl_sync(FULL, pc.npieces, p);
      uint32_t a = 0, b = 0, t = 0;
      if (p < np && c < C) {
        const uint32_t* carry = s.carry + (size_t)(p0 + p) * C + c;
        t = lists.tot[(size_t)node * C + c];
        a = npieces > 1 ? *carry : 0u;
        b = j + 1 < npieces ? carry[C] : t;
      }
      limit_set(limits[p], true, a, b, t);
    }
    __syncwarp();
    uint32_t live = 0;
    float limit = 0.f;
    for (uint32_t p = 0; p < np; ++p) {
      const uint32_t pn = __shfl_sync(FULL, n, p);
      const float best = limit_of(limits[p], C, pn);
      if (best > 0.f && best >= gain_bound(__shfl_sync(FULL, known, p), pn)) live |= 1u << p;
      if (lane == p) limit = best;
    }
    uint32_t at = 0;
    if (lane == 0) {
      s.rlive[i] = (uint8_t)live;
      if (live) at = atomicAdd(&s.ctr->n_live_pieces, (uint32_t)__popc(live));
    }
    at = __shfl_sync(FULL, at, 0) + (uint32_t)__popc(live & lanemask_lt());
    if ((live >> lane) & 1u) s.rscan[at] = make_uint2(p0 + lane, __float_as_uint(limit));
  });
}

// Value bits of the element before the piece (the last set bit before a
// run of ranks).  The piece is not the node's first with elements.
__device__ __forceinline__ uint32_t value_before(const View& v, const PieceStream& ps, const ct_node& nd,
                                                 const RowPiece& pc, uint32_t f, uint32_t scan_piece) {
  if (!ps.dense) return ps.base[-1].x;
  const uint32_t lane = lane_id();
  const uint32_t r0 = pc.j * dense_chunk(nd.n, v.n_rows, scan_piece);
  const uint32_t* bits = ps.words - r0 / 32;
  for (uint32_t w = r0 / 32; w > 0;) {  // 32 words at a time, the nearest on lane 0
    const uint32_t b = lane < w ? __ldg(bits + w - 1 - lane) : 0u;
    const unsigned any = __ballot_sync(FULL, b != 0u);
    if (any) {
      const uint32_t l = (uint32_t)__ffs(any) - 1;
      const uint32_t bw = __shfl_sync(FULL, b, l);
      return __ldg(&v.ranked[(size_t)f * v.n_rows + (w - 1 - l) * 32 + 31 - __clz(bw)].x);
    }
    w = w > 32 ? w - 32 : 0;
  }
  return 0u;
}

// Gini scan of one piece.  The candidate between two neighbours is judged
// when the upper one is met, so only the value before the piece comes from
// outside it.  A piece whose values all equal that one has no candidate.
// With more than SEQ_CLASSES classes one warp scans a piece; a round of 32
// elements matches its classes and scans the sums' increments.
template <bool Q>
__device__ __forceinline__ void row_scan_item(const View& vb, const StepLists& lists, const LevelScratch& s,
                                              uint32_t* smem, uint32_t pi) {
  const uint32_t C = vb.n_classes, lane = lane_id();
  uint32_t* cnt = smem + LIST_CAP / 2;
  uint32_t* T = cnt + C;
  const RowPiece pc = s.rpieces[pi];
  const ct_node nd = lists.nodes[pc.node];
  CT_JOB_REF(v, vb, nd.slot);
  const uint32_t* carry = pc.npieces > 1 ? s.carry + (size_t)pi * C : nullptr;
  const uint32_t* tot = lists.tot + (size_t)pc.node * C;
  const uint32_t n = nd.n;
  RowBest* out = s.rbest + (size_t)s.cap_nodes * vb.sel_stride + pi;
  const uint32_t f = s.sel[(size_t)pc.node * v.sel_stride + pc.slot];
  PieceStream ps = piece_stream(v, nd, pc, f, lists.scan_piece, smem);
  int64_t sl = 0, st2 = 0, a = 0;
  uint32_t before = 0;
  for (uint32_t c = lane; c < C; c += 32) {
    const uint32_t k = carry ? carry[c] : 0u;
    const uint32_t t = tot[c];
    cnt[c] = k;
    T[c] = t;
    before += k;
    sl += (int64_t)k * k;
    st2 += (int64_t)t * t;
    a += (int64_t)k * t;
  }
  sl = warp_sum_i64(sl);
  st2 = warp_sum_i64(st2);
  a = warp_sum_i64(a);
  uint32_t p0 = __reduce_add_sync(FULL, before);  // the batch's first position
  __syncwarp();
  const double nn = (double)n;
  double best = dinf();
  uint32_t bpos = NONE, bpure = 0;
  float bxl = 0.f, bxr = 0.f;
  const unsigned lt = lanemask_lt();
  constexpr uint32_t B = 32 * ROW_BATCH;
  uint32_t x_last = 0;
  bool first = true;
  while (ps.fill()) {
    if (first && p0 > 0) {
      x_last = value_before(v, ps, nd, pc, f, lists.scan_piece);
      // all of this batch equals the value before it: when the batch is the
      // whole piece, it has no candidate
      if (!ps.dense && __uint_as_float(ps.base[ps.count - 1].x) == __uint_as_float(x_last)) break;
    }
    uint2 cur[ROW_BATCH];
#pragma unroll
    for (uint32_t r = 0; r < ROW_BATCH; ++r)
      cur[r] = r * 32 + lane < ps.count ? ps.load(r * 32 + lane) : make_uint2(0u, NONE);
    if (first && p0 == 0) x_last = __shfl_sync(FULL, cur[0].x, 0);  // no candidate before the node's first row
    first = false;
    for (uint32_t base = 0; base < ps.count; base += B) {
      uint2 nxt[ROW_BATCH];
#pragma unroll
      for (uint32_t r = 0; r < ROW_BATCH; ++r) {
        const uint32_t i = base + B + r * 32 + lane;
        nxt[r] = i < ps.count ? ps.load(i) : make_uint2(0u, NONE);
      }
#pragma unroll
      for (uint32_t r = 0; r < ROW_BATCH; ++r) {
        if (base + r * 32 >= ps.count) break;
        const uint32_t i = base + r * 32 + lane;
        const bool valid = i < ps.count;
        const uint32_t c = cur[r].y;
        uint32_t xpb = __shfl_up_sync(FULL, cur[r].x, 1);
        if (lane == 0) xpb = x_last;
        x_last = __shfl_sync(FULL, cur[r].x, min(31u, ps.count - 1 - (base + r * 32)));
        const float x = __uint_as_float(cur[r].x), xp = __uint_as_float(xpb);
        const unsigned grp = __match_any_sync(FULL, c);
        int32_t dl = 0, dt = 0;
        if (valid) {
          dl = 2 * (int32_t)(cnt[c] + __popc(grp & lt)) + 1;
          dt = (int32_t)T[c];
        }
        __syncwarp();
        if (valid && (grp >> lane) == 1u) cnt[c] += __popc(grp);
        __syncwarp();
        // |partial sums| <= 32 (2 n + 1) < 2^31: n <= 2^22 here
        const int32_t il = warp_incl_scan_i32(dl), it = warp_incl_scan_i32(dt);
        const int64_t SL = sl + (il - dl);  // of the rows before this one
        const int64_t SR = st2 - 2 * (a + (it - dt)) + SL;
        sl += __shfl_sync(FULL, il, 31);
        a += __shfl_sync(FULL, it, 31);
        if (valid && is_candidate_sorted(xp, x)) {
          const Scored sc = score_at(SL, SR, p0 + i, nn);
          if (sc.score < best) {
            best = sc.score;
            bpos = p0 + i - 1;
            bpure = sc.pure;
            bxl = xp;
            bxr = x;
          }
        }
      }
#pragma unroll
      for (uint32_t r = 0; r < ROW_BATCH; ++r) cur[r] = nxt[r];
    }
    p0 += ps.count;
  }
  const uint32_t win = warp_best_lane(best, bpos);
  if (win == NONE ? lane == 0 : lane == win) *out = RowBest{best, bpos, bpure, bxl, bxr};
}

template <bool Q>
__global__ void __launch_bounds__(THREADS_PER_BLOCK, 7) k_row_scan(View v, LevelScratch s) {
  extern __shared__ uint32_t smem[];
  uint32_t* ws = smem + (threadIdx.x >> 5) * scan_words(v.n_classes);
  const uint32_t count = live_count(s, s.ctr->n_scan_pieces, s.cap_scan);
  const StepLists sl = *s.step;
  for_items(count, &s.ctr->claim[ITEM_SCAN], [&](uint32_t i) { row_scan_item<Q>(v, sl, s, ws, i); });
}

// The scan of the pieces k_row_limit left, with up to SEQ_CLASSES classes.
// They are few and may be long (a run of ranks can hold all of a node's rows),
// so what bounds it is how long one piece takes: the warps of a CTA share a
// piece.  Each counts the classes of its part, then knows the counts before
// it, and walks only the runs of up to SEQ_ROWS rows whose own limit reaches
// the bound.  One warp per piece took 120 us of a level of 20 covtype-shaped
// trees with 7% of the warps in flight (100 trees: 8.3 ms, here 2.9).
constexpr int SCAN_WARPS = 8;
constexpr uint32_t SCAN_WORDS = LIST_CAP / 2 + 2 * SEQ_SLOTS + SEQ_WORDS + sizeof(PieceLimit) / 4;  // of one warp
static_assert(SCAN_WORDS % 4 == 0 && (LIST_CAP / 2 + 2 * SEQ_SLOTS + SEQ_WORDS) % 4 == 0, "PieceLimit is aligned to 16 bytes");

template <bool Q>
__global__ void __launch_bounds__(32 * SCAN_WARPS, 3) k_row_scan_seq(View vb, LevelScratch s) {
  extern __shared__ __align__(16) uint32_t scan_sm[];
  __shared__ uint32_t s_piece;
  __shared__ uint32_t s_cnt[SCAN_WARPS][SEQ_CLASSES], s_rows[SCAN_WARPS], s_last[SCAN_WARPS];
  __shared__ RowBest s_best[SCAN_WARPS];
  const uint32_t count = live_count(s, s.ctr->n_live_pieces, s.cap_scan);
  const StepLists lists = *s.step;
  const uint32_t C = vb.n_classes, lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t* smem = scan_sm + warp * SCAN_WORDS;
  uint2* ent = reinterpret_cast<uint2*>(smem + LIST_CAP / 2);
  uint32_t* sq = smem + LIST_CAP / 2 + 2 * SEQ_SLOTS;
  uint32_t* before = sq + SEQ_BEFORE;
  PieceLimit& pl = *reinterpret_cast<PieceLimit*>(sq + SEQ_WORDS);
  RowBest* best = s.rbest + (size_t)s.cap_nodes * vb.sel_stride;
  uint32_t item = blockIdx.x;
  while (true) {
    if (threadIdx.x == 0) {
      uint32_t pi = NONE;
      for (; item < count; item = gridDim.x + atomicAdd(&s.ctr->claim[ITEM_SCAN], 1u)) {
        const uint2 live = s.rscan[item];
        const uint32_t node = s.rpieces[live.x].node;
        const float known = __uint_as_float(*reinterpret_cast<volatile uint32_t*>(s.node_q + node));
        if (__uint_as_float(live.y) >= gain_bound(known, lists.nodes[node].n)) {
          pi = live.x;
          item = gridDim.x + atomicAdd(&s.ctr->claim[ITEM_SCAN], 1u);
          break;
        }
        best[live.x] = RowBest{dinf(), NONE, 0u, 0.f, 0.f};  // other pieces' scans have raised the bound
      }
      s_piece = pi;
    }
    __syncthreads();
    const uint32_t pi = s_piece;
    if (pi == NONE) break;
    const RowPiece pc = s.rpieces[pi];
    const ct_node nd = lists.nodes[pc.node];
    CT_JOB_REF(v, vb, nd.slot);
    const uint32_t n = nd.n, f = s.sel[(size_t)pc.node * v.sel_stride + pc.slot];
    const uint32_t* tot = lists.tot + (size_t)pc.node * C;
    const PieceStream whole = piece_stream(v, nd, pc, f, lists.scan_piece, smem);
    PieceStream part = whole;  // this warp's part
    if (part.dense) {
      const uint32_t per = ceil_div(whole.n_words, (uint32_t)SCAN_WARPS), w0 = min(warp * per, whole.n_words);
      part.base += w0 * 32;
      part.words += w0;
      part.n_words = min(per, whole.n_words - w0);
    } else {
      const uint32_t per = ceil_div(whole.count, (uint32_t)SCAN_WARPS), i0 = min(warp * per, whole.count);
      part.base += i0;
      part.count = min(per, whole.count - i0);
    }
    const uint32_t carry = lane < C && pc.npieces > 1 ? s.carry[(size_t)pi * C + lane] : 0u;
    const uint32_t total = lane < C ? tot[lane] : 0u;
    seq_totals(sq, tot, C);
    auto stage = [&](const PieceStream& ps, uint32_t b, uint32_t k, uint32_t sh) {
      __syncwarp();
#pragma unroll 4
      for (uint32_t i = lane; i < k; i += 32) {
        const uint2 e = ps.load(b + i);
        ent[seq_at(i, sh)] = seq_entry(e.x, e.y);
      }
      __syncwarp();
    };
    // counts of a staged run: by lane in w, in all on lane c for class c
    auto count_run = [&](uint32_t k, uint32_t sh, uint32_t(&w)[4]) {
      const uint32_t i0 = min(lane << sh, k);
      seq_count(ent + seq_at(i0, sh), min(k - i0, 1u << sh), w);
      uint32_t t[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) t[h] = h < 2 || C > 4 ? __reduce_add_sync(FULL, w[h]) : 0u;
      return lane < C ? seq_field(t, lane) : 0u;
    };
    // classes, rows and last value of the part; one run of it stays staged
    PieceStream ps = part;
    bool more = ps.fill();
    const bool staged = more && !ps.more() && ps.count <= SEQ_ROWS;
    uint32_t w[4] = {0u, 0u, 0u, 0u}, mine = 0, x_last = 0;
    while (more) {
      for (uint32_t b = 0; b < ps.count; b += SEQ_ROWS) {
        const uint32_t k = min(SEQ_ROWS, ps.count - b), sh = seq_shift(k);
        stage(ps, b, k, sh);
        mine += count_run(k, sh, w);
        x_last = ent[seq_at(k - 1, sh)].x;
      }
      more = ps.more() && ps.fill();
    }
    const uint32_t rows = __reduce_add_sync(FULL, mine);
    if (lane < SEQ_CLASSES) s_cnt[warp][lane] = mine;
    if (lane == 0) {
      s_rows[warp] = rows;
      s_last[warp] = x_last;
    }
    __syncthreads();
    uint32_t a = carry, prev = NONE;  // counts before the part; the nearest part before it with rows
    for (uint32_t k = 0; k < warp; ++k) {
      if (lane < SEQ_CLASSES) a += s_cnt[k][lane];
      if (s_rows[k]) prev = k;
    }
    if (lane < SEQ_CLASSES) before[lane] = a;
    __syncwarp();
    const uint32_t* known = s.node_q + pc.node;
    auto reaches = [&](uint32_t lo, uint32_t run) {  // may a candidate of the run win
      __syncwarp();
      limit_set(pl, lane < SEQ_CLASSES, lo, lo + run, total);
      __syncwarp();
      const float g = limit_of(pl, C, n);
      return g > 0.f && g >= gain_bound(__uint_as_float(*reinterpret_cast<const volatile uint32_t*>(known)), n);
    };
    SeqBest bb{dinf(), NONE, 0u, 0.f, 0.f};
    if (rows > 0 && reaches(a, mine)) {
      uint32_t p0 = __reduce_add_sync(FULL, a);
      // no candidate before the node's first row
      x_last = prev != NONE ? s_last[prev] : p0 > 0 ? value_before(v, whole, nd, pc, f, lists.scan_piece) : NONE;
      bool first = p0 == 0;
      auto scan_run = [&](uint32_t k, uint32_t sh) {
        if (first) x_last = ent[0].x;
        first = false;
        const uint32_t i0 = min(lane << sh, k), m = min(k - i0, 1u << sh);
        const uint32_t x_end = ent[seq_at(k - 1, sh)].x;
        const uint32_t xp = i0 > 0 && m > 0 ? ent[seq_at(i0 - 1, sh)].x : x_last;
        seq_scan(ent + seq_at(i0, sh), m, sh, w, sq, C, __uint_as_float(xp), p0, n, s.node_q + pc.node, bb);
        x_last = x_end;
        p0 += k;
      };
      if (staged) {
        scan_run(rows, seq_shift(rows));
      } else {
        ps = part;
        uint32_t keep = 0;
        while (ps.fill(keep)) {
          keep = 0;
          for (uint32_t b = 0; b < ps.count; b += SEQ_ROWS) {
            const uint32_t k = min(SEQ_ROWS, ps.count - b);
            if (k < SEQ_ROWS && ps.more()) {  // with the next batch
              keep = k;
              break;
            }
            const uint32_t sh = seq_shift(k);
            stage(ps, b, k, sh);
            const uint32_t run = count_run(k, sh, w), lo = lane < SEQ_CLASSES ? before[lane] : 0u;
            if (reaches(lo, run)) {
              scan_run(k, sh);
            } else {
              if (lane < SEQ_CLASSES) before[lane] = lo + run;
              __syncwarp();
              x_last = ent[seq_at(k - 1, sh)].x;
              first = false;
              p0 += k;
            }
          }
        }
      }
    }
    const uint32_t win = warp_best_lane(bb.score, bb.pos);
    if (win == NONE ? lane == 0 : lane == win) s_best[warp] = RowBest{bb.score, bb.pos, bb.pure, bb.xl, bb.xr};
    __syncthreads();
    if (warp == 0) {
      const RowBest rb = lane < SCAN_WARPS ? s_best[lane] : RowBest{dinf(), NONE, 0u, 0.f, 0.f};
      const uint32_t wl = warp_best_lane(rb.score, rb.pos);
      if (wl == NONE ? lane == 0 : lane == wl) best[pi] = rb;
    }
  }
}

// ------------------------------------------------------------------------
// Best candidate of a node (lowest score, then feature, then position), its
// record in the tree, and the pieces of its rows' split.
template <bool Q>
__device__ __forceinline__ void row_reduce_item(const View& vb, const StepLists& lists, const LevelScratch& s,
                                                const TreeView& tv, uint32_t w) {
  const uint32_t lane = lane_id();
  const ct_node nd = lists.nodes[w];
  CT_JOB_REF(v, vb, nd.slot);
  const uint32_t C = v.n_classes, nsel = s.nsel[w], n = nd.n;
  const uint32_t* sel = s.sel + (size_t)w * v.sel_stride;
  RowBest bb{dinf(), NONE, 0u, 0.f, 0.f};
  uint32_t bf = NONE;
  auto take = [&](const RowBest& rb, uint32_t f) {
    if (rb.score < bb.score || (rb.score == bb.score && (f < bf || (f == bf && rb.pos < bb.pos)))) {
      bb = rb;
      bf = f;
    }
  };
  if (n <= GROUP_ROWS) {
    for (uint32_t q = lane; q < nsel; q += 32)
      if (!is_virtual(v, sel[q])) take(s.rbest[(size_t)w * v.sel_stride + q], sel[q]);
  } else {
    const uint32_t pb = s.piece_base[w], pn = s.piece_cnt[w];
    const RowBest* best = s.rbest + (size_t)s.cap_nodes * vb.sel_stride;
    for (uint32_t q = pb + lane; q < pb + pn; q += 32)
      if (C > SEQ_CLASSES || ((s.rlive[q / LIMIT_PIECES] >> (q % LIMIT_PIECES)) & 1u))
        take(best[q], sel[s.rpieces[q].slot]);
  }
  if (v.vmask) {
    // a virtual feature's one candidate (the last low-value row), scored from
    // the class counts of its high-value rows; one selected slot per lane
    for (uint32_t q = lane; q < nsel; q += 32) {
      const uint32_t f = sel[q];
      if (!is_virtual(v, f)) continue;
      const float2 lh = v.vval[f];
      if (!is_candidate_sorted(lh.x, lh.y)) continue;
      const uint32_t* hc = s.vcls + ((size_t)w * v.n_features + f) * C;
      const uint32_t* tc = lists.tot + (size_t)w * C;
      int64_t sl = 0, sr = 0;
      for (uint32_t c = 0; c < C; ++c) {
        const int64_t r = hc[c], l = (int64_t)tc[c] - r;
        sl += l * l;
        sr += r * r;
      }
      const uint32_t nl = n - s.vcnt[(size_t)w * 64 + f];
      const Scored sc = score_at(sl, sr, nl, (double)n);
      take(RowBest{sc.score, nl - 1, sc.pure, lh.x, lh.y}, f);
    }
  }
  // lowest (score, feature, position) over the lanes
  const uint64_t sb = (uint64_t)__double_as_longlong(bb.score);
  const uint32_t mhi = __reduce_min_sync(FULL, (uint32_t)(sb >> 32));
  const uint32_t mlo = __reduce_min_sync(FULL, (uint32_t)(sb >> 32) == mhi ? (uint32_t)sb : NONE);
  bool tie = (uint32_t)(sb >> 32) == mhi && (uint32_t)sb == mlo;
  const uint32_t mf = __reduce_min_sync(FULL, tie ? bf : NONE);
  tie = tie && bf == mf;
  const uint32_t mp = __reduce_min_sync(FULL, tie ? bb.pos : NONE);
  tie = tie && bb.pos == mp;
  const uint32_t win = (uint32_t)__ffs(__ballot_sync(FULL, tie)) - 1;
  uint32_t split = mhi < 0x7ff00000u;
  const size_t at = (size_t)(nd.slot + tv.slot_base) * tv.capacity + nd.raw_id;
  const uint32_t* rows = row_list(v, nd.buf, nd.slot) + nd.start;
  const uint32_t npp = ceil_div(n, PART_PIECE);
  uint32_t sidx = 0, base = 0, children = 0;
  if (split && lane == win) {
    children = atomicAdd(&tv.n_nodes[nd.slot + tv.slot_base], 2u);
    if (children + 2ull > tv.capacity) {
      atomicOr(&s.ctr->error, DEV_ERR_CAPACITY);
      split = 0;
    } else {
      tv.left[at] = children;
      tv.right[at] = children + 1;
      tv.feature[at] = bf;
      tv.threshold[at] = midpoint(bb.xl, bb.xr);
      tv.value[at] = 0;
      sidx = atomicAdd(&s.ctr->n_splits, 1u);
      atomicAdd(&s.ctr->split_total, (unsigned long long)n);
      if (npp > 1) atomicAdd(&s.ctr->part_elems, (unsigned long long)n);
      base = npp == 1 ? atomicAdd(&s.ctr->n_part_pieces, 1u) : atomicAdd(&s.ctr->n_status, npp);
      if (sidx >= s.cap_nodes || (npp == 1 ? base >= s.cap_part : base + (uint64_t)npp > s.cap_mpart)) {
        atomicOr(&s.ctr->error, DEV_ERR_CAPACITY);
        split = 0;
      } else {
        s.rsplits[sidx] = RowSplit{w, bf, bb.pos + 1, children, bb.xl, bb.pure};
      }
    }
  }
  const uint32_t src = win & 31u;
  const bool leaf = mhi >= 0x7ff00000u;
  split = __shfl_sync(FULL, split, src);
  if (leaf) {
    const uint32_t value = first_row_class(v, rows, n);
    if (lane == 0) write_leaf(tv, at, value);
    return;
  }
  if (!split) return;
  sidx = __shfl_sync(FULL, sidx, src);
  base = __shfl_sync(FULL, base, src);
  for (uint32_t c = lane; c < C; c += 32) s.split_left[(size_t)sidx * C + c] = 0;
  PartPiece* list = npp == 1 ? s.part : s.mpart;
  for (uint32_t j = lane; j < npp; j += 32) {
    list[base + j] = PartPiece{sidx, j, npp, 0};
    if (npp > 1) s.msup[base + j] = 0;
  }
}

template <bool Q>
__global__ void __launch_bounds__(THREADS_PER_BLOCK) k_row_reduce(View v, LevelScratch s, TreeView tv) {
  const uint32_t count = live_count(s, s.ctr->n_nodes, s.cap_nodes);
  const StepLists sl = *s.step;
  for_items(count, &s.ctr->claim[ITEM_REDUCE], [&](uint32_t w) { row_reduce_item<Q>(v, sl, s, tv, w); });
}

// ------------------------------------------------------------------------
// Left flags of a piece of a split node's rows: a row goes left when its
// value is at most the split's xl, in the presort's order (a virtual feature:
// when it has the low value).  Counts the left rows' classes.  A split of one piece moves its
// rows at once; a longer one keeps the flags and counts for k_row_move.
template <bool Q>
__device__ __forceinline__ void row_mark_item(const View& vb, const StepLists& lists, const LevelScratch& s,
                                              uint32_t* cnt, uint32_t nm, uint32_t i) {
  const uint32_t C = vb.n_classes, lane = lane_id();
  const bool multi = i < nm;
  const PartPiece pp = multi ? s.mpart[i] : s.part[i - nm];
  const RowSplit sr = s.rsplits[pp.split];
  const ct_node nd = lists.nodes[sr.node];
  CT_JOB_REF(v, vb, nd.slot);
  const bool virt = is_virtual(v, sr.feature);
  const uint32_t* rows = row_list(v, nd.buf, nd.slot) + nd.start;
  const float* xf = v.x_fm + (size_t)sr.feature * v.n_rows;
  const uint32_t lo = pp.j * PART_PIECE, hi = min(lo + PART_PIECE, nd.n);
  const uint32_t xl = f32_order(sr.xl);
  const unsigned lt = lanemask_lt();
  uint32_t e[PART_ROUNDS];
  unsigned lm[PART_ROUNDS];
#pragma unroll
  for (uint32_t r = 0; r < PART_ROUNDS; ++r) {
    const uint32_t p = lo + r * 32 + lane;
    e[r] = p < hi ? __ldcs(rows + p) : 0u;
  }
  uint32_t left = 0;  // bit r: this lane's row of round r goes left
  if (virt) {
#pragma unroll
    for (uint32_t r = 0; r < PART_ROUNDS; ++r)
      if (lo + r * 32 + lane < hi)
        left |= (uint32_t)(!((__ldg(v.vrow + entry_row(v, e[r])) >> sr.feature) & 1ull)) << r;
  } else {
#pragma unroll
    for (uint32_t r = 0; r < PART_ROUNDS; ++r)
      if (lo + r * 32 + lane < hi) left |= (uint32_t)(f32_order(__ldg(xf + entry_row(v, e[r]))) <= xl) << r;
  }
  uint32_t nleft = 0;
#pragma unroll
  for (uint32_t r = 0; r < PART_ROUNDS; ++r) {
    lm[r] = __ballot_sync(FULL, (left >> r) & 1u);
    nleft += __popc(lm[r]);
  }
  uint32_t* out = s.split_left + (size_t)pp.split * C;
  if (C <= 8) {
    uint64_t pk = 0;  // 8-bit field per class, at most 16 rows per lane
#pragma unroll
    for (uint32_t r = 0; r < PART_ROUNDS; ++r)
      if ((left >> r) & 1u) pk += 1ull << (8 * (e[r] >> v.lab_shift));
    const uint32_t fh[2] = {(uint32_t)pk, (uint32_t)(pk >> 32)};
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
      if (4 * h >= C) break;
      const uint32_t ev = __reduce_add_sync(FULL, fh[h] & 0x00ff00ffu), od = __reduce_add_sync(FULL, (fh[h] >> 8) & 0x00ff00ffu);
      const uint32_t val = (lane & 1u ? od : ev) >> ((lane & 2u) * 8) & 0xffffu;
      if (lane < 4 && 4 * h + lane < C && val) atomicAdd(&out[4 * h + lane], val);
    }
  } else {
    for (uint32_t c = lane; c < C; c += 32) cnt[c] = 0;
    __syncwarp();
#pragma unroll
    for (uint32_t r = 0; r < PART_ROUNDS; ++r) {
      if (lo + r * 32 >= hi) break;
      const uint32_t c = (left >> r) & 1u ? e[r] >> v.lab_shift : NONE;
      const unsigned grp = __match_any_sync(FULL, c);
      if (c != NONE && (grp >> lane) == 1u) cnt[c] += __popc(grp);
      __syncwarp();
    }
    for (uint32_t c = lane; c < C; c += 32)
      if (cnt[c]) atomicAdd(&out[c], cnt[c]);
  }
  if (multi) {
    uint32_t mine = 0;
#pragma unroll
    for (uint32_t r = 0; r < PART_ROUNDS; ++r)
      if (lane == r) mine = lm[r];
    if (lane < PART_ROUNDS) s.mbits[(size_t)i * PART_ROUNDS + lane] = mine;
    if (lane == 0) {
      s.mleft[i] = nleft;
      atomicAdd(&s.msup[i - pp.j + pp.j / 32], nleft);
    }
    return;
  }
  if (nleft != sr.nl) {  // the scan and the rows disagree
    if (lane == 0) atomicOr(&s.ctr->error, DEV_ERR_INTERNAL);
    return;
  }
  uint32_t* dst = row_list(v, nd.buf ^ 1u, nd.slot) + nd.start;
  uint32_t run = 0;
#pragma unroll
  for (uint32_t r = 0; r < PART_ROUNDS; ++r) {
    const uint32_t p = r * 32 + lane;
    const uint32_t rl = run + __popc(lm[r] & lt);
    if (p < hi) dst[(left >> r) & 1u ? rl : sr.nl + (p - rl)] = e[r];
    run += __popc(lm[r]);
  }
}

template <bool Q>
__global__ void __launch_bounds__(THREADS_PER_BLOCK) k_row_mark(View v, LevelScratch s) {
  extern __shared__ uint32_t smem[];
  uint32_t* cnt = smem + (threadIdx.x >> 5) * v.n_classes;
  const uint32_t nm = live_count(s, s.ctr->n_status, s.cap_mpart);
  const uint32_t count = nm + live_count(s, s.ctr->n_part_pieces, s.cap_part);
  const StepLists sl = *s.step;
  for_items(count, &s.ctr->claim[ITEM_FILL], [&](uint32_t i) { row_mark_item<Q>(v, sl, s, cnt, nm, i); });
}

template <bool Q>
__global__ void __launch_bounds__(THREADS_PER_BLOCK) k_row_move(View vb, LevelScratch s) {
  const uint32_t count = live_count(s, s.ctr->n_status, s.cap_mpart);
  const StepLists lists = *s.step;
  const uint32_t lane = lane_id();
  const unsigned lt = lanemask_lt();
  for_items(count, &s.ctr->claim[ITEM_MOVE], [&](uint32_t i) {
    const PartPiece pp = s.mpart[i];
    const RowSplit sr = s.rsplits[pp.split];
    const ct_node nd = lists.nodes[sr.node];
    CT_JOB_REF(v, vb, nd.slot);
    const uint32_t lo = pp.j * PART_PIECE, hi = min(lo + PART_PIECE, nd.n);
    const uint32_t* rows = row_list(v, nd.buf, nd.slot) + nd.start;
    uint32_t* dst = row_list(v, nd.buf ^ 1u, nd.slot) + nd.start;
    uint32_t e[PART_ROUNDS];
#pragma unroll
    for (uint32_t r = 0; r < PART_ROUNDS; ++r) {
      const uint32_t p = lo + r * 32 + lane;
      e[r] = p < hi ? __ldcs(rows + p) : 0u;
    }
    const uint32_t mine = lane < PART_ROUNDS ? s.mbits[(size_t)i * PART_ROUNDS + lane] : 0u;
    // left rows of the split's earlier pieces: whole runs of 32 pieces, then
    // the pieces of this one's run
    const uint32_t first = i - pp.j, blk = pp.j / 32;
    uint32_t before = 0;
    for (uint32_t k = lane; k < blk; k += 32) before += s.msup[first + k];
    if (blk * 32 + lane < pp.j) before += s.mleft[first + blk * 32 + lane];
    uint32_t run = __reduce_add_sync(FULL, before);
#pragma unroll
    for (uint32_t r = 0; r < PART_ROUNDS; ++r) {
      const uint32_t p = lo + r * 32 + lane;
      const unsigned m = __shfl_sync(FULL, mine, r);
      const uint32_t rl = run + __popc(m & lt);
      if (p < hi) {
        const uint32_t d = (m >> lane) & 1u ? rl : sr.nl + (p - rl);
        if (d < nd.n) dst[d] = e[r];
      }
      run += __popc(m);
    }
    if (pp.j + 1 == pp.npieces && run != sr.nl && lane == 0) atomicOr(&s.ctr->error, DEV_ERR_INTERNAL);
  });
}

// ------------------------------------------------------------------------
// Children of the step's splits: leaves, subtree roots, and the next level's
// nodes with their class totals and constant-feature masks.
template <bool Q>
__device__ __forceinline__ void row_children_item(const View& vb, const StepLists& lists, const LevelScratch& s,
                                                  const TreeView& tv, uint32_t cap_next, uint32_t small_cut,
                                                  ct_node* small, uint32_t cap_small, uint32_t w) {
  const uint32_t lane = lane_id();
  const RowSplit sr = s.rsplits[w];
  const ct_node nd = lists.nodes[sr.node];
  CT_JOB_REF(v, vb, nd.slot);
  const uint32_t C = v.n_classes;
  for (uint32_t side = 0; side < 2; ++side) {
    ct_node ch;
    ch.slot = nd.slot;
    ch.n = side ? nd.n - sr.nl : sr.nl;
    ch.start = side ? nd.start + sr.nl : nd.start;
    ch.raw_id = sr.children + side;
    ch.key = child_key(nd.key, (int)side);
    ch.impurity = 1.0f;
    ch.buf = nd.buf ^ 1u;
    const bool pure = (sr.pure >> side) & 1u;
    if (pure || ch.n < v.mss) {
      const uint32_t* rows = row_list(v, ch.buf, ch.slot) + ch.start;
      const uint32_t value = pure ? rows[0] >> v.lab_shift : first_row_class(v, rows, ch.n);
      if (lane == 0) write_leaf(tv, (size_t)(nd.slot + tv.slot_base) * tv.capacity + ch.raw_id, value);
      continue;
    }
    if (small_cut != 0 && ch.n <= small_cut) {
      uint32_t placed = 0;
      if (lane == 0) {
        const uint32_t idx = atomicAdd(&s.ctr->n_small, 1u);
        if (idx < cap_small) {
          small[idx] = ch;
          atomicAdd(&s.ctr->small_total, (unsigned long long)ch.n);
          placed = 1;
        }
      }
      if (__shfl_sync(FULL, placed, 0)) continue;
      // the subtree list is full: the level steps split this child
    }
    uint32_t idx = 0;
    if (lane == 0) {
      idx = atomicAdd(&s.ctr->n_next, 1u);
      if (idx < cap_next) {
        lists.next[idx] = ch;
        atomicAdd(&s.ctr->next_total, (unsigned long long)ch.n);
      } else {
        atomicOr(&s.ctr->error, DEV_ERR_CAPACITY);
      }
    }
    idx = __shfl_sync(FULL, idx, 0);
    if (idx >= cap_next) continue;
    for (uint32_t c = lane; c < C; c += 32) {
      const uint32_t left = s.split_left[(size_t)w * C + c];
      lists.next_tot[(size_t)idx * C + c] = side ? lists.tot[(size_t)sr.node * C + c] - left : left;
    }
    if (lists.next_mask) {
      // the parent's constant features; a two-valued split feature is constant in both children
      const uint32_t mw = mask_words(v.n_features);
      const uint64_t* pm = lists.node_mask + (size_t)sr.node * v.mask_stride;
      uint64_t* cm = lists.next_mask + (size_t)idx * v.mask_stride;
      const bool tv2 = two_valued(v, sr.feature);
      for (uint32_t k = lane; k < mw; k += 32)
        cm[k] = pm[k] | (tv2 && (sr.feature >> 6) == k ? 1ull << (sr.feature & 63) : 0ull);
    }
  }
}

template <bool Q>
__global__ void __launch_bounds__(THREADS_PER_BLOCK)
k_row_children(View v, LevelScratch s, TreeView tv, uint32_t cap_next, uint32_t small_cut, ct_node* small,
               uint32_t cap_small) {
  const uint32_t count = live_count(s, s.ctr->n_splits, s.cap_nodes);
  const StepLists sl = *s.step;
  for_items(count, &s.ctr->claim[ITEM_CHILDREN], [&](uint32_t w) {
    row_children_item<Q>(v, sl, s, tv, cap_next, small_cut, small, cap_small, w);
  });
}

// ------------------------------------------------------------------------
// Subtrees of at most 32 rows, one warp each, one row per lane (lanes in
// feature-0 order, so a node's leaf label is its lowest lane's).  Most nodes
// here hold a few rows, so a node of n rows takes lane groups of
// g = next_pow2(n) lanes and evaluates 32 / g features of its permutation at
// once, one per group: the rows are gathered into every group, sorted there by
// 32-bit keys (rank above row index) and scanned with the exact score.  A lane
// keeps its best candidate over all features; one reduction at the end gives
// the node's.  A virtual feature's values come from the rows' value bits, read
// once per subtree.  Wide data (55 features per node): 11.6 ms per 200 trees
// with one feature at a time -> 4.6 ms.
struct RowSub {
  uint32_t mask;
  uint32_t raw;
  uint64_t key;
};

__device__ __forceinline__ void grow_rows(const View& v, const LevelScratch& s, const TreeView& tv, uint32_t tslot,
                                          uint32_t row, uint32_t lab, uint64_t vbits, RowSub cur, RowSub* stack,
                                          uint8_t* map, uint32_t lane) {
  const uint32_t F = v.n_features, m = v.max_features;
  const size_t toff = (size_t)tslot * tv.capacity;
  const unsigned lt = lanemask_lt();
  int sp = 0;
  while (true) {
    const uint32_t mask = cur.mask, n = __popc(mask);
    const bool in = (mask >> lane) & 1u;
    const uint32_t tcls = __popc(__match_any_sync(FULL, in ? lab : NONE));  // rows of this row's class
    const int32_t st2 = (int32_t)__reduce_add_sync(FULL, in ? tcls : 0u);
    // lane groups: lane r of every group holds the node's r-th row
    const uint32_t lg = n <= 2 ? 1u : 32u - (uint32_t)__clz((int)(n - 1)), g = 1u << lg;
    const uint32_t r = lane & (g - 1), q = lane >> lg, base = lane - r, per = 32u >> lg;
    const unsigned gmask = (g == 32 ? FULL : (1u << g) - 1u) << base;
    const bool valid = r < n;
    if (in) map[__popc(mask & lt)] = (uint8_t)lane;
    __syncwarp();
    const uint32_t src = map[valid ? r : 0u];
    __syncwarp();
    const uint32_t crow = __shfl_sync(FULL, row, src), clab = __shfl_sync(FULL, lab, src),
                   ct = __shfl_sync(FULL, tcls, src);
    uint64_t cvb = 0;
    if (v.vmask)
      cvb = (uint64_t)__shfl_sync(FULL, (uint32_t)vbits, src) |
            ((uint64_t)__shfl_sync(FULL, (uint32_t)(vbits >> 32), src) << 32);
    const double nn = (double)n;
    double best = dinf();
    uint32_t bf = NONE, bpure = 0;
    float bxl = 0.f, bxr = 0.f;
    uint32_t taken = 0;
    uint32_t perm = feature_perm(min(lane, F - 1), F, cur.key, v.feistel_h);  // permutation positions [0, 32)
    uint32_t f_nx = __shfl_sync(FULL, perm, q);
    if (q >= F) f_nx = NONE;
    uint2 pr_nx = make_uint2(0u, 0u);
    if (valid && f_nx != NONE && !is_virtual(v, f_nx)) pr_nx = __ldg(v.pair + (size_t)f_nx * v.n_rows + crow);
    for (uint32_t i = 0; i < F && taken < m; i += per) {
      const uint32_t f = f_nx;
      const uint2 pr = pr_nx;
      if (i + per < F) {  // the next features' values are gathered while these are sorted and scanned
        if (((i + per) & 31u) == 0u) perm = feature_perm(min(i + per + lane, F - 1), F, cur.key, v.feistel_h);
        f_nx = __shfl_sync(FULL, perm, (i + per + q) & 31u);
        if (i + per + q >= F) f_nx = NONE;
        if (valid && f_nx != NONE && !is_virtual(v, f_nx)) pr_nx = __ldg(v.pair + (size_t)f_nx * v.n_rows + crow);
      }
      uint32_t rank = pr.x;
      float xv = __uint_as_float(pr.y);
      if (f != NONE && is_virtual(v, f)) {
        const float2 lh = v.vval[f];
        rank = (uint32_t)(cvb >> f) & 1u;
        xv = rank ? lh.y : lh.x;
      }
      const uint32_t ord = f32_order(xv);
      const uint32_t o0 = __shfl_sync(FULL, ord, base);
      const bool varies = (__ballot_sync(FULL, valid && f != NONE && ord != o0) & gmask) != 0u;
      const unsigned um = __ballot_sync(FULL, varies && r == 0);
      if (um == 0u) continue;
      const bool use = varies && taken + __popc(um & ((1u << base) - 1u)) < m;
      taken += __popc(um);
      uint32_t key = valid ? (rank << 5) | r : NONE;
#pragma unroll
      for (uint32_t size = 2; size <= 32; size <<= 1) {
        if (size > g) break;
#pragma unroll
        for (uint32_t j = size >> 1; j > 0; j >>= 1) {
          const uint32_t o = __shfl_xor_sync(FULL, key, j);
          const bool lower = ((r & size) == 0u) == ((r & j) == 0u);  // size = g: ascending
          key = lower ? min(key, o) : max(key, o);
        }
      }
      const uint32_t from = base + (key & (g - 1));
      const float x = __shfl_sync(FULL, xv, from);
      const uint32_t c = __shfl_sync(FULL, clab, from), t = __shfl_sync(FULL, ct, from);
      const float xn = __shfl_down_sync(FULL, x, 1);
      const unsigned grp = __match_any_sync(FULL, valid ? c | (q << 16) : NONE);
      uint32_t incl = valid ? (2u * (uint32_t)__popc(grp & lt) + 1u) | (t << 16) : 0u;
#pragma unroll
      for (uint32_t d = 1; d < 32; d <<= 1) {
        if (d >= g) break;
        const uint32_t o = __shfl_up_sync(FULL, incl, d);
        if (r >= d) incl += o;
      }
      if (use && r + 1 < n && is_candidate_sorted(x, xn)) {
        const int32_t SL = (int32_t)(incl & 0xffffu);
        const Scored sc = score_at(SL, st2 - 2 * (int32_t)(incl >> 16) + SL, r + 1, nn);
        if (sc.score < best || (sc.score == best && f < bf)) {
          best = sc.score;
          bf = f;
          bpure = sc.pure;
          bxl = x;
          bxr = xn;
        }
      }
    }
    // lowest (score, feature, position) over the lanes
    const uint64_t sb = (uint64_t)__double_as_longlong(best);
    const uint32_t mhi = __reduce_min_sync(FULL, (uint32_t)(sb >> 32));
    bool split = mhi < 0x7ff00000u;
    unsigned left = 0;
    uint32_t c0 = 0;
    if (split) {
      const uint32_t mlo = __reduce_min_sync(FULL, (uint32_t)(sb >> 32) == mhi ? (uint32_t)sb : NONE);
      bool tie = (uint32_t)(sb >> 32) == mhi && (uint32_t)sb == mlo;
      const uint32_t mf = __reduce_min_sync(FULL, tie ? bf : NONE);
      tie = tie && bf == mf;
      const uint32_t mr = __reduce_min_sync(FULL, tie ? r : NONE);
      const uint32_t win = (uint32_t)__ffs(__ballot_sync(FULL, tie && r == mr)) - 1;
      bf = mf;
      bpure = __shfl_sync(FULL, bpure, win);
      bxl = __shfl_sync(FULL, bxl, win);
      bxr = __shfl_sync(FULL, bxr, win);
      bool low = false;
      if (in) {
        if (is_virtual(v, bf)) low = !((vbits >> bf) & 1ull);
        else low = f32_order(__ldg(v.x_fm + (size_t)bf * v.n_rows + row)) <= f32_order(bxl);
      }
      left = __ballot_sync(FULL, low);
      if (lane == 0) {
        c0 = atomicAdd(&tv.n_nodes[tslot], 2u);
        if (c0 + 2ull > tv.capacity) {
          atomicOr(&s.ctr->error, DEV_ERR_CAPACITY);
          split = false;
        }
      }
      split = __shfl_sync(FULL, split, 0);
      c0 = __shfl_sync(FULL, c0, 0);
    }
    if (!split) {
      const uint32_t value = __shfl_sync(FULL, lab, __ffs(mask) - 1);
      if (lane == 0) write_leaf(tv, toff + cur.raw, value);
    } else {
      if (lane == 0) {
        tv.left[toff + cur.raw] = c0;
        tv.right[toff + cur.raw] = c0 + 1;
        tv.feature[toff + cur.raw] = bf;
        tv.threshold[toff + cur.raw] = midpoint(bxl, bxr);
        tv.value[toff + cur.raw] = 0;
      }
      for (uint32_t side = 0; side < 2; ++side) {
        const uint32_t cm = side ? mask & ~left : left;
        if (((bpure >> side) & 1u) || (uint32_t)__popc(cm) < v.mss) {
          const uint32_t value = __shfl_sync(FULL, lab, __ffs(cm) - 1);
          if (lane == 0) write_leaf(tv, toff + c0 + side, value);
        } else if (sp < 33) {
          if (lane == 0) stack[sp] = RowSub{cm, c0 + side, child_key(cur.key, (int)side)};
          ++sp;
        } else {
          if (lane == 0) atomicOr(&s.ctr->error, DEV_ERR_INTERNAL);
        }
      }
    }
    __syncwarp();
    if (sp == 0) break;
    --sp;
    cur = stack[sp];
    __syncwarp();
  }
}

template <bool Q>
__global__ void __launch_bounds__(THREADS_PER_BLOCK, 6)
k_row_subtree(View vb, const ct_node* __restrict__ small, LevelScratch s, TreeView tv, uint32_t cap_small) {
  __shared__ RowSub stack_all[WARPS_PER_BLOCK][33];
  __shared__ uint8_t map_all[WARPS_PER_BLOCK][32];
  const uint32_t lane = lane_id();
  const uint32_t count = live_count(s, s.ctr->n_small, cap_small);
  for_items(count, &s.ctr->claim[ITEM_SUBTREE], [&](uint32_t w) {
    const ct_node nd = small[w];
    CT_JOB_REF(v, vb, nd.slot);
    const uint32_t* rows = row_list(v, nd.buf, nd.slot) + nd.start;
    const bool have = lane < nd.n;
    uint32_t e = have ? rows[lane] : 0u;
    // lanes in feature-0 order
    const uint32_t k0 = have ? (__ldg(&v.pair[entry_row(v, e)].x) << 5) | lane : NONE;
    uint32_t sk[1] = {k0};
    warp_sort_keys<1>(sk, lane);
    e = __shfl_sync(FULL, e, sk[0] & 31u);
    const uint32_t row = have ? entry_row(v, e) : 0u;
    const uint32_t lab = have ? e >> v.lab_shift : NONE;
    const uint64_t vbits = have && v.vmask ? __ldg(v.vrow + row) : 0ull;
    const RowSub cur{nd.n >= 32 ? FULL : ((1u << nd.n) - 1u), nd.raw_id, nd.key};
    grow_rows(v, s, tv, nd.slot + tv.slot_base, row, lab, vbits, cur, stack_all[threadIdx.x >> 5],
              map_all[threadIdx.x >> 5], lane);
  });
}

uint32_t sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return (uint32_t)std::max(1, sms);
}

inline uint32_t clamp32(uint64_t x) { return x > 0xffffffffull ? 0xffffffffu : (uint32_t)x; }

// A kernel of CTAs that claim bitmap work: as many as are resident at once.
template <typename K, typename... A>
int launch_bitmap(K kernel, int threads, size_t smem, uint32_t items, cudaStream_t st, const A&... args) {
  CT_TRY(allow_smem(kernel, (int)ORDER_SMEM_MAX));
  int per = 1;
  CT_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem));
  kernel<<<std::min<uint32_t>(items, sm_count() * (uint32_t)std::max(1, per)), threads, smem, st>>>(args...);
  CT_CUDA_TRY(cudaGetLastError());
  return CT_OK;
}

template <bool Q>
int row_step(const View& v, const LevelScratch& s, LevelBounds b, uint32_t n_max, const TreeView& tv,
             uint32_t cap_next, uint32_t small_cut, ct_node* small, uint32_t cap_small, const ForkStreams* fork,
             cudaStream_t st) {
  Prof* pf = current_prof();
  const uint32_t C = v.n_classes;
  const size_t sm1 = (size_t)WARPS_PER_BLOCK * C * sizeof(uint32_t);
  const uint64_t nodes = std::min<uint64_t>(b.nodes, s.cap_nodes);
  const uint32_t sms = sm_count();
  if (v.vmask) {
    pf->begin(CT_K_SCAN);
    CT_TRY(launch_virtual_counts(v, s, nodes, s.cap_vpieces, st));
    pf->end();
    pf->launched(CT_K_SCAN, 2);
  }
  pf->begin(CT_K_SELECT);
  k_row_select<Q><<<grid_for(k_row_select<Q>, nodes, 0, true), THREADS_PER_BLOCK, 0, st>>>(v, s);
  pf->launched(CT_K_SELECT);
  if (n_max > SELECT_ROWS) {  // (a bitmap of several slices needs more rows than that)
    k_row_select_big<Q><<<std::min(s.cap_big, sms), 512, 0, st>>>(v, s);
    pf->launched(CT_K_SELECT);
  }
  pf->end();
  // The orders and scans of the size classes are independent: in a graph they
  // are branches, so the latency of one class's kernels (a level has few large
  // nodes) hides behind the others'.  The bitmaps' chain is the longest and
  // stays on st.
  cudaStream_t br[ForkStreams::N];
  for (int i = 0; i < ForkStreams::N; ++i) br[i] = fork ? fork->st[i] : st;
  const bool forked = fork && n_max > GROUP_SMALL_ROWS;
  if (forked) {
    CT_CUDA_TRY(cudaEventRecord(fork->fork, st));
    for (int i = 0; i < ForkStreams::N; ++i) CT_CUDA_TRY(cudaStreamWaitEvent(br[i], fork->fork, 0));
  } else {
    for (int i = 0; i < ForkStreams::N; ++i) br[i] = st;
  }
  const size_t smw = (size_t)WARPS_PER_BLOCK * warp_item_words(C) * sizeof(uint32_t);
  if (n_max > GROUP_ROWS) {
    pf->begin(CT_K_PARTITION);
    CT_TRY(launch_bitmap(k_row_bits<Q>, BITS_THREADS, (size_t)bits_words(n_max) * 4, s.cap_units, st, v, s, n_max));
    pf->launched(CT_K_PARTITION);
    if (!row_dense(GROUP_ROWS + 1, n_max)) {  // some nodes above the group size may be sparse
      CT_TRY(launch_bitmap(k_row_order<Q>, ORDER_THREADS, order_smem(n_max), s.cap_order, st, v, s));
      pf->launched(CT_K_PARTITION);
    }
    pf->end();
  }
  pf->begin(CT_K_SCAN);
  if (n_max > GROUP_SMALL_ROWS) {
    const size_t smg = group_words<GROUP_WARPS>(C, n_max) * sizeof(uint32_t);
    if (group_by_buckets<GROUP_WARPS>(n_max))
      CT_TRY(launch_bitmap(k_row_group<Q, GROUP_WARPS, true>, 32 * GROUP_WARPS, smg, s.cap_order, br[0], v, s, n_max));
    else
      CT_TRY(launch_bitmap(k_row_group<Q, GROUP_WARPS, false>, 32 * GROUP_WARPS, smg, s.cap_order, br[0], v, s, n_max));
    pf->launched(CT_K_SCAN);
  }
  if (n_max > WARP_ROWS) {
    const size_t smg = group_words<GROUP_SMALL_WARPS>(C, n_max) * sizeof(uint32_t);
    if (group_by_buckets<GROUP_SMALL_WARPS>(n_max))
      CT_TRY(launch_bitmap(k_row_group<Q, GROUP_SMALL_WARPS, true>, 32 * GROUP_SMALL_WARPS, smg, s.cap_order, br[1], v, s,
                           n_max));
    else
      CT_TRY(launch_bitmap(k_row_group<Q, GROUP_SMALL_WARPS, false>, 32 * GROUP_SMALL_WARPS, smg, s.cap_order, br[1], v,
                           s, n_max));
    pf->launched(CT_K_SCAN);
  }
  k_row_warp<Q><<<grid_for(k_row_warp<Q>, s.cap_w, smw, true), THREADS_PER_BLOCK, smw, br[2]>>>(v, s);
  pf->launched(CT_K_SCAN);
  if (n_max > GROUP_ROWS) {
    const size_t smh = (size_t)WARPS_PER_BLOCK * hist_words(C) * sizeof(uint32_t);
    const size_t sms2 = (size_t)WARPS_PER_BLOCK * scan_words(C) * sizeof(uint32_t);
    // every list is a bitmap whose classes k_row_bits counts, unless some are
    // sparse or the shortest pieces are too many for it
    const bool hist = !row_dense(GROUP_ROWS + 1, n_max) || (uint64_t)ceil_div(n_max, 1024) * C > BITS_COUNTS;
    if (hist) k_row_hist<Q><<<grid_for(k_row_hist<Q>, s.cap_scan, smh, true), THREADS_PER_BLOCK, smh, st>>>(v, s);
    k_row_carry<<<grid_for(k_row_carry, (uint64_t)s.cap_order * C, 0, true), THREADS_PER_BLOCK, 0, st>>>(s, C);
    if (C <= SEQ_CLASSES) {
      k_row_bound<Q><<<sms * 8, 256, 0, st>>>(v, s);
      k_row_limit<<<grid_for(k_row_limit, ceil_div(s.cap_scan, LIMIT_PIECES), 0, true), THREADS_PER_BLOCK, 0, st>>>(s, C);
      pf->launched(CT_K_SCAN, 2);
    }
    if (C <= SEQ_CLASSES)
      CT_TRY(launch_bitmap(k_row_scan_seq<Q>, 32 * SCAN_WARPS, SCAN_WARPS * SCAN_WORDS * sizeof(uint32_t), s.cap_scan, st,
                           v, s));
    else
      k_row_scan<Q><<<grid_for(k_row_scan<Q>, s.cap_scan, sms2, true), THREADS_PER_BLOCK, sms2, st>>>(v, s);
    pf->launched(CT_K_SCAN, hist ? 3 : 2);
  }
  pf->end();
  if (forked)
    for (int i = 0; i < ForkStreams::N; ++i) {
      CT_CUDA_TRY(cudaEventRecord(fork->join[i], br[i]));
      CT_CUDA_TRY(cudaStreamWaitEvent(st, fork->join[i], 0));
    }
  pf->begin(CT_K_REDUCE);
  k_row_reduce<Q><<<grid_for(k_row_reduce<Q>, nodes, 0, true), THREADS_PER_BLOCK, 0, st>>>(v, s, tv);
  pf->end();
  pf->launched(CT_K_REDUCE);
  pf->begin(CT_K_MARK);
  k_row_mark<Q><<<grid_for(k_row_mark<Q>, (uint64_t)s.cap_mpart + s.cap_part, sm1, true), THREADS_PER_BLOCK, sm1, st>>>(
      v, s);
  pf->end();
  pf->launched(CT_K_MARK);
  if (n_max > PART_PIECE) {
    pf->begin(CT_K_PARTITION);
    k_row_move<Q><<<grid_for(k_row_move<Q>, s.cap_mpart, 0, true), THREADS_PER_BLOCK, 0, st>>>(v, s);
    pf->end();
    pf->launched(CT_K_PARTITION);
  }
  pf->begin(CT_K_CHILDREN);
  k_row_children<Q><<<grid_for(k_row_children<Q>, nodes, 0, true), THREADS_PER_BLOCK, 0, st>>>(
      v, s, tv, cap_next, small_cut, small, cap_small);
  pf->end();
  pf->launched(CT_K_CHILDREN);
  CT_CUDA_TRY(cudaGetLastError());
  return CT_OK;
}

}  // namespace

// ---------------------------------------------------------------------------
// Sorted planes (8 bytes per row and slot) that fit behind the row list in
// each of the two list buffers (4 bytes per row and slot of n_features *
// index_bytes); the others take workspace.  (With all of them there as soon as
// one did not fit, a fit of 1,000,000 x 100 rows, all features selected, 100
// trees, asked for 97 GB of workspace instead of 18.)
uint32_t rows_planes_in_lists(const ct_problem* p) {
  const uint64_t per_row = (uint64_t)p->n_features * p->index_bytes;
  return per_row < 16 ? 0u : (uint32_t)std::min<uint64_t>((per_row - 8) / 8, 1u << 20);
}
bool rows_have_large(uint32_t n_rows) { return n_rows > GROUP_ROWS; }
uint32_t rows_planes_in_workspace(const ct_problem* p) {
  const uint32_t needed = rows_have_large(p->n_rows) ? std::min(p->max_features, p->n_features) : 0u;
  const uint32_t there = 2 * rows_planes_in_lists(p);
  return needed > there ? needed - there : 0u;
}

// Tables on which list growth is the faster of the two: row-list growth sorts
// each selected feature anew, in shared memory that holds fewer items at once
// the more rows there are, so with many rows, many classes (a scan by class
// match) and a good part of the features selected it loses.  ct_fit and the
// read-back of 8 trees, lists / rows: 700,000 x 20, 20 classes, 10 selected 30 /
// 46 ms; 8 classes, 20 selected 39 / 52; 950,000 x 20, 20 classes, 5 selected 31 /
// 42; 450,000 x 20, 20 classes, 20 selected 30 / 34; but 560,000 x 20, 20 classes,
// 5 selected 22 / 17; 700,000 x 20, 4 classes, 10 selected 23 / 21; 581,012 x 54
// covtype-shaped, all selected 32 / 19.
static bool rows_slower(const ct_problem* p) {
  const uint64_t m = std::min(p->max_features, p->n_features), F = p->n_features;
  return (p->n_rows > 600000 && p->n_classes >= SEQ_CLASSES && 8 * m >= F) ||
         (p->n_rows > 400000 && p->n_classes > SEQ_CLASSES && 2 * m >= F);
}

// A row id and a label share 32 bits, the row list fits a list buffer, and the
// rank bitmap fits shared memory.
bool rows_possible(const ct_problem* p) {
  if (rows_slower(p)) return false;
  const uint32_t row_bits = p->n_rows > 1 ? 32u - (uint32_t)__builtin_clz(p->n_rows - 1) : 1u;
  const uint32_t lab_bits = p->n_classes > 1 ? 32u - (uint32_t)__builtin_clz(p->n_classes - 1) : 0u;
  return row_bits + lab_bits <= 32 && row_bits <= 22 && (uint64_t)p->n_features * p->index_bytes >= 4 &&
         order_smem(p->n_rows) <= ORDER_SMEM_MAX && (size_t)bits_words(p->n_rows) * 4 <= ORDER_SMEM_MAX &&
         (p->n_rows <= WARP_ROWS ||
          group_words<GROUP_SMALL_WARPS>(p->n_classes, p->n_rows) * sizeof(uint32_t) <= ORDER_SMEM_MAX) &&
         (p->n_rows <= GROUP_SMALL_ROWS ||
          group_words<GROUP_WARPS>(p->n_classes, p->n_rows) * sizeof(uint32_t) <= ORDER_SMEM_MAX) &&
         p->n_features < 65535u;
}

bool carve_row_scratch(Arena& a, const View& v, LevelBounds b, uint32_t scan_piece, LevelScratch* s, bool virt) {
  const size_t C = v.n_classes, m = v.sel_stride;
  LevelScratch& t = *s;
  t = LevelScratch{};
  t.cap_nodes = clamp32(b.nodes);
  // Nodes above the group size make pieces: a sparse one at most n / piece + 1
  // per slot, a dense one at most 2 n / piece + 1 (its runs of ranks hold half a
  // piece at the least) or, at the longest run and 64 n >= n_rows, n / 512 + 1.
  const uint64_t large = b.samples / (WARP_ROWS + 1);  // nodes above the warp size
  t.cap_scan = clamp32(m * (std::max<uint64_t>(2 * b.samples / scan_piece, b.samples / 512) +
                            b.samples / (GROUP_ROWS + 1)) + 1);
  t.cap_order = clamp32(m * large + 1);
  t.cap_units = clamp32(m * (b.samples / BITS_SLICE + large) + 1);
  t.cap_w = clamp32(m * b.nodes + 1);
  t.cap_part = t.cap_nodes;
  t.cap_mpart = clamp32(b.samples / PART_PIECE + b.samples / (PART_PIECE + 1) + 1);
  t.cap_big = clamp32(b.samples / SELECT_ROWS + 1);
  t.cap_vpieces = virt ? clamp32(b.samples / MIN_VPIECE + b.nodes + 1) : 0u;
  t.ctr = a.take<Counters>(1);
  t.step = a.take<StepLists>(1);
  t.sel = a.take<uint32_t>(t.cap_nodes * m);
  t.nsel = a.take<uint32_t>(t.cap_nodes);
  t.node_q = a.take<uint32_t>(t.cap_nodes);
  t.piece_base = a.take<uint32_t>(t.cap_nodes);
  t.piece_cnt = a.take<uint32_t>(t.cap_nodes);
  t.witems = a.take<uint2>(t.cap_w);
  t.oitems = a.take<uint2>(t.cap_order);
  t.bunits = a.take<uint4>(t.cap_units);
  t.bzero = a.take<uint4>(t.cap_order);
  t.citems = a.take<uint2>(t.cap_order);
  t.gsmall = a.take<uint2>(t.cap_order);
  t.glarge = a.take<uint2>(t.cap_order);
  t.rpieces = a.take<RowPiece>(t.cap_scan);
  t.rbest = a.take<RowBest>((size_t)t.cap_nodes * m + t.cap_scan);
  t.rscan = C <= SEQ_CLASSES ? a.take<uint2>(t.cap_scan) : nullptr;
  t.rlive = C <= SEQ_CLASSES ? a.take<uint8_t>(t.cap_scan / LIMIT_PIECES + 1) : nullptr;
  t.carry = a.take<uint32_t>((size_t)t.cap_scan * C);
  t.rsplits = a.take<RowSplit>(t.cap_nodes);
  t.split_left = a.take<uint32_t>((size_t)t.cap_nodes * C);
  t.part = a.take<PartPiece>(t.cap_part);
  t.mpart = a.take<PartPiece>(t.cap_mpart);
  t.mbits = a.take<uint32_t>((size_t)t.cap_mpart * PART_ROUNDS);
  t.mleft = a.take<uint32_t>(t.cap_mpart);
  t.msup = a.take<uint32_t>(t.cap_mpart);
  t.big_nodes = a.take<uint32_t>(t.cap_big);
  t.vcnt = virt ? a.take<uint32_t>((size_t)t.cap_nodes * 64) : nullptr;
  t.vcls = virt ? a.take<uint32_t>((size_t)t.cap_nodes * v.n_features * C) : nullptr;
  t.vpieces = virt ? a.take<uint2>(t.cap_vpieces) : nullptr;
  return a.ok();
}

template <typename IdxT, typename LabT>
static void row_pairs(const View& v, const ct_problem* p, uint2* pair, uint2* ranked, uint32_t* rank,
                      cudaStream_t st) {
  const dim3 grid(std::min<uint32_t>(ceil_div(p->n_rows, 1024), 512u), p->n_features);
  k_row_pairs<IdxT, LabT><<<grid, 256, 0, st>>>(reinterpret_cast<const IdxT*>(p->presort), p->x_fm,
                                                reinterpret_cast<const LabT*>(p->labels), p->n_rows, v.vmask, pair,
                                                ranked, rank);
}
int launch_row_pairs(const View& v, const ct_problem* p, uint2* pair, uint2* ranked, uint32_t* rank, cudaStream_t st) {
  if (p->index_bytes == 2 && p->label_bytes == 1) row_pairs<uint16_t, uint8_t>(v, p, pair, ranked, rank, st);
  else if (p->index_bytes == 2) row_pairs<uint16_t, uint16_t>(v, p, pair, ranked, rank, st);
  else if (p->label_bytes == 1) row_pairs<uint32_t, uint8_t>(v, p, pair, ranked, rank, st);
  else row_pairs<uint32_t, uint16_t>(v, p, pair, ranked, rank, st);
  CT_CUDA_TRY(cudaGetLastError());
  return CT_OK;
}

int launch_row_roots(const View& v, const ct_problem* p, uint32_t slot_lo, uint32_t n_slots, uint32_t tree_lo,
                     uint32_t* n_in, const TreeView& tv, ct_node* out, uint32_t* out_tot, uint32_t cap, Counters* ctr,
                     uint64_t* out_mask, const float2* vals, cudaStream_t st) {
  const size_t smem = ((size_t)(p->n_rows + 31) / 32 + v.n_classes) * sizeof(uint32_t);
  const uint32_t threads = p->n_rows >= 8192 ? 1024u : p->n_rows >= 1024 ? 512u : 128u;
  if (p->label_bytes == 1) {
    CT_TRY(allow_smem(k_row_roots<uint8_t>, (int)ORDER_SMEM_MAX));
    k_row_roots<uint8_t><<<n_slots, threads, smem, st>>>(v, p->seed, p->bootstrap, slot_lo, tree_lo, n_in, tv, out,
                                                         out_tot, cap, ctr, out_mask, vals);
  } else {
    CT_TRY(allow_smem(k_row_roots<uint16_t>, (int)ORDER_SMEM_MAX));
    k_row_roots<uint16_t><<<n_slots, threads, smem, st>>>(v, p->seed, p->bootstrap, slot_lo, tree_lo, n_in, tv, out,
                                                          out_tot, cap, ctr, out_mask, vals);
  }
  CT_CUDA_TRY(cudaGetLastError());
  return CT_OK;
}

int launch_row_step(const View& v, const LevelScratch& s, LevelBounds b, uint32_t n_max, const TreeView& tv,
                    uint32_t cap_next, uint32_t small_cut, ct_node* small, uint32_t cap_small, const ForkStreams* fork,
                    cudaStream_t st) {
  return v.jobs ? row_step<true>(v, s, b, n_max, tv, cap_next, small_cut, small, cap_small, fork, st)
                : row_step<false>(v, s, b, n_max, tv, cap_next, small_cut, small, cap_small, fork, st);
}

int launch_row_subtrees(const View& v, const ct_node* small, uint32_t cap_small, uint32_t bound, const LevelScratch& s,
                        const TreeView& tv, cudaStream_t st) {
  if (cap_small == 0 || bound == 0) return CT_OK;
  Prof* pf = current_prof();
  pf->begin(CT_K_SUBTREE);
  const uint32_t items = std::min(bound, cap_small);
  if (v.jobs)
    k_row_subtree<true><<<grid_for(k_row_subtree<true>, items, 0, true), THREADS_PER_BLOCK, 0, st>>>(v, small, s, tv,
                                                                                                      cap_small);
  else
    k_row_subtree<false><<<grid_for(k_row_subtree<false>, items, 0, true), THREADS_PER_BLOCK, 0, st>>>(v, small, s, tv,
                                                                                                        cap_small);
  pf->end();
  pf->launched(CT_K_SUBTREE);
  CT_CUDA_TRY(cudaGetLastError());
  return CT_OK;
}

}  // namespace ct
