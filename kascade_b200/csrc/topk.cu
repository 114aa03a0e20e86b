// Exact per-row Top-k (one CTA per row): the k-th largest score is bracketed from a sample, the few
// candidates inside the bracket are selected among exactly in shared memory, and the selected positions are
// written in ascending index order.
//
// Replaces the torch.topk call sites of the reference's efficient path
// (strategies/EfficientKascadeStrategy.py:82,90,111).
//
//   1. Bracket: 4096 (8192 for rows beyond 65536) evenly spaced samples of the row go into a 512-bin histogram
//      over the samples' own key range, and those in the bins around the sample ranks k/n * samples -/+
//      (5 sigma + 16) into a second one over just these bins; its bins give two keys lo <= hi.
//   2. One pass over the row: every warp owns a contiguous piece of it, counts its scores above hi and appends
//      its keys in [lo, hi] (a few per cent of the row) to a list of its own in shared memory.  If
//      count(> hi) < k <= count(> hi) + |lists|  and the lists fit, the k-th largest score is the
//      (k - count(> hi))-th largest of the lists: a radix select over them (9-bit digits of key - lo, only as
//      many as hi - lo has bits) finds it exactly, and every warp learns from its own list how many of its scores
//      lie above / at the threshold.  Rows of up to 4096 scores skip the sample: the whole row goes to the lists.
//   3. Otherwise (the sample misjudged the row, which the check above detects, or a list overflowed) the k-th
//      largest key is found by four 9/9/9/5-bit histogram passes over the row itself, and a counting pass
//      gives the warps their numbers.
//   4. The last pass writes the selected positions of every warp's piece in index order, with warp-local prefix
//      sums only, taking ties at the threshold from the lowest index upwards.
// The row is read from HBM once; the later passes find it in L1 / L2.
//
// A few long rows (the anchor layers of a decode step with a handful of sequences) would leave most SMs idle: a
// cluster of 2, 4 or 8 CTAs then takes a row together.  Each takes the whole sample and comes to the same bracket,
// streams its own piece of the row, and the lists of all of them (a few thousand keys) are gathered over distributed
// shared memory, so that the radix select needs no exchange either.
#include <cooperative_groups.h>

#include "common.cuh"

namespace kb200 {

constexpr int kTopkWarpsMax = 16;
constexpr int kDigit = 9;
constexpr int kTopkBins = 1 << kDigit;                            // 9-bit digits: one warp can search a histogram
constexpr int kMergedCap = 8192;                          // keys the gathered list of a cluster holds
// keys a warp's candidate list holds; the lists of a CTA hold 8192 together (4 warps: 4096)
constexpr int warp_list(int warps) { return warps == 16 ? 512 : 1024; }
constexpr int kListRow = 4096;                            // rows up to this length are selected from directly
constexpr int kTopkMergedBytes = kMergedCap * 4;            // dynamic shared memory of a cluster's CTA
constexpr int kTopkUnroll = 4;                            // 16-byte loads a lane keeps in flight in the streaming passes

// order-preserving map float -> uint32 (larger float <=> larger key)
__device__ __forceinline__ uint32_t float_key(float x) {
  const uint32_t b = __float_as_uint(x);
  return b ^ ((uint32_t)((int32_t)b >> 31) | 0x80000000u);   // flips all bits of a negative, the sign of the rest
}
// Keys of one 16-byte piece.  Positions beyond the row (only the row's last piece has any, and the lanes past
// the end) get key 0, which no score has (it would be a NaN with all bits set) and which the passes below never
// count: they compare against keys >= 1.
__device__ __forceinline__ void piece_keys(const float4& x, int i4, int n4, int n, uint32_t (&u)[4]) {
  u[0] = float_key(x.x); u[1] = float_key(x.y); u[2] = float_key(x.z); u[3] = float_key(x.w);
  if (i4 >= n4 - 1) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (i4 * 4 + e >= n) u[e] = 0u;
  }
}

template <int NW>                      // warps of a CTA
struct TopkShared {
  uint32_t hist[kTopkBins];
  uint32_t cand[NW * warp_list(NW)];
  uint32_t red[NW], red2[NW];
  uint32_t warp_gt[NW], warp_eq[NW], list_len[NW];
  uint32_t digit, remaining;
  uint32_t cta_gt, cta_cand, cta_max_list;               // clusters: scores above hi_key, list entries, longest list
  uint32_t cta_above, cta_equal;                         // clusters: scores above / at the threshold in this CTA's piece
  uint32_t list_at[8 * kTopkWarpsMax];                   // clusters: where each list starts in the gathered one
};

// Bin d of sh.hist with  count(bins > d) < r <= count(bins >= d)  (1 <= r <= total); every thread gets d and
// r - count(bins > d).  All threads of the CTA call it, after a barrier that completed the histogram; one warp
// does the search (16 bins per lane) - the per-row costs of this kernel are instructions, and sixteen warps
// searching together would issue ten times as many.
template <int NW>
__device__ __forceinline__ void find_bin(TopkShared<NW>& sh, uint32_t r, uint32_t& digit, uint32_t& rest) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == 0) {
    constexpr int kPer = kTopkBins / 32;
    uint32_t c[kPer], ssum = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) { c[i] = sh.hist[lane * kPer + i]; ssum += c[i]; }
    uint32_t suf = ssum;                                 // sum over lanes >= lane
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t v = __shfl_down_sync(0xFFFFFFFFu, suf, off);
      if (lane + off < 32) suf += v;
    }
    const uint32_t above = suf - ssum;                   // in the bins of higher lanes
    if (above < r && r <= above + ssum) {
      uint32_t acc = above;
#pragma unroll
      for (int i = kPer - 1; i >= 0; --i) {
        if (acc < r && acc + c[i] >= r) {
          sh.digit = (uint32_t)(lane * kPer + i);
          sh.remaining = r - acc;
        }
        acc += c[i];
      }
    }
  }
  __syncthreads();
  digit = sh.digit;
  rest = sh.remaining;
  __syncthreads();
}

// sum / minimum / maximum over the per-warp values of an array in shared memory: one load per lane and a few
// shuffles instead of a load per warp and thread
template <int NW>
__device__ __forceinline__ uint32_t warps_sum(const uint32_t (&a)[NW]) {
  uint32_t v = a[threadIdx.x & (NW - 1)];
#pragma unroll
  for (int off = NW / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
  return v;
}
template <int NW>
__device__ __forceinline__ uint32_t warps_min(const uint32_t (&a)[NW]) {
  uint32_t v = a[threadIdx.x & (NW - 1)];
#pragma unroll
  for (int off = NW / 2; off > 0; off >>= 1) v = min(v, __shfl_xor_sync(0xFFFFFFFFu, v, off));
  return v;
}
template <int NW>
__device__ __forceinline__ uint32_t warps_max(const uint32_t (&a)[NW]) {
  uint32_t v = a[threadIdx.x & (NW - 1)];
#pragma unroll
  for (int off = NW / 2; off > 0; off >>= 1) v = max(v, __shfl_xor_sync(0xFFFFFFFFu, v, off));
  return v;
}
template <int NW>
__device__ __forceinline__ uint32_t block_sum(TopkShared<NW>& sh, uint32_t v) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
  if (lane == 0) sh.red[warp] = v;
  __syncthreads();
  const uint32_t t = warps_sum(sh.red);
  __syncthreads();
  return t;
}

// Key budget of a decode step over a cache of n tokens (strategies/KascadeStrategy.py:127-129; up to 128 tokens
// attend to everything), computed per row here: as tensors the budgets took a dozen element-wise launches per anchor
// layer, more host time than the rest of the layer.
struct DecodeBudget {
  const int32_t* seq_lens;      // [rows / groups], or NULL: n_valid / k_row say how much to select
  int groups;
  double share;                 // k / 100
  int tile;
};
__device__ __forceinline__ int decode_budget(const DecodeBudget& d, int n) {
  if (n <= 128) return n;
  return min(max(128, (int)(d.share * (double)n)), n) - d.tile;
}

template <int C, int kTopkWarps>       // CTAs that share a row (a cluster of C), warps per CTA
__global__ void __launch_bounds__(kTopkWarps * 32, 32 / kTopkWarps)
topk_select_kernel(const float* scores, int64_t row_stride, int n_cols,
                   const int32_t* n_valid, const int32_t* k_row, int k_max,
                   int32_t* __restrict__ out_idx, int64_t idx_stride, int32_t* __restrict__ out_count,
                   int64_t rows, const DecodeBudget budget) {
  namespace cg = cooperative_groups;
  using TopkShared = TopkShared<kTopkWarps>;
  constexpr int kTopkThreads = kTopkWarps * 32, kWarpList = warp_list(kTopkWarps);
  __shared__ TopkShared sh;
  extern __shared__ uint32_t merged[];                    // C > 1: the lists of all CTAs of the cluster
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = C > 1 ? (int)cg::this_cluster().block_rank() : 0;
  pdl_wait();

  for (int64_t row = blockIdx.x / C; row < rows; row += gridDim.x / C) {
    int n, k;
    if (budget.seq_lens) {
      n = budget.seq_lens[row / budget.groups];
      k = min(decode_budget(budget, n), k_max);
    } else {
      n = n_valid ? n_valid[row] : n_cols;
      k = k_row ? min(k_row[row], k_max) : k_max;
    }
    n = max(0, min(n, n_cols));
    k = max(0, min(k, n));
    int32_t* out = out_idx + row * idx_stride;
    if (tid == 0 && rank == 0 && out_count) out_count[row] = k;
    if (k == 0) continue;
    if (k == n) {  // every candidate is selected
      for (int i = rank * kTopkThreads + tid; i < n; i += C * kTopkThreads) out[i] = i;
      continue;
    }
    const float4* row4 = reinterpret_cast<const float4*>(scores + row * row_stride);
    const int n4 = (n + 3) >> 2;
    // every warp (of the cluster) owns the 16-byte pieces [w_begin, w_end) of the row
    const int seg4 = (n4 + C * kTopkWarps - 1) / (C * kTopkWarps);
    const int w_begin = min((rank * kTopkWarps + warp) * seg4, n4), w_end = min(w_begin + seg4, n4);
    const int w_iters = (w_end - w_begin + 31) >> 5;

    // ---- 1. bracket [lo_key, hi_key] of the k-th largest key from a sample ----------------------------
    // Two histogram levels: 512 bins over the sample's key range, then 512 bins over the few bins the two
    // ranks fell into - scores of a row often sit in a narrow band far below the row's maximum, and the first
    // level alone would cut that band into a dozen bins.
    uint32_t lo_key = 0u, hi_key = 0xFFFFFFFFu;
    const bool sampled = n > kListRow;
    if (sampled) {
      constexpr int kF4 = 1024 / kTopkThreads;           // 16-byte pieces per thread that make 4096 sampled scores
      constexpr int kMaxF4 = kTopkWarps == 4 ? kF4 : 2 * kF4;
      const int f4 = n > 65536 ? kMaxF4 : kF4;           // 8192 for long rows (four warps are not given those)
      const int n_samp = f4 * kTopkThreads * 4;
      uint32_t sk[4 * kMaxF4], smin = 0xFFFFFFFFu, smax = 0u;
#pragma unroll
      for (int it = 0; it < kMaxF4; ++it) {
        if (it < f4) {
          const int pos = (int)(((int64_t)(it * kTopkThreads + tid) * n4) >> (f4 == kF4 ? 10 : 11));  // < n4 - 1
          const float4 x = row4[pos];
          sk[it * 4 + 0] = float_key(x.x); sk[it * 4 + 1] = float_key(x.y);
          sk[it * 4 + 2] = float_key(x.z); sk[it * 4 + 3] = float_key(x.w);
        } else {
          sk[it * 4 + 0] = sk[it * 4 + 1] = sk[it * 4 + 2] = sk[it * 4 + 3] = sk[0];
        }
      }
#pragma unroll
      for (int i = 0; i < 4 * kMaxF4; ++i) { smin = min(smin, sk[i]); smax = max(smax, sk[i]); }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        smin = min(smin, __shfl_xor_sync(0xFFFFFFFFu, smin, off));
        smax = max(smax, __shfl_xor_sync(0xFFFFFFFFu, smax, off));
      }
      if (lane == 0) { sh.red[warp] = smin; sh.red2[warp] = smax; }
      for (int i = tid; i < kTopkBins; i += kTopkThreads) sh.hist[i] = 0;
      __syncthreads();
      const uint32_t bottom = warps_min(sh.red), top = warps_max(sh.red2);
      const float ks = (float)k * (float)n_samp / (float)n;                          // sample rank of the threshold
      const float margin = 5.f * sqrtf(ks) + 16.f;
      int r_hi = (int)(ks - margin), r_lo = (int)(ks + margin) + 1;                  // ranks from the top, 1-based
      // level 1
      uint32_t z_lo = bottom, z_hi = top, above = 0;     // zoom window and the samples above it
      {
        const uint32_t range = top - bottom;
        const int shift = (range >> kDigit) ? (32 - __clz(range) - kDigit) : 0;      // (range >> shift) < kTopkBins
#pragma unroll
        for (int i = 0; i < 4 * kF4; ++i) atomicAdd(&sh.hist[(sk[i] - bottom) >> shift], 1u);
        if (f4 != kF4) {
#pragma unroll
          for (int i = 4 * kF4; i < 4 * kMaxF4; ++i) atomicAdd(&sh.hist[(sk[i] - bottom) >> shift], 1u);
        }
        __syncthreads();
        uint32_t b, rest;
        if (r_hi >= 1) {
          find_bin(sh, (uint32_t)r_hi, b, rest);
          above = (uint32_t)r_hi - rest;                                             // samples in the bins above b
          const uint64_t edge = (uint64_t)bottom + ((uint64_t)(b + 1) << shift);      // first key above bin b
          if (edge - 1 < (uint64_t)top) z_hi = (uint32_t)(edge - 1);
        }
        if (r_lo <= n_samp) {
          find_bin(sh, (uint32_t)r_lo, b, rest);
          z_lo = bottom + (b << shift);
        }
      }
      // level 2: the samples inside [z_lo, z_hi]
      {
        const uint32_t range = z_hi - z_lo;
        const int shift = (range >> kDigit) ? (32 - __clz(range) - kDigit) : 0;
        for (int i = tid; i < kTopkBins; i += kTopkThreads) sh.hist[i] = 0;
        __syncthreads();
        uint32_t inside = 0;
#pragma unroll
        for (int i = 0; i < 4 * kF4; ++i) {
          if (sk[i] - z_lo <= range) {                     // z_lo <= key <= z_hi
            atomicAdd(&sh.hist[(sk[i] - z_lo) >> shift], 1u);
            ++inside;
          }
        }
        if (f4 != kF4) {
#pragma unroll
          for (int i = 4 * kF4; i < 4 * kMaxF4; ++i) {
            if (sk[i] - z_lo <= range) {
              atomicAdd(&sh.hist[(sk[i] - z_lo) >> shift], 1u);
              ++inside;
            }
          }
        }
        const uint32_t n_inside = block_sum(sh, inside);  // (its barriers also publish the histogram)
        r_hi -= (int)above;
        r_lo -= (int)above;
        uint32_t b, rest;
        if (r_hi >= 1 && (uint32_t)r_hi <= n_inside) {    // keys above the bin of rank r_hi: (very likely) all selected
          find_bin(sh, (uint32_t)r_hi, b, rest);
          const uint64_t edge = (uint64_t)z_lo + ((uint64_t)(b + 1) << shift);
          hi_key = edge - 1 < (uint64_t)z_hi ? (uint32_t)(edge - 1) : z_hi;
        } else if (r_hi >= 1) {
          hi_key = z_hi;
        }
        if (r_lo >= 1 && (uint32_t)r_lo <= n_inside) {    // keys below the bin of rank r_lo: (very likely) none selected
          find_bin(sh, (uint32_t)r_lo, b, rest);
          lo_key = z_lo + (b << shift);
        } else if (r_lo > (int)n_inside && r_lo + (int)above <= n_samp) {
          lo_key = z_lo;
        }
      }
      if (hi_key < lo_key) { lo_key = 0u; hi_key = 0xFFFFFFFFu; }
    }

    // ---- 2. count the keys above hi_key, collect those in [lo_key, hi_key] --------------------------------
    // Every warp walks its own piece of the row and appends to a list of its own, so that nothing is shared
    // (one counter for the whole CTA would serialise a thousand atomics per row), and so that the list later
    // tells the warp how many of its scores lie above / at the threshold.
    lo_key = max(lo_key, 1u);
    uint32_t cnt_gt = 0, my_cand = 0;                     // my_cand: entries in this warp's list (warp-uniform)
    uint32_t* const my_list = sh.cand + warp * kWarpList;
    {
      for (int it0 = 0; it0 < w_iters; it0 += kTopkUnroll) {
        float4 xs[kTopkUnroll];                           // several loads in flight per lane
#pragma unroll
        for (int j = 0; j < kTopkUnroll; ++j) {
          const int i4 = w_begin + (it0 + j) * 32 + lane;
          xs[j] = i4 < w_end ? row4[i4] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int j = 0; j < kTopkUnroll; ++j) {
          if (it0 + j >= w_iters) break;                  // (the same for the whole warp)
          const int i4 = w_begin + (it0 + j) * 32 + lane;
          uint32_t u[4];
          piece_keys(xs[j], i4 < w_end ? i4 : n4, n4, n, u);
          bool cand[4];
          uint32_t c = 0;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const bool gt = u[e] > hi_key;
            cand[e] = !gt && u[e] >= lo_key;
            cnt_gt += gt;
            c += cand[e];
          }
          if (__any_sync(0xFFFFFFFFu, c != 0)) {
            uint32_t incl = c;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
              const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, off);
              if (lane >= off) incl += v;
            }
            uint32_t pos = my_cand + incl - c;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if (cand[e]) {
                if (pos < (uint32_t)kWarpList) my_list[pos] = u[e];
                ++pos;
              }
            }
            my_cand += __shfl_sync(0xFFFFFFFFu, incl, 31);
          }
        }
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) cnt_gt += __shfl_xor_sync(0xFFFFFFFFu, cnt_gt, off);
    const uint32_t my_gt_hi = cnt_gt;                     // scores of this warp's piece above hi_key
    if (lane != 0) cnt_gt = 0;
    if (lane == 0) sh.list_len[warp] = my_cand;
    uint32_t n_gt = block_sum(sh, cnt_gt);                // (its barriers also publish the lists and their lengths)
    uint32_t n_cand = warps_sum(sh.list_len);
    bool fits = warps_max(sh.list_len) <= (uint32_t)kWarpList;
    if constexpr (C > 1) {
      cg::cluster_group cluster = cg::this_cluster();
      const uint32_t longest = warps_max(sh.list_len);
      if (tid == 0) { sh.cta_gt = n_gt; sh.cta_cand = n_cand; sh.cta_max_list = longest; }
      cluster.sync();
      n_gt = n_cand = 0;
#pragma unroll
      for (int r = 0; r < C; ++r) {
        const TopkShared* peer = cluster.map_shared_rank(&sh, r);
        n_gt += peer->cta_gt;
        n_cand += peer->cta_cand;
        fits = fits && peer->cta_max_list <= (uint32_t)kWarpList;
      }
      fits = fits && n_cand <= (uint32_t)kMergedCap;
      if (fits) {                                         // (the same for the whole cluster)
        if (warp == 0) {                                  // C / 2 lists per lane
          constexpr int kPer = C * kTopkWarps / 32;
          uint32_t len[kPer], sum = 0;
#pragma unroll
          for (int i = 0; i < kPer; ++i) {
            const int l = lane * kPer + i;
            len[i] = cluster.map_shared_rank(&sh, l / kTopkWarps)->list_len[l % kTopkWarps];
            sum += len[i];
          }
          uint32_t incl = sum;
#pragma unroll
          for (int off = 1; off < 32; off <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, off);
            if (lane >= off) incl += v;
          }
          uint32_t at = incl - sum;
#pragma unroll
          for (int i = 0; i < kPer; ++i) { sh.list_at[lane * kPer + i] = at; at += len[i]; }
        }
        __syncthreads();
        for (int l = warp; l < C * kTopkWarps; l += kTopkWarps) {
          const uint32_t begin = sh.list_at[l], end = l + 1 < C * kTopkWarps ? sh.list_at[l + 1] : n_cand;
          const uint32_t* src = cluster.map_shared_rank(&sh, l / kTopkWarps)->cand + (l % kTopkWarps) * kWarpList;
          for (uint32_t i = lane; i < end - begin; i += 32) merged[begin + i] = src[i];
        }
        __syncthreads();
      }
    }
    // the candidates: every warp walks its own list, or the CTA the gathered one
    const uint32_t* const cand_list = C > 1 ? merged : my_list;
    const uint32_t cand_n = C > 1 ? n_cand : my_cand, cand_first = C > 1 ? tid : lane, cand_step = C > 1 ? kTopkThreads : 32;

    if (!sampled) {
      // the whole row is the list: its own key range instead of all 32 bits, so that the first digit spreads
      uint32_t cmin = 0xFFFFFFFFu, cmax = 0u;
      if (fits)
        for (uint32_t i = cand_first; i < cand_n; i += cand_step) { cmin = min(cmin, cand_list[i]); cmax = max(cmax, cand_list[i]); }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        cmin = min(cmin, __shfl_xor_sync(0xFFFFFFFFu, cmin, off));
        cmax = max(cmax, __shfl_xor_sync(0xFFFFFFFFu, cmax, off));
      }
      if (lane == 0) { sh.red[warp] = cmin; sh.red2[warp] = cmax; }
      __syncthreads();
      cmin = warps_min(sh.red);
      cmax = warps_max(sh.red2);
      __syncthreads();
      lo_key = cmin;
      hi_key = cmax;
    }
    uint32_t tau = 0, need_eq = 0;
    if (fits && n_gt < (uint32_t)k && (uint32_t)k <= n_gt + n_cand) {
      // ---- the k-th largest key is the (k - n_gt)-th largest of the list --------------------------------
      const uint32_t range = hi_key - lo_key;
      const int nb = range ? 32 - __clz(range) : 0;
      uint32_t prefix = 0, mask = 0, remaining = (uint32_t)k - n_gt;
#pragma unroll 1
      for (int hb = nb; hb > 0; hb -= kDigit) {
        const int shift = max(hb - kDigit, 0);
        const uint32_t dmask = (1u << (hb - shift)) - 1u;
        for (int i = tid; i < kTopkBins; i += kTopkThreads) sh.hist[i] = 0;
        __syncthreads();
        for (uint32_t i = cand_first; i < cand_n; i += cand_step) {
          const uint32_t v = cand_list[i] - lo_key;
          if ((v & mask) == prefix) atomicAdd(&sh.hist[(v >> shift) & dmask], 1u);
        }
        __syncthreads();
        uint32_t d;
        find_bin(sh, remaining, d, remaining);
        prefix |= d << shift;
        mask |= dmask << shift;
      }
      tau = lo_key + prefix;
      need_eq = remaining;
      // this warp's scores above / at the threshold: those above hi_key, and what its own list says
      uint32_t g = 0, q = 0;
      for (uint32_t i = lane; i < my_cand; i += 32) {
        const uint32_t v = my_list[i];
        g += v > tau;
        q += v == tau;
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        g += __shfl_xor_sync(0xFFFFFFFFu, g, off);
        q += __shfl_xor_sync(0xFFFFFFFFu, q, off);
      }
      if (lane == 0) { sh.warp_gt[warp] = my_gt_hi + g; sh.warp_eq[warp] = q; }
    } else {
      // ---- 3. the sample misjudged the row: four histogram passes over the row itself -------------------
      const int iters = (n4 + kTopkThreads - 1) / kTopkThreads;
      uint32_t prefix = 0, mask = 0, remaining = (uint32_t)k;
#pragma unroll 1
      for (int hb = 32; hb > 0; hb -= kDigit) {
        const int shift = max(hb - kDigit, 0);
        const uint32_t dmask = (1u << (hb - shift)) - 1u;
        for (int i = tid; i < kTopkBins; i += kTopkThreads) sh.hist[i] = 0;
        __syncthreads();
        for (int it = 0; it < iters; ++it) {
          const int i4 = it * kTopkThreads + tid;
          const float4 x = i4 < n4 ? row4[i4] : make_float4(0.f, 0.f, 0.f, 0.f);
          uint32_t u[4];
          piece_keys(x, i4 < n4 ? i4 : n4, n4, n, u);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const bool valid = u[e] != 0u && ((u[e] & mask) == prefix);
            const uint32_t digit = (u[e] >> shift) & dmask;
            // equal digits are common here (that is why the sample failed): aggregate within the warp
            const uint32_t peers = __match_any_sync(0xFFFFFFFFu, valid ? digit : 0xFFFFu);
            if (valid && (__ffs(peers) - 1) == lane) atomicAdd(&sh.hist[digit], (uint32_t)__popc(peers));
          }
        }
        __syncthreads();
        uint32_t d;
        find_bin(sh, remaining, d, remaining);
        prefix |= d << shift;
        mask |= dmask << shift;
      }
      tau = prefix;
      need_eq = remaining;
      // per warp: scores above / equal to the threshold in its piece (one more pass over the row)
      {
        uint32_t g = 0, q = 0;
        for (int it0 = 0; it0 < w_iters; it0 += kTopkUnroll) {
          float4 xs[kTopkUnroll];
  #pragma unroll
          for (int j = 0; j < kTopkUnroll; ++j) {
            const int i4 = w_begin + (it0 + j) * 32 + lane;
            xs[j] = i4 < w_end ? row4[i4] : make_float4(0.f, 0.f, 0.f, 0.f);
          }
  #pragma unroll
          for (int j = 0; j < kTopkUnroll; ++j) {
            const int i4 = w_begin + (it0 + j) * 32 + lane;
            const bool in = i4 < w_end;
            const uint32_t u[4] = {float_key(xs[j].x), float_key(xs[j].y), float_key(xs[j].z), float_key(xs[j].w)};
  #pragma unroll
            for (int e = 0; e < 4; ++e) {
              const bool ok = in && (i4 * 4 + e < n);
              g += ok && u[e] > tau;
              q += ok && u[e] == tau;
            }
          }
        }
  #pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          g += __shfl_xor_sync(0xFFFFFFFFu, g, off);
          q += __shfl_xor_sync(0xFFFFFFFFu, q, off);
        }
        if (lane == 0) { sh.warp_gt[warp] = g; sh.warp_eq[warp] = q; }
      }
    }
    // tau = key of the k-th largest score; `need_eq` keys equal to it are wanted, the lowest positions first

    __syncthreads();
    uint32_t gt_before, eq_before;                        // in the pieces of the warps before this one
    {
      const int w = lane & (kTopkWarps - 1);
      uint32_t g = w < warp ? sh.warp_gt[w] : 0u, q = w < warp ? sh.warp_eq[w] : 0u;
#pragma unroll
      for (int off = kTopkWarps / 2; off > 0; off >>= 1) {
        g += __shfl_xor_sync(0xFFFFFFFFu, g, off);
        q += __shfl_xor_sync(0xFFFFFFFFu, q, off);
      }
      gt_before = g;
      eq_before = q;
    }
    if constexpr (C > 1) {                                // ... and in the pieces of the CTAs before this one
      cg::cluster_group cluster = cg::this_cluster();
      const uint32_t above = warps_sum(sh.warp_gt), equal = warps_sum(sh.warp_eq);
      if (tid == 0) { sh.cta_above = above; sh.cta_equal = equal; }
      cluster.sync();
      for (int r = 0; r < rank; ++r) {
        const TopkShared* peer = cluster.map_shared_rank(&sh, r);
        gt_before += peer->cta_above;
        eq_before += peer->cta_equal;
      }
    }
    if (row + gridDim.x / C >= rows) pdl_trigger();       // the CTA's last row, and its last pass
    // ---- 4. write the selected positions of this warp's piece, in index order -----------------------------
    for (int it0 = 0; it0 < w_iters; it0 += kTopkUnroll) {
      float4 xs[kTopkUnroll];
#pragma unroll
      for (int j = 0; j < kTopkUnroll; ++j) {
        const int i4 = w_begin + (it0 + j) * 32 + lane;
        xs[j] = i4 < w_end ? row4[i4] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int j = 0; j < kTopkUnroll; ++j) {
        if (it0 + j >= w_iters) break;                    // (the same for the whole warp)
        const int i4 = w_begin + (it0 + j) * 32 + lane;
        uint32_t u[4];
        piece_keys(xs[j], i4 < w_end ? i4 : n4, n4, n, u);
        uint32_t gt[4], packed = 0;
        bool any_eq = false;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          gt[e] = u[e] > tau;
          packed += gt[e];
          any_eq |= u[e] == tau;
        }
        if (!__any_sync(0xFFFFFFFFu, any_eq)) {
          // no score at the threshold among these 128: positions follow from the counts of the lanes before
          uint32_t incl = packed;
#pragma unroll
          for (int off = 1; off < 32; off <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, off);
            if (lane >= off) incl += v;
          }
          uint32_t at = gt_before + min(eq_before, need_eq) + incl - packed;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (gt[e]) out[at++] = i4 * 4 + e;
          }
          gt_before += __shfl_sync(0xFFFFFFFFu, incl, 31);
        } else {
          uint32_t eq[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            eq[e] = u[e] == tau;
            packed += eq[e] << 16;
          }
          uint32_t incl = packed;                          // (eq << 16 | gt) of the lanes up to this one
#pragma unroll
          for (int off = 1; off < 32; off <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, off);
            if (lane >= off) incl += v;
          }
          const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
          const uint32_t excl = incl - packed;
          uint32_t g0 = gt_before + (excl & 0xFFFFu), q0 = eq_before + (excl >> 16);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const bool sel = gt[e] || (eq[e] && q0 < need_eq);
            if (sel) out[g0 + min(q0, need_eq)] = i4 * 4 + e;
            g0 += gt[e];
            q0 += eq[e];
          }
          gt_before += total & 0xFFFFu;
          eq_before += total >> 16;
        }
      }
    }
    if constexpr (C > 1) cg::this_cluster().sync();       // ... and read by the other CTAs until here
    else __syncthreads();                                 // the shared arrays are reused by the next row
  }
}

__global__ void prefill_budgets_kernel(int32_t* n_valid, int32_t* k_row, int num_tiles, int total,
                                       int k_max, float pct, int rolling) {
  pdl_begin();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  int t = i % num_tiles;
  int start = t * kTile;
  n_valid[i] = start;
  int k = k_max;
  if (rolling) {
    // strategies/KascadeStrategy.py:137: (pct * tile_start) // 100, at least 128
    int r = (int)floor((double)pct * (double)start / 100.0);
    k = min(k_max, max(128, r));
  }
  k_row[i] = k;
}

// per-sequence budgets of a ragged batch: the reference's formulas for a prompt of seq_len[b] tokens
// (strategies/KascadeStrategy.py:127-139); tiles beyond a sequence's end get no candidates
__global__ void prefill_budgets_ragged_kernel(int32_t* n_valid, int32_t* k_row, const int32_t* seq_len, int groups,
                                              int num_tiles, int total, int k_cap, float pct, int rolling) {
  pdl_begin();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int t = i % num_tiles, b = i / (num_tiles * groups);
  const int L = max(seq_len[b], 0), start = t * kTile;
  int kk = min(max(128, (int)((double)pct / 100.0 * (double)L)), L) - kTile;
  kk = max(kk, 0);
  int k = kk;
  if (rolling && L > 128) {
    int r = (int)floor((double)pct * (double)start / 100.0);
    k = min(kk, max(128, r));
  }
  const bool live = start < L;
  n_valid[i] = live ? start : 0;
  k_row[i] = live ? min(k, k_cap) : 0;
}

}  // namespace kb200

extern "C" int kb200_prefill_budgets_ragged(int32_t* n_valid, int32_t* k_row, const int32_t* seq_len, int batch,
                                            int num_kv_heads, int num_tiles, int k_cap, float pct, int rolling,
                                            void* stream) {
  using namespace kb200;
  KB_ENTRY(n_valid, "prefill_budgets_ragged: n_valid");
  KB_REQUIRE(n_valid && k_row && seq_len, "prefill_budgets_ragged: null pointer");
  int total = batch * num_kv_heads * num_tiles;
  if (total <= 0) return 0;
  KB_LAUNCH("prefill_budgets_ragged_kernel",
            launch_pdl(prefill_budgets_ragged_kernel, dim3(ceil_div(total, 256)), 256, 0, (cudaStream_t)stream, 1, n_valid,
                       k_row, seq_len, num_kv_heads, num_tiles, total, k_cap, pct, rolling));
  return 0;
}

namespace kb200 {
// CTAs per row: doubled while all rows together leave an SM for each CTA and a CTA keeps at least 4096 scores; below
// that, and for rows under 16384, its fixed phases (the sample, the lists) cost more than a shorter piece saves.
// Measured, us with one CTA / a cluster: 8 rows of 16384 / 32768 / 131072 scores 17.2 / 25.4 / 69.9 -> 15.2 / 18.5 / 27.1,
// 32 x 65536 41.4 -> 23.7 (29.2 with two CTAs on an SM), 64 x 32768 25.7 -> 21.1; 128 x 16384 17.8 -> 20.3 with two, 8 x 8192
// 13.3 -> 13.7: not taken.  A cluster needs places for all its CTAs in one group of SMs, so where the CTAs of clusters of four
// or eight would fill the chip some share an SM: they leave an eighth of it free, unless four have long rows to share
// (37 rows of 16384 / 32768 / 65536 / 131072 in clusters of two / four 16.0 / 18.6, 21.1 / 22.7, 31.4 / 30.6, 48.2 / 44.0;
// 18 of 65536 in four / eight 24.2 / 28.5).
static int topk_cluster(int64_t rows, int n_cols) {
  int c = 1;
  if (n_cols < 16384) return c;
  const int sms = sm_count();
  while (c < 8 && n_cols / (2 * c) >= 4096 &&
         rows * (2 * c) <= (c == 1 || (c == 2 && n_cols >= 65536) ? sms : sms * 7 / 8))
    c *= 2;
  return c;
}

// Warps of a CTA that has a row to itself.  A row's serial phases (some thirty CTA barriers) are what bounds this kernel
// when there are many rows, so smaller CTAs, of which more are resident (a thousand threads per SM at 64 registers),
// hide more of them.  Few rows want many warps each, and rows that do not fit the lists of four warps (about 65536
// scores) at least eight.  Measured, us with 16 / 8 / 4 warps: 512 prompt rows of up to 2048 scores 18.2 / 12.6 / 12.5,
// 3008 x 3001 88 / 50 / 40, 2048 x 8192 92 / 63 / 58, 8192 x 32768 626 / 490 / 505, 24576 x 98304 3776 / 3428 / 7405;
// decode rows 512 x 32768 68 / 61 / 77, 256 x 16000 23 / 25 / 37, 192 x 65536 58 / 73 / 435.
// The longer the rows, the more of the time is passes over them and the more the last CTAs to end weigh, above all
// where the rows differ in length: beyond 32768 scores eight warps need rows for several rounds.  us with 16 / 8: 512
// rows of up to 65536 / 131072 scores 96 / 101, 161 / 194; 600 equal ones 154 / 171, 278 / 317; 1024 212 / 208, 389 / 392, of up
// to that many 156 / 159, 261 / 289; 2048 equal ones 406 / 392, 738 / 745.  A second round of a few rows costs as much:
// 600 x 24000 / 32768 75.5 / 73.9, 91.2 / 95.5, 800 x 32768 107.4 / 104.4.
static int topk_warps(int64_t rows, int n_cols) {
  const int64_t sms = sm_count();
  if (rows < 3 * sms) return 16;
  if (n_cols <= 8192) return 4;
  if (n_cols > 32768 && rows < (n_cols <= 65536 ? 8 : 14) * sms) return 16;
  if (n_cols > 24576 && rows > 4 * sms && rows <= 5 * sms) return 16;
  return 8;
}

int init_topk() {
  KB_CUDA(cudaFuncSetAttribute(topk_select_kernel<2, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTopkMergedBytes));
  KB_CUDA(cudaFuncSetAttribute(topk_select_kernel<4, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTopkMergedBytes));
  KB_CUDA(cudaFuncSetAttribute(topk_select_kernel<8, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTopkMergedBytes));
  return 0;
}

static int topk_launch(const float* scores, int64_t row_stride, int n_cols, const int32_t* n_valid,
                       const int32_t* k_row, int k_max, int32_t* out_idx, int64_t idx_stride, int32_t* out_count,
                       int64_t rows, const DecodeBudget& budget, void* stream) {
  KB_ENTRY(scores, "topk_select: scores");
  KB_REQUIRE(scores && out_idx, "topk_select: null pointer");
  KB_REQUIRE(rows >= 0 && n_cols >= 0 && k_max >= 0, "topk_select: negative size");
  KB_REQUIRE(n_cols <= row_stride, "topk_select: n_cols (%d) exceeds row_stride (%lld)", n_cols,
             (long long)row_stride);
  KB_REQUIRE(row_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(scores) & 15) == 0,
             "topk_select: rows must be 16-byte aligned (row_stride %% 4 == 0)");
  KB_REQUIRE(idx_stride >= (int64_t)k_max, "topk_select: idx_stride (%lld) smaller than k_max (%d)",
             (long long)idx_stride, k_max);
  if (rows == 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  const int c = topk_cluster(rows, n_cols);
  auto* kernel = topk_select_kernel<1, 16>;
  int warps = 16;
  if (c == 1) {
    warps = topk_warps(rows, n_cols);
    kernel = warps == 4 ? topk_select_kernel<1, 4> : warps == 8 ? topk_select_kernel<1, 8> : topk_select_kernel<1, 16>;
  } else {
    kernel = c == 8 ? topk_select_kernel<8, 16> : c == 4 ? topk_select_kernel<4, 16> : topk_select_kernel<2, 16>;
  }
  const int64_t most = (int64_t)sm_count() * 1024 / warps;
  const dim3 grid((unsigned)(c > 1 || rows < most ? rows * c : most));
  KB_LAUNCH("topk_select_kernel",
            launch_pdl(kernel, grid, warps * 32, c > 1 ? kTopkMergedBytes : 0, st, c, scores, row_stride, n_cols, n_valid, k_row,
                       k_max, out_idx, idx_stride, out_count, rows, budget));
  return 0;
}
}  // namespace kb200

extern "C" int kb200_topk_select(const float* scores, int64_t row_stride, int n_cols,
                                 const int32_t* n_valid, const int32_t* k_row, int k_max,
                                 int32_t* out_idx, int64_t idx_stride, int32_t* out_count,
                                 int64_t rows, void* stream) {
  return kb200::topk_launch(scores, row_stride, n_cols, n_valid, k_row, k_max, out_idx, idx_stride, out_count, rows,
                            kb200::DecodeBudget{}, stream);
}

extern "C" int kb200_topk_select_decode(const float* scores, int64_t row_stride, int n_cols, const int32_t* seq_lens,
                                        int num_kv_heads, double share, int tile, int k_max, int32_t* out_idx,
                                        int64_t idx_stride, int32_t* out_count, int batch, void* stream) {
  using namespace kb200;
  KB_REQUIRE(seq_lens, "topk_select_decode: null pointer");
  KB_REQUIRE(batch >= 0 && num_kv_heads > 0 && tile >= 0 && share >= 0.0 && share <= 1.0,
             "topk_select_decode: batch %d, %d KV heads, tile %d, share %g", batch, num_kv_heads, tile, share);
  return topk_launch(scores, row_stride, n_cols, nullptr, nullptr, k_max, out_idx, idx_stride, out_count,
                     (int64_t)batch * num_kv_heads, DecodeBudget{seq_lens, num_kv_heads, share, tile}, stream);
}

extern "C" int kb200_prefill_budgets(int32_t* n_valid, int32_t* k_row, int batch, int num_kv_heads,
                                     int num_tiles, int k_max, float pct, int rolling, void* stream) {
  using namespace kb200;
  KB_ENTRY(n_valid, "prefill_budgets: n_valid");
  KB_REQUIRE(n_valid && k_row, "prefill_budgets: null pointer");
  int total = batch * num_kv_heads * num_tiles;
  if (total <= 0) return 0;
  KB_LAUNCH("prefill_budgets_kernel",
            launch_pdl(prefill_budgets_kernel, dim3(ceil_div(total, 256)), 256, 0, (cudaStream_t)stream, 1, n_valid, k_row,
                       num_tiles, total, k_max, pct, rolling));
  return 0;
}
