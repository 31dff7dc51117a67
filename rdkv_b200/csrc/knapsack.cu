// Batched Lagrangian bit allocator: the whole multiplier search inside one kernel, a cluster of CTAs per
// long row (sorted into buckets in shared memory), a warp per short one.
//
// Control flow and rounding follow the reference solver
// (knapsack_solver.py:121-248): cost = score*eps[n] + lambda*bits[n] with each
// product and the sum rounded to fp32 separately, first-index argmin, mean =
// exact integer sum / N in fp32, and the batch-wide exits of the lambda_hi
// doubling loop.
#include <cooperative_groups.h>

#include "rdkv_common.cuh"

namespace rdkv {

constexpr int KNAP_THREADS = 1024;
constexpr int KNAP_MAX_OPT = 8;
constexpr int KNAP_SMEM_ROW_BYTES = 200 * 1024;

struct KnapOpts {
  float bits[KNAP_MAX_OPT];
  float eps[KNAP_MAX_OPT];
  int ibits[KNAP_MAX_OPT];
  int n;
  float budget;                                             // of every row, where no budgets are given
};

__device__ __forceinline__ float row_budget(const float* budget, int b, const KnapOpts& o) { return budget != nullptr ? budget[b] : o.budget; }

__device__ __forceinline__ int choose(float s, const float* se_unused, const KnapOpts& o, const float* lb) {
  int best = 0;
  float bc = __fadd_rn(__fmul_rn(s, o.eps[0]), lb[0]);
#pragma unroll
  for (int n = 1; n < KNAP_MAX_OPT; ++n) {
    if (n < o.n) {
      const float c = __fadd_rn(__fmul_rn(s, o.eps[n]), lb[n]);
      if (c < bc) { bc = c; best = n; }
    }
  }
  return best;
}

// Block-wide exact sum of the chosen bit costs for multiplier lam.
__device__ unsigned long long sweep_sum(const float* row, int len, float lam, const KnapOpts& o,
                                        unsigned long long* s_red) {
  float lb[KNAP_MAX_OPT];
#pragma unroll
  for (int n = 0; n < KNAP_MAX_OPT; ++n) lb[n] = n < o.n ? __fmul_rn(lam, o.bits[n]) : 0.f;
  unsigned int local = 0;
  for (int i = threadIdx.x; i < len; i += KNAP_THREADS) local += (unsigned)o.ibits[choose(row[i], nullptr, o, lb)];
  unsigned long long v = local;
#pragma unroll
  for (int ofs = 16; ofs > 0; ofs >>= 1) v += __shfl_xor_sync(0xffffffffu, v, ofs);
  __syncthreads();                       // s_red may still be read from the previous sweep
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
  __syncthreads();
  unsigned long long tot = 0;
  for (int w = 0; w < KNAP_THREADS / 32; ++w) tot += s_red[w];
  return tot;
}

__device__ __forceinline__ float mean_of(unsigned long long sum, int len) {
  return __fdiv_rn((float)sum, (float)len);
}

__device__ const float* stage_row(const float* grow, int len, float* smem_row, bool use_smem) {
  if (!use_smem) return grow;
  for (int i = threadIdx.x; i < len; i += KNAP_THREADS) smem_row[i] = grow[i];
  __syncthreads();
  return smem_row;
}

// ── rows sorted into buckets: a sweep looks at the elements near the thresholds only ─────────────
// The search asks, for up to a hundred multipliers, what the row's choices cost.  Evaluating every element
// each time is bound by instruction issue (about 20 instructions an element and sweep: 2.8 us of an SM for
// 32768 elements).  But over a short interval of scores the choice is nearly always the same for every
// element.  So a row is sorted once by the leading bits of its scores (sign, exponent, five mantissa
// bits: 32 buckets an octave, the lowest bucket takes everything below 2^-32 of the maximum), and a sweep
//   * evaluates every bucket at its two ends.  If one option is cheaper than every other at both ends by
//     more than 2^-20 of the two costs (plus 1e-37 for products that underflow), it is the choice of every
//     element between: the exact costs are linear in the score, so their difference minus 2^-20 of their
//     sum is positive all along the bucket, and the computed costs are off by less than 2^-22 of their
//     sum.  The bucket then counts (elements) x (bits);
//   * evaluates the elements of the other buckets (around the thresholds, one or two buckets each) one by
//     one, as the reference does.
// The sums are integers, so they equal a full sweep's bit for bit.  Scores that are negative, infinite
// or NaN share the lowest bucket, which is then always evaluated element by element.
// 256 rows x 32768: 94 us (every element in every sweep, two kernels: 371).
// (Tried and slower, times of a whole call with its channel rows while it took 205 us: thresholds worked out by
// one warp and runs of buckets between them tested, 230; a first test per octave, 231; three multipliers a
// sweep, 480.  Later, kernel alone: buckets whose choice is the same at both ends of the multiplier's interval
// left out of later sweeps, 96 instead of 91; the scores kept in registers for the sort, 88 here but 43
// instead of 40 for 8 rows.)
// A row is spread over a cluster of CTAs (each sorts its own part; partial sums meet in every CTA's shared
// memory), so that a few rows still fill the chip and a row of 262144 fits.
// What a sum of chosen bits means for the search: 0 = within `tol` of the budget, 1 = above it, -1 = not above.
// The reference divides twice (the mean, the relative distance).  Where the sum is further than tol + 1e-5 from
// the budget's share, both answers follow from one comparison: the three roundings together are below 4e-7.
__device__ __forceinline__ int budget_side(unsigned sum, int len, float bud, float tol) {
  if (bud > 1e-6f) {
    const float t = __fmul_rn(bud, (float)len), d = __fsub_rn((float)sum, t);
    if (fabsf(d) > (fmaxf(tol, 0.f) + 1e-5f) * t) return d > 0.f ? 1 : -1;
  }
  const float avg = mean_of(sum, len);
  const float rel = __fdiv_rn(fabsf(__fsub_rn(avg, bud)), fmaxf(bud, 1e-8f));
  return rel < tol ? 0 : avg > bud ? 1 : -1;
}
__device__ __forceinline__ bool above(unsigned sum, int len, float bud) {   // mean > budget
  return budget_side(sum, len, bud, 0.f) > 0;
}

// choose, giving the option's bits (no indexed look-up: the options stay launch constants)
__device__ __forceinline__ unsigned choose_bits(float s, const KnapOpts& o, const float* lb) {
  unsigned bits = (unsigned)o.ibits[0];
  float bc = __fadd_rn(__fmul_rn(s, o.eps[0]), lb[0]);
#pragma unroll
  for (int n = 1; n < KNAP_MAX_OPT; ++n) {
    if (n < o.n) {
      const float c = __fadd_rn(__fmul_rn(s, o.eps[n]), lb[n]);
      if (c < bc) { bc = c; bits = (unsigned)o.ibits[n]; }
    }
  }
  return bits;
}

constexpr int KB_BUCKETS = 1024;
constexpr int KB_SHIFT = 18;                                // float bits below the bucket number: 5 mantissa bits stay
constexpr int KB_MAX_CLUSTER = 8;
constexpr int KB_MAX_CHUNK = 32768;                         // elements per CTA
constexpr int KB_SMALL_CHUNK = 16384;                       // up to here with 512 threads, above with 1024
constexpr int KB_PIECE = 64;                                // elements a warp takes at a time
constexpr int KB_BATCH = 4;                                 // loads in flight per thread
// dynamic shared memory: the part's scores in bucket order and the list of pieces to look at
__host__ __device__ constexpr size_t kb_smem_bytes(int chunk) { return (size_t)chunk * 4 + ((size_t)KB_BUCKETS + chunk / KB_PIECE) * 4; }

template <int KB_THREADS>
struct KnapShared {
  int end[KB_BUCKETS];                                      // bucket k = sorted[k ? end[k-1] : 0 .. end[k])
  int wtot[KB_THREADS / 32];
  unsigned sum[2];
  int n_pieces[2];
  int irregular;
  float fmax_slot[KB_MAX_CLUSTER];
  unsigned sum_slot[2][KB_MAX_CLUSTER];
};

// KB_THREADS: 512, or 1024 for parts of more than 16384 scores (one CTA per SM then).
template <int S, int KB_THREADS>
__global__ void __launch_bounds__(KB_THREADS)
knapsack_bucket_kernel(const float* __restrict__ scores, int64_t row_stride, int len, const float* __restrict__ budget,
                       KnapOpts o, int max_iters, float tol, int chunk, float* __restrict__ lam0_out,
                       int* __restrict__ ndbl_out, int64_t* __restrict__ out) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char kb_smem[];
  __shared__ KnapShared<KB_THREADS> sh;
  float* sorted = reinterpret_cast<float*>(kb_smem);                              // [chunk]
  unsigned* pieces = reinterpret_cast<unsigned*>(kb_smem + (size_t)chunk * 4);    // [KB_BUCKETS + chunk / KB_PIECE]: first element | count << 16
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = S > 1 ? (int)cluster.block_rank() : 0;
  const int b = blockIdx.x / S;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* row = scores + (int64_t)b * row_stride + (int64_t)rank * chunk;
  const int n = max(0, min(chunk, len - rank * chunk));

  // the row's maximum (NaN ignored) over all CTAs
  float mx = -INFINITY;
#pragma unroll 8
  for (int i = tid; i < n; i += KB_THREADS) mx = fmaxf(mx, row[i]);
  mx = warp_max(mx);
  if (lane == 0) sh.wtot[warp] = __float_as_int(mx);
  for (int k = tid; k < KB_BUCKETS; k += KB_THREADS) sh.end[k] = 0;
  if (tid == 0) { sh.irregular = 0; sh.sum[0] = sh.sum[1] = 0u; sh.n_pieces[0] = sh.n_pieces[1] = 0; }
  __syncthreads();
  mx = -INFINITY;
#pragma unroll
  for (int w = 0; w < KB_THREADS / 32; ++w) mx = fmaxf(mx, __int_as_float(sh.wtot[w]));
  if (S > 1) {
    cluster.sync();                                         // (every CTA of the cluster runs before anybody writes to it)
    if (tid < S) *cluster.map_shared_rank(&sh.fmax_slot[rank], tid) = mx;
    cluster.sync();
#pragma unroll
    for (int r = 0; r < S; ++r) mx = fmaxf(mx, sh.fmax_slot[r]);
  } else {
    __syncthreads();
  }

  // counting sort by bucket
  const int top = (int)(min(__float_as_uint(fmaxf(mx, 0.f)), 0x7F7FFFFFu) >> KB_SHIFT), base = top - (KB_BUCKETS - 1);
  auto bucket_of = [&](float s, bool& odd) {
    const unsigned u = __float_as_uint(s);
    odd = u >= 0x7F800000u;                                 // negative (or -0), infinite, NaN
    return odd ? 0 : min(max((int)(u >> KB_SHIFT) - base, 0), KB_BUCKETS - 1);
  };
  for (int i0 = tid; i0 < n; i0 += KB_BATCH * KB_THREADS) {
    float s[KB_BATCH];
#pragma unroll
    for (int u = 0; u < KB_BATCH; ++u) s[u] = i0 + u * KB_THREADS < n ? row[i0 + u * KB_THREADS] : 0.f;
#pragma unroll
    for (int u = 0; u < KB_BATCH; ++u) {
      if (i0 + u * KB_THREADS >= n) break;
      bool odd;
      const int k = bucket_of(s[u], odd);
      atomicAdd(&sh.end[k], 1);
      if (odd) sh.irregular = 1;
    }
  }
  __syncthreads();
  {
    constexpr int PER = KB_BUCKETS / KB_THREADS;
    int c[PER], tot = 0;
#pragma unroll
    for (int e = 0; e < PER; ++e) { c[e] = sh.end[tid * PER + e]; tot += c[e]; }
    int incl = tot;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += x;
    }
    if (lane == 31) sh.wtot[warp] = incl;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; ++w) before += sh.wtot[w];
    int start = before + incl - tot;
#pragma unroll
    for (int e = 0; e < PER; ++e) { sh.end[tid * PER + e] = start; start += c[e]; }
  }
  __syncthreads();
  for (int i0 = tid; i0 < n; i0 += KB_BATCH * KB_THREADS) {
    float s[KB_BATCH];
    int at[KB_BATCH];
#pragma unroll
    for (int u = 0; u < KB_BATCH; ++u) s[u] = i0 + u * KB_THREADS < n ? row[i0 + u * KB_THREADS] : 0.f;
#pragma unroll
    for (int u = 0; u < KB_BATCH; ++u) {
      bool odd;
      at[u] = i0 + u * KB_THREADS < n ? atomicAdd(&sh.end[bucket_of(s[u], odd)], 1) : -1;   // (the order inside a bucket does not matter)
    }
#pragma unroll
    for (int u = 0; u < KB_BATCH; ++u)
      if (at[u] >= 0) sorted[at[u]] = s[u];
  }
  __syncthreads();
  const bool irregular = sh.irregular != 0;

  int turn = 0;
  auto sweep = [&](float lam) -> unsigned {                 // the whole row's sum of chosen bits, the same in every thread
    float lb[KNAP_MAX_OPT];
#pragma unroll
    for (int x = 0; x < KNAP_MAX_OPT; ++x) lb[x] = x < o.n ? __fmul_rn(lam, o.bits[x]) : 0.f;
    const int p = turn & 1;
    ++turn;
    unsigned tot = 0;
#pragma unroll
    for (int k = tid; k < KB_BUCKETS; k += KB_THREADS) {
      const int start = k > 0 ? sh.end[k - 1] : 0, cnt = sh.end[k] - start;
      if (cnt == 0) continue;
      const float lo = k == 0 ? 0.f : __uint_as_float((unsigned)max(base + k, 0) << KB_SHIFT);
      const float hi = __uint_as_float((unsigned)max(base + k + 1, 0) << KB_SHIFT);
      // the choice at the upper end, with its costs at both ends
      int best = 0;
      unsigned bits = (unsigned)o.ibits[0];
      float ch = __fadd_rn(__fmul_rn(hi, o.eps[0]), lb[0]), cl = __fadd_rn(__fmul_rn(lo, o.eps[0]), lb[0]);
#pragma unroll
      for (int x = 1; x < KNAP_MAX_OPT; ++x) {
        if (x < o.n) {
          const float c = __fadd_rn(__fmul_rn(hi, o.eps[x]), lb[x]);
          if (c < ch) { ch = c; cl = __fadd_rn(__fmul_rn(lo, o.eps[x]), lb[x]); best = x; bits = (unsigned)o.ibits[x]; }
        }
      }
      bool pure = !(k == 0 && irregular);
#pragma unroll
      for (int x = 0; x < KNAP_MAX_OPT; ++x) {
        if (x < o.n && x != best) {
          const float al = __fadd_rn(__fmul_rn(lo, o.eps[x]), lb[x]), ah = __fadd_rn(__fmul_rn(hi, o.eps[x]), lb[x]);
          pure = pure && (al - cl > fmaf(9.5367431640625e-7f, al + cl, 1e-37f)) && (ah - ch > fmaf(9.5367431640625e-7f, ah + ch, 1e-37f));
        }
      }
      if (pure) {
        tot += (unsigned)cnt * bits;
      } else {
        const int np = (cnt + KB_PIECE - 1) / KB_PIECE, at = atomicAdd(&sh.n_pieces[p], np);
        for (int q = 0; q < np; ++q) pieces[at + q] = (unsigned)(start + q * KB_PIECE) | (unsigned)min(KB_PIECE, cnt - q * KB_PIECE) << 16;
      }
    }
    __syncthreads();
    const int np = sh.n_pieces[p];
    for (int q = warp; q < np; q += KB_THREADS / 32) {
      const unsigned w = pieces[q];
      const int start = (int)(w & 0xFFFFu), cnt = (int)(w >> 16);
      for (int e = lane; e < cnt; e += 32) tot += choose_bits(sorted[start + e], o, lb);
    }
    tot = __reduce_add_sync(0xffffffffu, tot);
    if (lane == 0 && tot != 0u) atomicAdd(&sh.sum[p], tot);
    if (tid == 0) { sh.sum[p ^ 1] = 0u; sh.n_pieces[p ^ 1] = 0; }   // (last read before this sweep's first barrier)
    __syncthreads();
    if (S == 1) return sh.sum[p];
    if (tid < S) *cluster.map_shared_rank(&sh.sum_slot[p][rank], tid) = sh.sum[p];
    cluster.sync();
    unsigned all = 0;
#pragma unroll
    for (int r = 0; r < S; ++r) all += sh.sum_slot[p][r];
    return all;
  };

  const float bud = row_budget(budget, b, o);
  const float lam0 = fmaxf(__fmul_rn(mx, 0.375f), 1e-8f);
  float lam = lam0;
  int k = 0;
  for (; k < 40; ++k) {
    if (!above(sweep(lam), len, bud)) break;
    lam = __fmul_rn(lam, 2.0f);
  }
  if (rank == 0 && tid == 0) { lam0_out[b] = lam0; ndbl_out[b] = k; }
  // (every doubling this row asked for; where the reference's batch-wide loop would have ended earlier,
  //  knapsack_cut_kernel does the row again)
  float lam_lo = 0.f, lam_hi = ldexpf(lam0, k), lam_final = 0.f;
  if (above(sweep(0.f), len, bud)) {
    float lam_mid = 0.f;
    for (int it = 0; it < max_iters; ++it) {
      lam_mid = __fdiv_rn(__fadd_rn(lam_lo, lam_hi), 2.0f);
      const int j = budget_side(sweep(lam_mid), len, bud, tol);
      if (j == 0) break;
      if (j > 0) lam_lo = lam_mid; else lam_hi = lam_mid;
    }
    lam_final = lam_mid;
  }
  float lb[KNAP_MAX_OPT];
#pragma unroll
  for (int x = 0; x < KNAP_MAX_OPT; ++x) lb[x] = x < o.n ? __fmul_rn(lam_final, o.bits[x]) : 0.f;
  int64_t* orow = out + (int64_t)b * len + (int64_t)rank * chunk;
  for (int i = tid; i < n; i += KB_THREADS) orow[i] = (int64_t)choose_bits(row[i], o, lb);
  if (S > 1) cluster.sync();                                // nobody leaves while others may still write to its slots
}

// Short rows (K channels, small blocks): a warp per row, PER scores per lane in registers.  A sweep is PER
// evaluations a lane and one warp-wide addition, without a barrier.
// ALONE: up to 16 rows (the heads of a layer) in one CTA, which replays the batch-wide exit of the doubling
// loop on the seeds it has in shared memory, so that no second launch has to look for rows to do again (one
// layer selected and packed: 286 -> 280 us; four blocks of 64 tokens: 954 -> 920 us).  More rows than one CTA
// has warps would not share its memory, and their second launch is a small part of their call.
constexpr int KW_WARPS = 4;
constexpr int KW_ALONE = 16;
template <int PER, bool ALONE>
__global__ void __launch_bounds__((ALONE ? KW_ALONE : KW_WARPS) * 32)
knapsack_warp_kernel(const float* __restrict__ scores, int64_t row_stride, int n_rows, int len,
                     const float* __restrict__ budget, KnapOpts o, int max_iters, float tol, float* __restrict__ lam0_out,
                     int* __restrict__ ndbl_out, int64_t* __restrict__ out) {
  __shared__ float s_lam0[KW_ALONE];
  __shared__ int s_ndbl[KW_ALONE];
  const int b = ALONE ? threadIdx.x >> 5 : blockIdx.x * KW_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (b >= n_rows) return;                                  // (ALONE: exactly n_rows warps)
  const float* row = scores + (int64_t)b * row_stride;
  float s[PER];
  float mx = -INFINITY;
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    const int i = e * 32 + lane;
    s[e] = i < len ? row[i] : 0.f;
    if (i < len) mx = fmaxf(mx, s[e]);
  }
  mx = warp_max(mx);
  auto sweep = [&](float lam) -> unsigned {
    float lb[KNAP_MAX_OPT];
#pragma unroll
    for (int x = 0; x < KNAP_MAX_OPT; ++x) lb[x] = x < o.n ? __fmul_rn(lam, o.bits[x]) : 0.f;
    unsigned tot = 0;
#pragma unroll
    for (int e = 0; e < PER; ++e) {
      const unsigned c = choose_bits(s[e], o, lb);
      tot += e * 32 + lane < len ? c : 0u;
    }
    return __reduce_add_sync(0xffffffffu, tot);
  };
  const float bud = row_budget(budget, b, o);
  const float lam0 = fmaxf(__fmul_rn(mx, 0.375f), 1e-8f);
  float lam = lam0;
  int k = 0;
#pragma unroll 1
  for (; k < 40; ++k) {
    if (!above(sweep(lam), len, bud)) break;
    lam = __fmul_rn(lam, 2.0f);
  }
  int rounds = 40;
  if (ALONE) {
    if (lane == 0) { s_lam0[b] = lam0; s_ndbl[b] = k; }
    __syncthreads();
    if (k >= 2 && ldexpf(lam0, k - 1) >= 1e12f) {           // (only then can the others have ended this row's doublings)
      rounds = 0;
      for (; rounds < 40; ++rounds) {
        bool need = false, big = true;
        for (int r = 0; r < n_rows; ++r) {
          need = need || s_ndbl[r] > rounds;
          big = big && ldexpf(s_lam0[r], min(rounds + 1, s_ndbl[r])) >= 1e12f;
        }
        if (!need) break;
        if (big) { ++rounds; break; }
      }
    }
  } else if (lane == 0) {
    lam0_out[b] = lam0; ndbl_out[b] = k;
  }
  float lam_lo = 0.f, lam_hi = ldexpf(lam0, min(rounds, k)), lam_final = 0.f;
  if (above(sweep(0.f), len, bud)) {
    float lam_mid = 0.f;
#pragma unroll 1
    for (int it = 0; it < max_iters; ++it) {
      lam_mid = __fdiv_rn(__fadd_rn(lam_lo, lam_hi), 2.0f);
      const int j = budget_side(sweep(lam_mid), len, bud, tol);
      if (j == 0) break;
      if (j > 0) lam_lo = lam_mid; else lam_hi = lam_mid;
    }
    lam_final = lam_mid;
  }
  float lb[KNAP_MAX_OPT];
#pragma unroll
  for (int x = 0; x < KNAP_MAX_OPT; ++x) lb[x] = x < o.n ? __fmul_rn(lam_final, o.bits[x]) : 0.f;
#pragma unroll
  for (int e = 0; e < PER; ++e)
    if (e * 32 + lane < len) out[(int64_t)b * len + e * 32 + lane] = (int64_t)choose_bits(s[e], o, lb);
}

// ── every element in every sweep: rows of more than 262144 scores, and negative distortions ──────────
// Phase 1: lambda_hi seed and the number of doublings this row asks for (<= 40).
__global__ void __launch_bounds__(KNAP_THREADS)
knapsack_seed_kernel(const float* __restrict__ scores, int64_t row_stride, int len,
                     const float* __restrict__ budget, KnapOpts o, int use_smem,
                     float* __restrict__ lam0_out, int* __restrict__ ndbl_out) {
  extern __shared__ float smem_row[];
  __shared__ unsigned long long s_red[KNAP_THREADS / 32];
  __shared__ float s_max[KNAP_THREADS / 32];
  const int b = blockIdx.x;
  const float* row = stage_row(scores + (int64_t)b * row_stride, len, smem_row, use_smem != 0);
  float mx = -INFINITY;
  for (int i = threadIdx.x; i < len; i += KNAP_THREADS) mx = fmaxf(mx, row[i]);
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = -INFINITY;
  for (int w = 0; w < KNAP_THREADS / 32; ++w) mx = fmaxf(mx, s_max[w]);
  const float lam0 = fmaxf(__fmul_rn(mx, 0.375f), 1e-8f);
  const float bud = row_budget(budget, b, o);
  float lam = lam0;
  int k = 0;
  for (; k < 40; ++k) {
    const float avg = mean_of(sweep_sum(row, len, lam, o, s_red), len);
    if (!(avg > bud)) break;
    lam = __fmul_rn(lam, 2.0f);
  }
  if (threadIdx.x == 0) { lam0_out[b] = lam0; ndbl_out[b] = k; }
}

// Phase 2: batch-wide doubling count, lambda = 0 shortcut, bisection, final choice, row by row.
// The reference doubles lambda_hi for all rows inside ONE loop that ends when no row needs more or every
// lambda_hi reached 1e12; replay that loop on the seeds.
__device__ int batch_rounds(int n_rows, const float* __restrict__ lam0_all, const int* __restrict__ ndbl_all) {
  int rounds = 40;
  for (int it = 0; it < 40; ++it) {
    int any_need = 0, all_big = 1;
    for (int r = threadIdx.x; r < n_rows; r += KNAP_THREADS) {
      const int k = ndbl_all[r];
      if (k > it) any_need = 1;
      const float lam = ldexpf(lam0_all[r], min(it + 1, k));
      if (!(lam >= 1e12f)) all_big = 0;
    }
    any_need = __syncthreads_or(any_need);
    all_big = __syncthreads_and(all_big);
    if (!any_need) { rounds = it; break; }
    if (all_big) { rounds = it + 1; break; }
  }
  return rounds;
}

__device__ void solve_row(const float* row, int len, float bud, float lam_hi, const KnapOpts& o, int max_iters, float tol,
                          unsigned long long* s_red, int64_t* __restrict__ orow) {
  float lam_lo = 0.f, lam_final = 0.f;
  bool converged = !(mean_of(sweep_sum(row, len, 0.f, o, s_red), len) > bud);
  if (!converged) {
    float lam_mid = 0.f;
    for (int it = 0; it < max_iters; ++it) {
      lam_mid = __fdiv_rn(__fadd_rn(lam_lo, lam_hi), 2.0f);
      const float avg = mean_of(sweep_sum(row, len, lam_mid, o, s_red), len);
      const float rel = __fdiv_rn(fabsf(__fsub_rn(avg, bud)), fmaxf(bud, 1e-8f));
      if (rel < tol) { converged = true; break; }
      if (avg > bud) lam_lo = lam_mid; else lam_hi = lam_mid;
    }
    lam_final = lam_mid;                  // frozen value, or the last round's when never converged
  }
  float lb[KNAP_MAX_OPT];
#pragma unroll
  for (int n = 0; n < KNAP_MAX_OPT; ++n) lb[n] = n < o.n ? __fmul_rn(lam_final, o.bits[n]) : 0.f;
  for (int i = threadIdx.x; i < len; i += KNAP_THREADS) orow[i] = (int64_t)o.ibits[choose(row[i], nullptr, o, lb)];
}

__global__ void __launch_bounds__(KNAP_THREADS)
knapsack_solve_kernel(const float* __restrict__ scores, int64_t row_stride, int n_rows, int len,
                      const float* __restrict__ budget, KnapOpts o, int max_iters, float tol,
                      int use_smem, const float* __restrict__ lam0_all,
                      const int* __restrict__ ndbl_all, int64_t* __restrict__ out) {
  extern __shared__ float smem_row[];
  __shared__ unsigned long long s_red[KNAP_THREADS / 32];
  const int b = blockIdx.x;
  const int rounds = batch_rounds(n_rows, lam0_all, ndbl_all);
  const float* row = stage_row(scores + (int64_t)b * row_stride, len, smem_row, use_smem != 0);
  solve_row(row, len, row_budget(budget, b, o), ldexpf(lam0_all[b], min(rounds, ndbl_all[b])), o, max_iters, tol, s_red, out + (int64_t)b * len);
}

// The rows are solved already, with every doubling they asked for; do those again whose doublings the
// batch-wide loop would have cut short.  That takes lambda_hi >= 1e12 in EVERY row while the row still asks for
// more, so only a row whose own lambda_hi got there before its last doubling can be one: usually there is
// none and the one CTA leaves after a look at the seeds.
__global__ void __launch_bounds__(KNAP_THREADS)
knapsack_cut_kernel(const float* __restrict__ scores, int64_t row_stride, int n_rows, int len,
                    const float* __restrict__ budget, KnapOpts o, int max_iters, float tol,
                    const float* __restrict__ lam0_all, const int* __restrict__ ndbl_all, int64_t* __restrict__ out) {
  __shared__ unsigned long long s_red[KNAP_THREADS / 32];
  auto late = [&](int b) { return ndbl_all[b] >= 2 && ldexpf(lam0_all[b], ndbl_all[b] - 1) >= 1e12f; };
  int any = 0;
  for (int b = threadIdx.x; b < n_rows; b += KNAP_THREADS) any |= late(b) ? 1 : 0;
  if (!__syncthreads_or(any)) return;
  const int rounds = batch_rounds(n_rows, lam0_all, ndbl_all);
  for (int b = 0; b < n_rows; ++b)
    if (late(b) && rounds < ndbl_all[b])
      solve_row(scores + (int64_t)b * row_stride, len, row_budget(budget, b, o), ldexpf(lam0_all[b], rounds), o, max_iters, tol, s_red,
                out + (int64_t)b * len);
}

// The single-row form of the reference (knapsack_solver.py:39-118) differs from the batched one in
// its arithmetic: the multiplier is bisected in double precision (Python floats) and enters the cost
// as its fp32 rounding, means and the tolerance test are compared in double, lambda_hi has no 1e-8
// floor and is doubled row by row until the mean fits or it reaches 1e12.  One CTA per row, rows
// independent.  (The reference does not terminate on a row whose scores are all zero while its
// cheapest option is above the budget — lambda_hi stays 0; the doubling here stops after 200 rounds.)
__global__ void __launch_bounds__(KNAP_THREADS)
knapsack_scalar_kernel(const float* __restrict__ scores, int64_t row_stride, int len,
                       const double* __restrict__ budget, KnapOpts o, int max_iters, double tol,
                       int use_smem, int64_t* __restrict__ out) {
  extern __shared__ float smem_row[];
  __shared__ unsigned long long s_red[KNAP_THREADS / 32];
  __shared__ float s_max[KNAP_THREADS / 32];
  const int b = blockIdx.x;
  const float* row = stage_row(scores + (int64_t)b * row_stride, len, smem_row, use_smem != 0);
  float mx = -INFINITY;
  for (int i = threadIdx.x; i < len; i += KNAP_THREADS) mx = fmaxf(mx, row[i]);
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = -INFINITY;
  for (int w = 0; w < KNAP_THREADS / 32; ++w) mx = fmaxf(mx, s_max[w]);
  const double bud = budget[b];
  auto avg_at = [&](double lam) { return (double)mean_of(sweep_sum(row, len, (float)lam, o, s_red), len); };
  double lam_lo = 0.0, lam_hi = (double)mx * 0.375;
  for (int k = 0; k < 200 && avg_at(lam_hi) > bud && lam_hi < 1e12; ++k) lam_hi *= 2.0;
  double lam_final = 0.0;
  if (!(avg_at(0.0) <= bud)) {
    double lam_mid = 0.0;
    for (int it = 0; it < max_iters; ++it) {
      lam_mid = (lam_lo + lam_hi) / 2.0;
      const double avg = avg_at(lam_mid);
      if (fabs(avg - bud) / fmax(bud, 1e-8) < tol) break;
      if (avg > bud) lam_lo = lam_mid; else lam_hi = lam_mid;
    }
    lam_final = lam_mid;
  }
  float lb[KNAP_MAX_OPT];
#pragma unroll
  for (int n = 0; n < KNAP_MAX_OPT; ++n) lb[n] = n < o.n ? __fmul_rn((float)lam_final, o.bits[n]) : 0.f;
  int64_t* orow = out + (int64_t)b * len;
  for (int i = threadIdx.x; i < len; i += KNAP_THREADS) orow[i] = (int64_t)o.ibits[choose(row[i], nullptr, o, lb)];
}

// The K allocation's budgets from the V allocation's result: a row's kept tokens counted, then
// k_budget_bits / (head_dim * max(kept, 1)) in the rounding of the reference's expression (a number divided by
// an fp32 tensor: the reciprocal, then the product; obkv_fast.py:983, 1033-1035).  One CTA per row, 16-byte
// loads; stands for seven element-wise launches.
__global__ void __launch_bounds__(1024)
k_budget_kernel(const int64_t* __restrict__ v_bits, int64_t row_stride, int len, int head_dim, float k_budget_bits,
                float* __restrict__ out) {
  __shared__ int s_cnt[32];
  const int64_t* row = v_bits + (int64_t)blockIdx.x * row_stride;
  int cnt = 0;
  const int lead = (int)((reinterpret_cast<uintptr_t>(row) >> 3) & 1);      // elements ahead of the first 16-byte boundary
  const int pairs = (len - lead) / 2;
  const longlong2* p = reinterpret_cast<const longlong2*>(row + lead);
#pragma unroll 4
  for (int i = threadIdx.x; i < pairs; i += 1024) {
    const longlong2 v = __ldg(p + i);
    cnt += (int)(v.x > 0) + (int)(v.y > 0);
  }
  if (threadIdx.x == 0 && lead != 0 && len > 0) cnt += row[0] > 0;
  if (threadIdx.x == 1 && lead + 2 * pairs < len) cnt += row[len - 1] > 0;
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if ((threadIdx.x & 31) == 0) s_cnt[threadIdx.x >> 5] = cnt;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int kept = max(__reduce_add_sync(0xffffffffu, s_cnt[threadIdx.x]), 1);
    if (threadIdx.x == 0)
      out[blockIdx.x] = __fmul_rn(__fdiv_rn(1.f, __fmul_rn((float)head_dim, (float)kept)), k_budget_bits);
  }
}

// Bits a layer's packed form stands for: V bits times head_dim, plus every head's K bits per kept token
// (obkv_accel/blockwise_decode.py:665-678).  One CTA per layer, a warp per head; the maps are a block's
// (some thousand elements), so the launch is what it costs.
__global__ void __launch_bounds__(256)
logical_bits_kernel(const int64_t* __restrict__ v_bits, const int64_t* __restrict__ k_bits, int H, int T, int head_dim,
                    int64_t* __restrict__ out) {
  __shared__ unsigned long long s_sum;
  const int64_t* v = v_bits + (int64_t)blockIdx.x * H * T;
  const int64_t* k = k_bits + (int64_t)blockIdx.x * H * head_dim;
  if (threadIdx.x == 0) s_sum = 0ull;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int h = threadIdx.x >> 5; h < H; h += blockDim.x >> 5) {
    int64_t vs = 0, ks = 0, kept = 0;
    for (int i = lane; i < T; i += 32) { const int64_t b = v[(int64_t)h * T + i]; vs += b; kept += b > 0; }
    for (int i = lane; i < head_dim; i += 32) ks += k[(int64_t)h * head_dim + i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      vs += __shfl_xor_sync(0xffffffffu, vs, o); ks += __shfl_xor_sync(0xffffffffu, ks, o); kept += __shfl_xor_sync(0xffffffffu, kept, o);
    }
    if (lane == 0) atomicAdd(&s_sum, (unsigned long long)(vs * head_dim + ks * kept));
  }
  __syncthreads();
  if (threadIdx.x == 0) out[blockIdx.x] = (int64_t)s_sum;
}

}  // namespace rdkv

using namespace rdkv;

static int fill_options(KnapOpts& o, const float* option_bits, const float* option_eps, int n_options, int len) {
  o.n = n_options;
  o.budget = 0.f;
  float max_bit = 0.f;
  for (int n = 0; n < KNAP_MAX_OPT; ++n) {
    o.bits[n] = n < n_options ? option_bits[n] : 0.f;
    o.eps[n] = n < n_options ? option_eps[n] : 0.f;
    o.ibits[n] = (int)o.bits[n];
    if (n < n_options) {
      if (o.bits[n] < 0.f || (float)o.ibits[n] != o.bits[n]) return RDKV_ERR_BAD_ARG;
      max_bit = o.bits[n] > max_bit ? o.bits[n] : max_bit;
    }
  }
  if ((double)len * (double)max_bit >= 16777216.0) return RDKV_ERR_TOO_LARGE;
  return RDKV_OK;
}

static int launch_warp_rows(const float* scores, int64_t row_stride, int n_rows, int len, const float* budget,
                            const KnapOpts& o, int max_iters, float tol, float* lam0, int* ndbl, int64_t* out, cudaStream_t st) {
  const bool alone = n_rows <= KW_ALONE;
  const int grid = alone ? 1 : (n_rows + KW_WARPS - 1) / KW_WARPS, threads = (alone ? n_rows : KW_WARPS) * 32;
  const auto kernel = len <= 128 ? (alone ? knapsack_warp_kernel<4, true> : knapsack_warp_kernel<4, false>)
                                 : (alone ? knapsack_warp_kernel<8, true> : knapsack_warp_kernel<8, false>);
  kernel<<<grid, threads, 0, st>>>(scores, row_stride, n_rows, len, budget, o, max_iters, tol, lam0, ndbl, out);
  return launch_status();
}

template <int S, int THREADS>
static int launch_bucket_rows_of(const float* scores, int64_t row_stride, int n_rows, int len, const float* budget,
                              const KnapOpts& o, int max_iters, float tol, int chunk, float* lam0, int* ndbl, int64_t* out,
                              cudaStream_t st) {
  const size_t smem = kb_smem_bytes(chunk);
  if ((int64_t)n_rows * S > 0x7fffffffLL) return RDKV_ERR_TOO_LARGE;
  // (the size of the longest part the instance takes)
  cudaError_t e = allow_dynamic_smem(knapsack_bucket_kernel<S, THREADS>, kb_smem_bytes(THREADS == 1024 ? KB_MAX_CHUNK : KB_SMALL_CHUNK));
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_rows * S);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, knapsack_bucket_kernel<S, THREADS>, scores, row_stride, len, budget, o, max_iters, tol, chunk, lam0, ndbl, out);
  }
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return RDKV_ERR_LAUNCH; }
  return launch_status();
}

template <int S>
static int launch_bucket_rows(const float* scores, int64_t row_stride, int n_rows, int len, const float* budget,
                              const KnapOpts& o, int max_iters, float tol, int chunk, float* lam0, int* ndbl, int64_t* out,
                              cudaStream_t st) {
  return (chunk > KB_SMALL_CHUNK ? launch_bucket_rows_of<S, 1024> : launch_bucket_rows_of<S, 512>)(
      scores, row_stride, n_rows, len, budget, o, max_iters, tol, chunk, lam0, ndbl, out, st);
}

extern "C" int rdkv_knapsack_rows(const float* scores, int64_t row_stride, int n_rows, int len, const double* budget,
                                  const float* option_bits, const float* option_eps, int n_options, int max_iters,
                                  double tol, int64_t* out, void* stream) {
  if (scores == nullptr || budget == nullptr || option_bits == nullptr || option_eps == nullptr || out == nullptr)
    return RDKV_ERR_BAD_ARG;
  if (n_rows < 0 || len <= 0 || max_iters < 0) return RDKV_ERR_BAD_ARG;
  if (n_options <= 0 || n_options > KNAP_MAX_OPT) return RDKV_ERR_BAD_SHAPE;
  if (n_rows == 0) return RDKV_OK;
  KnapOpts o;
  const int rc = fill_options(o, option_bits, option_eps, n_options, len);
  if (rc != RDKV_OK) return rc;
  const size_t row_bytes = (size_t)len * sizeof(float);
  const int use_smem = row_bytes <= (size_t)KNAP_SMEM_ROW_BYTES ? 1 : 0;
  const size_t smem = use_smem ? row_bytes : 0;
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(knapsack_scalar_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KNAP_SMEM_ROW_BYTES);
  knapsack_scalar_kernel<<<n_rows, KNAP_THREADS, smem, (cudaStream_t)stream>>>(scores, row_stride, len, budget, o,
                                                                              max_iters, tol, use_smem, out);
  return launch_status();
}

// budget: per row, or null with one for all rows in budget_all.
static int knapsack_batched(const float* scores, int64_t row_stride, int n_rows, int len, const float* budget, float budget_all,
                            const float* option_bits, const float* option_eps, int n_options, int max_iters, float tol,
                            int64_t* out, void* scratch, void* stream) {
  if (scores == nullptr || option_bits == nullptr || option_eps == nullptr || out == nullptr || scratch == nullptr)
    return RDKV_ERR_BAD_ARG;
  if (n_rows < 0 || len <= 0 || max_iters < 0) return RDKV_ERR_BAD_ARG;
  if (n_options <= 0 || n_options > KNAP_MAX_OPT) return RDKV_ERR_BAD_SHAPE;
  if (n_rows == 0) return RDKV_OK;
  KnapOpts o;
  const int orc = fill_options(o, option_bits, option_eps, n_options, len);
  if (orc != RDKV_OK) return orc;
  o.budget = budget_all;
  float* lam0 = reinterpret_cast<float*>(scratch);
  int* ndbl = reinterpret_cast<int*>(lam0 + 2 * (size_t)n_rows);
  cudaStream_t st = (cudaStream_t)stream;
  // How many CTAs share a row: one where the rows fill the chip by themselves, else as many as that takes
  // (but no part below 2048 scores: a sweep's barriers would outweigh its work); more where a part
  // would not fit its shared memory.
  // 256 rows x 32768: 362 us (every element in every sweep) -> 94 us with one CTA per row; 126
  // with two, 203 with four.  8 rows x 32768: 178 -> 36 us with eight, 58 with one.  8 x 131072: 727 -> 54.
  int dev = 0, sms = 0, cluster = 1;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    g_last_cuda_error = (int)cudaGetLastError();
    return RDKV_ERR_LAUNCH;
  }
  while (cluster < KB_MAX_CLUSTER && ((len / (2 * cluster) >= 2048 && (int64_t)n_rows * 2 * cluster <= 2 * sms) || len > cluster * KB_MAX_CHUNK))
    cluster *= 2;
  const int chunk = ((len + cluster - 1) / cluster + 3) & ~3;
  bool eps_ok = true;                                       // (the bucket test bounds rounding errors by the costs: no negative terms)
  for (int x = 0; x < n_options; ++x) eps_ok = eps_ok && o.eps[x] >= 0.f;
  if (eps_ok && chunk <= KB_MAX_CHUNK) {
    int rc = len <= 256 ? launch_warp_rows(scores, row_stride, n_rows, len, budget, o, max_iters, tol, lam0, ndbl, out, st)
           : cluster == 8 ? launch_bucket_rows<8>(scores, row_stride, n_rows, len, budget, o, max_iters, tol, chunk, lam0, ndbl, out, st)
           : cluster == 4 ? launch_bucket_rows<4>(scores, row_stride, n_rows, len, budget, o, max_iters, tol, chunk, lam0, ndbl, out, st)
           : cluster == 2 ? launch_bucket_rows<2>(scores, row_stride, n_rows, len, budget, o, max_iters, tol, chunk, lam0, ndbl, out, st)
                          : launch_bucket_rows<1>(scores, row_stride, n_rows, len, budget, o, max_iters, tol, chunk, lam0, ndbl, out, st);
    if (rc != RDKV_OK || (len <= 256 && n_rows <= KW_ALONE)) return rc;
    knapsack_cut_kernel<<<1, KNAP_THREADS, 0, st>>>(scores, row_stride, n_rows, len, budget, o, max_iters, tol, lam0, ndbl, out);
    return launch_status();
  }
  const size_t row_bytes = (size_t)len * sizeof(float);
  const int use_smem = row_bytes <= (size_t)KNAP_SMEM_ROW_BYTES ? 1 : 0;
  const size_t smem = use_smem ? row_bytes : 0;
  if (smem > 48 * 1024) {
    cudaFuncSetAttribute(knapsack_seed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KNAP_SMEM_ROW_BYTES);
    cudaFuncSetAttribute(knapsack_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KNAP_SMEM_ROW_BYTES);
  }
  knapsack_seed_kernel<<<n_rows, KNAP_THREADS, smem, st>>>(scores, row_stride, len, budget, o, use_smem, lam0, ndbl);
  int rc = launch_status();
  if (rc != RDKV_OK) return rc;
  knapsack_solve_kernel<<<n_rows, KNAP_THREADS, smem, st>>>(scores, row_stride, n_rows, len, budget, o,
                                                           max_iters, tol, use_smem, lam0, ndbl, out);
  return launch_status();
}

extern "C" int rdkv_knapsack_batched(const float* scores, int64_t row_stride, int n_rows, int len,
                                     const float* budget, const float* option_bits,
                                     const float* option_eps, int n_options, int max_iters, float tol,
                                     int64_t* out, void* scratch, void* stream) {
  if (budget == nullptr) return RDKV_ERR_BAD_ARG;
  return knapsack_batched(scores, row_stride, n_rows, len, budget, 0.f, option_bits, option_eps, n_options, max_iters, tol, out,
                          scratch, stream);
}

extern "C" int rdkv_knapsack_batched_uniform(const float* scores, int64_t row_stride, int n_rows, int len, float budget,
                                             const float* option_bits, const float* option_eps, int n_options,
                                             int max_iters, float tol, int64_t* out, void* scratch, void* stream) {
  return knapsack_batched(scores, row_stride, n_rows, len, nullptr, budget, option_bits, option_eps, n_options, max_iters, tol, out,
                          scratch, stream);
}

// ── allocation-free variant ──────────────────────────────────────────────────
// Some callers cannot provide the per-row scratch of rdkv_knapsack_batched because
// they are not allowed to allocate device memory at the point of the call: a
// prefill step that runs inside an engine's fixed memory plan after warm-up, or a
// plugin interface that hands over input and output buffers only.
// For them the scratch lives in this library's own device image: a file-scope
// array that every GPU loading the library carries until the process exits.
// (One warm-up call per device, made before the memory plan is frozen and before any
// stream capture, looks the array's address up and lets the runtime load the module
// and every kernel that a call of any shape may choose: with lazy loading a kernel's code
// would otherwise be loaded by the first launch of it.)
constexpr int KNAP_STATIC_MAX_ROWS = 4096;                 // 3 words per row -> 48 KiB per GPU
static __device__ __align__(256) unsigned int g_knap_static_scratch[3 * KNAP_STATIC_MAX_ROWS];

#include <mutex>
namespace {
constexpr int KNAP_MAX_DEVICES = 64;
std::mutex g_knap_static_mutex;
void* g_knap_static_addr[KNAP_MAX_DEVICES] = {nullptr};   // device address of the array, per device
}  // namespace

template <typename... Kernels>
static cudaError_t load_kernels(Kernels... kernels) {
  cudaError_t e = cudaSuccess;
  cudaFuncAttributes attr;
  ((e = e == cudaSuccess ? cudaFuncGetAttributes(&attr, kernels) : e), ...);   // (loads the code, lazy or not)
  return e;
}

// Every kernel that knapsack_batched chooses from.
static cudaError_t load_batched_kernels() {
  return load_kernels(knapsack_bucket_kernel<1, 512>, knapsack_bucket_kernel<2, 512>, knapsack_bucket_kernel<4, 512>,
                      knapsack_bucket_kernel<8, 512>, knapsack_bucket_kernel<1, 1024>, knapsack_bucket_kernel<2, 1024>,
                      knapsack_bucket_kernel<4, 1024>, knapsack_bucket_kernel<8, 1024>, knapsack_warp_kernel<4, false>,
                      knapsack_warp_kernel<4, true>, knapsack_warp_kernel<8, false>, knapsack_warp_kernel<8, true>,
                      knapsack_cut_kernel, knapsack_seed_kernel, knapsack_solve_kernel);
}

extern "C" int rdkv_knapsack_static_max_rows(void) { return KNAP_STATIC_MAX_ROWS; }

extern "C" int rdkv_knapsack_batched_static(const float* scores, int64_t row_stride, int n_rows, int len,
                                            const float* budget, const float* option_bits,
                                            const float* option_eps, int n_options, int max_iters, float tol,
                                            int64_t* out, void* stream) {
  if (n_rows > KNAP_STATIC_MAX_ROWS) return RDKV_ERR_TOO_LARGE;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= KNAP_MAX_DEVICES) {
    g_last_cuda_error = (int)e;
    return RDKV_ERR_NO_DEVICE;
  }
  void* scratch = nullptr;
  {
    // The array's name is only a host-side handle; the address a kernel can use is
    // looked up once per device, with that device current.
    std::lock_guard<std::mutex> lock(g_knap_static_mutex);
    if (g_knap_static_addr[dev] == nullptr) {
      void* p = nullptr;
      e = load_batched_kernels();
      if (e == cudaSuccess) e = cudaGetSymbolAddress(&p, g_knap_static_scratch);
      if (e != cudaSuccess || p == nullptr) {
        g_last_cuda_error = (int)e;
        return RDKV_ERR_LAUNCH;
      }
      g_knap_static_addr[dev] = p;
    }
    scratch = g_knap_static_addr[dev];
  }
  return rdkv_knapsack_batched(scores, row_stride, n_rows, len, budget, option_bits, option_eps, n_options,
                               max_iters, tol, out, scratch, stream);
}

extern "C" int rdkv_k_budgets(const int64_t* v_bits, int64_t row_stride, int n_rows, int len, int head_dim,
                              float k_budget_bits, float* out, void* stream) {
  if (n_rows < 0 || len < 0 || head_dim <= 0) return RDKV_ERR_BAD_ARG;
  if (n_rows == 0) return RDKV_OK;
  if (v_bits == nullptr || out == nullptr || (reinterpret_cast<uintptr_t>(v_bits) & 7)) return RDKV_ERR_BAD_ARG;
  k_budget_kernel<<<n_rows, 1024, 0, (cudaStream_t)stream>>>(v_bits, row_stride, len, head_dim, k_budget_bits, out);
  return launch_status();
}

extern "C" int rdkv_logical_bits(const int64_t* v_bits, const int64_t* k_bits, int n_layers, int H, int T, int head_dim,
                                 int64_t* out, void* stream) {
  if (n_layers < 0 || H <= 0 || T < 0 || head_dim <= 0) return RDKV_ERR_BAD_ARG;
  if (n_layers == 0) return RDKV_OK;
  if ((T > 0 && v_bits == nullptr) || k_bits == nullptr || out == nullptr) return RDKV_ERR_BAD_ARG;
  logical_bits_kernel<<<n_layers, 256, 0, (cudaStream_t)stream>>>(v_bits, k_bits, H, T, head_dim, out);
  return launch_status();
}
