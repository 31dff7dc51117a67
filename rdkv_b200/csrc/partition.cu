// Stable partition of bit maps into classes, and the small per-head tables that follow from it.
//
// Replaces the argsort(stable) / nonzero calls of the reference's packer (obkv_accel/packing.py:715-778,
// :399-440) and the host arithmetic of its stacking step (:1236-1290).
#include <cooperative_groups.h>

#include "rdkv_common.cuh"

namespace rdkv {

// ── partition ────────────────────────────────────────────────────────────────
// Bound by the reads of the maps (8 bytes an element as the allocator returns them) and, for few rows, by
// latency.  A row is cut into runs for a cluster of CTAs, a CTA's run into runs for its warps, a warp's run
// into tiles of 256 elements: eight neighbouring ones per lane (vector loads where they are aligned).  A lane
// classifies its eight elements once and keeps what the second step needs as one word per tile in shared
// memory (four bits an element: kept, class bit 0, class bit 1, compressed); that step writes every kept
// element to its place and does not read the map again.  Places: counts per lane, scanned over the warp tile by tile,
// over the warps once, over the cluster once (distributed shared memory).
// One CTA per row with one run per thread (an earlier form) read 64-bit maps 1 KB apart within a warp
// and left most SMs idle.  64-bit maps, kernel time: 32 rows x 131072 813 us (four launches of 8 rows) -> 18 us,
// 256 x 32768 55 -> 29 us, 8 x 32768 28 -> 8 us; 16-bit maps, 256 x 32768: 23 -> 28 us (every tile is turned into
// flags first), 32 x 131072: 770 -> 17 us.
// (Two CTAs per SM, classes in registers and the loops unrolled by the tiles: 26, 38, 10, 32 and 23 us, 28 us for
// four layers of 131072 rows in one launch, now 21; most of a warp's time went into instruction fetches.)
constexpr int PT_THREADS = 512;
constexpr int PT_WARPS = PT_THREADS / 32;
constexpr int PT_TILES = 8;                                 // tiles of a warp whose classes are kept
constexpr int PT_MAX_CLUSTER = 8;

struct PartSet {
  const void* bits; int64_t row_stride; int elem_size, n_rows, len, mode;   // mode 0: tokens (2, 4, 8, 16), 1: channels (16 counts as 8)
  int32_t* order; int32_t* counts; int32_t* rank;
};

// Elements i .. i+7 of a row (those below hi; the others read as 0) as small unsigned numbers: 0 for what is
// not positive, 3 for positive values of more than 32 bits (no class has either).
template <int ES>
__device__ __forceinline__ void part_load8(const void* row, int64_t i, int64_t hi, bool vec, uint32_t (&w)[8]) {
  if (vec && i + 8 <= hi) {
    if (ES == 8) {
      const uint4* p = reinterpret_cast<const uint4*>(reinterpret_cast<const int64_t*>(row) + i);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint4 v = __ldg(p + u);
        w[2 * u] = v.y == 0u ? v.x : (int)v.y > 0 ? 3u : 0u;
        w[2 * u + 1] = v.w == 0u ? v.z : (int)v.w > 0 ? 3u : 0u;
      }
    } else if (ES == 4) {
      const int4* p = reinterpret_cast<const int4*>(reinterpret_cast<const int32_t*>(row) + i);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int4 v = __ldg(p + u);
        w[4 * u] = max(v.x, 0); w[4 * u + 1] = max(v.y, 0); w[4 * u + 2] = max(v.z, 0); w[4 * u + 3] = max(v.w, 0);
      }
    } else if (ES == 2) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const int16_t*>(row) + i));
      const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) { w[2 * u] = max((int)(int16_t)x[u], 0); w[2 * u + 1] = max((int)x[u] >> 16, 0); }
    } else {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const int8_t*>(row) + i));
#pragma unroll
      for (int u = 0; u < 8; ++u) w[u] = max((int)(int8_t)((u < 4 ? v.x : v.y) >> (8 * (u & 3))), 0);
    }
    return;
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    w[u] = 0u;
    if (i + u < hi) {
      const int64_t b = ES == 8 ? reinterpret_cast<const int64_t*>(row)[i + u] : ES == 4 ? reinterpret_cast<const int32_t*>(row)[i + u]
                      : ES == 2 ? reinterpret_cast<const int16_t*>(row)[i + u] : reinterpret_cast<const int8_t*>(row)[i + u];
      w[u] = b <= 0 ? 0u : b > 0x7fffffffLL ? 3u : (uint32_t)b;
    }
  }
}

// Bytes of flags of eight elements: kept | class bit 0 << 8 | class bit 1 << 16 | compressed << 24.
__device__ __forceinline__ uint32_t part_flags(const uint32_t (&w)[8], int mode) {
  const uint32_t t_keep = 1u << 2 | 1u << 4 | 1u << 8 | 1u << 16;
  const uint32_t t_b0 = 1u << 4 | (mode == 0 ? 1u << 16 : 0u), t_b1 = 1u << 8 | 1u << 16;
  uint32_t f = 0u;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const uint32_t x = min(w[u], 31u);
    const uint32_t one = ((t_keep >> x) & 1u) | ((t_b0 >> x) & 1u) << 8 | ((t_b1 >> x) & 1u) << 16 |
                         (uint32_t)(x != 0u && x != 16u) << 24;
    f |= one << u;
  }
  return f;
}

// A lane's counts of one tile: classes 0 and 1, classes 2 and 3 (16 bits each), compressed elements.
struct PartCount { uint32_t c01, c23, comp; };
__device__ __forceinline__ PartCount part_count(uint32_t f) {
  const uint32_t k = f & 0xFFu, b0 = (f >> 8) & 0xFFu, b1 = (f >> 16) & 0xFFu;
  PartCount c;
  c.c01 = (uint32_t)__popc(k & ~b0 & ~b1) | (uint32_t)__popc(b0 & ~b1) << 16;
  c.c23 = (uint32_t)__popc(b1 & ~b0) | (uint32_t)__popc(b0 & b1) << 16;
  c.comp = (uint32_t)__popc(f >> 24);
  return c;
}

// Two sets of rows in one launch (a layer's token maps and its channel maps); a cluster per row.
// fill: entries past a row's kept count become -1.  rank (may be null): for every place in a compressed
// class the element's number among the row's compressed elements (bits > 0 and not 16) in ascending order.
template <int ES>
__device__ __forceinline__ void partition_row(const PartSet& P, int row, int fill, uint32_t (*s_flags)[PT_THREADS], int (*s_warp)[5], int* s_cta) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), n_cta = (int)cluster.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int len = P.len, mode = P.mode;
  const void* src = reinterpret_cast<const unsigned char*>(P.bits) + (int64_t)row * P.row_stride * ES;
  const bool vec = (reinterpret_cast<uintptr_t>(src) & (ES == 1 ? 7 : 15)) == 0;
  // elements of this warp: whole tiles
  const int per_warp = (((len + n_cta * PT_WARPS - 1) / (n_cta * PT_WARPS)) + 255) & ~255;
  const int64_t lo = min((int64_t)len, (int64_t)(rank * PT_WARPS + warp) * per_warp);
  const int64_t hi = min((int64_t)len, lo + per_warp);
  const int tiles = (int)((hi - lo + 255) >> 8);
  const bool cached = per_warp <= PT_TILES * 256;           // every tile's classes are kept
  PartCount sum = {0u, 0u, 0u};
  auto tile_flags = [&](int t) {
    uint32_t w[8];
    part_load8<ES>(src, lo + 256 * t + 8 * lane, hi, vec, w);
    return part_flags(w, mode);
  };
  auto note = [&](uint32_t f) {
    const PartCount c = part_count(f);
    sum.c01 += c.c01; sum.c23 += c.c23; sum.comp += c.comp;
  };
  int cnt[5] = {0, 0, 0, 0, 0};
  auto warp_totals = [&]() {                                // (at most 8 x 8 per lane and field: no carry between the halves)
    const uint32_t a = __reduce_add_sync(0xffffffffu, sum.c01), b = __reduce_add_sync(0xffffffffu, sum.c23);
    cnt[0] += a & 0xFFFFu; cnt[1] += a >> 16; cnt[2] += b & 0xFFFFu; cnt[3] += b >> 16;
    cnt[4] += __reduce_add_sync(0xffffffffu, sum.comp);
    sum = {0u, 0u, 0u};
  };
  // (both loops over the tiles are kept short: a CTA goes through its code once or twice, and unrolled by
  //  the tiles it waited for instruction fetches seven cycles per instruction)
#pragma unroll 1
  for (int t = 0; t < tiles; ++t) {
    const uint32_t f = tile_flags(t);
    if (cached) s_flags[t][tid] = f;
    note(f);
    if ((t & 7) == 7) warp_totals();
  }
  warp_totals();
  if (lane == 0)
#pragma unroll
    for (int c = 0; c < 5; ++c) s_warp[warp][c] = cnt[c];
  __syncthreads();
  if (tid < 5) {                                            // exclusive sums over the warps
    int t = 0;
#pragma unroll
    for (int w = 0; w < PT_WARPS; ++w) { const int x = s_warp[w][tid]; s_warp[w][tid] = t; t += x; }
    s_cta[tid] = t;
  }
  cluster.sync();
  int before[5] = {0, 0, 0, 0, 0}, total[5] = {0, 0, 0, 0, 0};
  for (int q = 0; q < n_cta; ++q) {
    const int* t = cluster.map_shared_rank(s_cta, q);
#pragma unroll
    for (int c = 0; c < 5; ++c) { const int x = t[c]; if (q < rank) before[c] += x; total[c] += x; }
  }
  if (rank == 0 && tid < 4) P.counts[row * 4 + tid] = tid == 0 ? total[0] : tid == 1 ? total[1] : tid == 2 ? total[2] : total[3];
  int pos[4], comp_at = before[4] + s_warp[warp][4];
  pos[0] = before[0] + s_warp[warp][0];
  pos[1] = total[0] + before[1] + s_warp[warp][1];
  pos[2] = total[0] + total[1] + before[2] + s_warp[warp][2];
  pos[3] = total[0] + total[1] + total[2] + before[3] + s_warp[warp][3];
  const int kept = total[0] + total[1] + total[2] + total[3];
  int32_t* orow = P.order + (int64_t)row * len;
  int32_t* rrow = P.rank != nullptr ? P.rank + (int64_t)row * len : nullptr;
  auto place = [&](int t, uint32_t f) {
    const PartCount c = part_count(f);
    uint32_t i01 = c.c01, i23 = c.c23, icomp = c.comp;      // inclusive sums over the lanes
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, i01, d), y = __shfl_up_sync(0xffffffffu, i23, d), z = __shfl_up_sync(0xffffffffu, icomp, d);
      if (lane >= d) { i01 += x; i23 += y; icomp += z; }
    }
    const uint32_t t01 = __shfl_sync(0xffffffffu, i01, 31), t23 = __shfl_sync(0xffffffffu, i23, 31), tcomp = __shfl_sync(0xffffffffu, icomp, 31);
    i01 -= c.c01; i23 -= c.c23; icomp -= c.comp;
    int at[4] = {pos[0] + (int)(i01 & 0xFFFFu), pos[1] + (int)(i01 >> 16), pos[2] + (int)(i23 & 0xFFFFu), pos[3] + (int)(i23 >> 16)};
    const int first = (int)lo + 256 * t + 8 * lane, comp0 = comp_at + (int)icomp;
    for (uint32_t m = f & 0xFFu; m != 0u; m &= m - 1) {     // kept elements in ascending order
      const int u = __ffs(m) - 1;
      const int b0 = (f >> (8 + u)) & 1u, b1 = (f >> (16 + u)) & 1u;
      const int where = b1 ? (b0 ? at[3] : at[2]) : (b0 ? at[1] : at[0]);
      if (b1) { if (b0) ++at[3]; else ++at[2]; } else { if (b0) ++at[1]; else ++at[0]; }
      orow[where] = first + u;
      if (rrow != nullptr && !(b0 && b1)) rrow[where] = comp0 + __popc((f >> 24) & ((1u << u) - 1u));
    }
    pos[0] += (int)(t01 & 0xFFFFu); pos[1] += (int)(t01 >> 16); pos[2] += (int)(t23 & 0xFFFFu); pos[3] += (int)(t23 >> 16);
    comp_at += (int)tcomp;
  };
#pragma unroll 1
  for (int t = 0; t < tiles; ++t) place(t, cached ? s_flags[t][tid] : tile_flags(t));
  if (fill)
    for (int i = kept + rank * PT_THREADS + tid; i < len; i += n_cta * PT_THREADS) orow[i] = -1;
  cluster.sync();                                           // (the totals are read by the other CTAs)
}

__global__ void __launch_bounds__(PT_THREADS, 3)
partition_pair_kernel(const __grid_constant__ PartSet A, const __grid_constant__ PartSet B, int fill) {
  __shared__ uint32_t s_flags[PT_TILES][PT_THREADS];        // a lane's classes of its warp's tiles
  __shared__ int s_warp[PT_WARPS][5];                       // per warp: elements of classes 0..3, compressed elements
  __shared__ int s_cta[5];                                  // the CTA's totals (read by the whole cluster)
  const int r = blockIdx.x / (int)cooperative_groups::this_cluster().num_blocks();
  const PartSet& P = r < A.n_rows ? A : B;
  const int row = r < A.n_rows ? r : r - A.n_rows;
  switch (P.elem_size) {
    case 1: partition_row<1>(P, row, fill, s_flags, s_warp, s_cta); break;
    case 2: partition_row<2>(P, row, fill, s_flags, s_warp, s_cta); break;
    case 4: partition_row<4>(P, row, fill, s_flags, s_warp, s_cta); break;
    default: partition_row<8>(P, row, fill, s_flags, s_warp, s_cta); break;
  }
}

// ── per-head tables of a packed layer ─────────────────────────────────────────
// Row counts per head as the packed layer carries them, and the additive softmax mask [H*gqa][t_k]: 0 on a
// head's live rows ([0, t_v) and [max_t_v, max_t_v + n16)), -inf on stripe padding (obkv_accel/packing.py:
// 1236-1257); and the first head's V sort order (rank_row[0 .. n_sort) as 64-bit integers).  One launch for up to eight layers instead of some twenty element-wise ones each.  Bound by the launch and, for
// long stripes, by the mask's 4 bytes per query head and row.
constexpr int PM_THREADS = 256;
constexpr int PM_COLS = 4096;                               // mask columns per CTA

constexpr int PM_LAYERS = 8;                                // layers per launch (their records are launch arguments)
struct MetaJobs { rdkv_pack_meta_job j[PM_LAYERS]; };

__global__ void __launch_bounds__(PM_THREADS)
pack_meta_kernel(const __grid_constant__ MetaJobs jobs, int gqa) {
  const rdkv_pack_meta_job& J = jobs.j[blockIdx.z];
  const int hq = blockIdx.y, h = hq / gqa;
  const int max_t_v = J.max_t_v, t_k = J.t_k;
  const int4 c = *reinterpret_cast<const int4*>(J.counts + 4 * h);
  const int t_v = c.x + c.y + c.z, n16 = c.w;
  if (blockIdx.x == 0 && hq == h * gqa && threadIdx.x == 0) {
    J.seg_bounds[3 * h] = c.x; J.seg_bounds[3 * h + 1] = c.y; J.seg_bounds[3 * h + 2] = c.z;
    J.t_eff[h] = t_v; J.n_v16[h] = n16; J.t_eff_k[h] = t_v + n16;
  }
  const int c0 = blockIdx.x * PM_COLS;
  if (hq == 0)
    for (int i = c0 + threadIdx.x; i < min(J.n_sort, c0 + PM_COLS); i += PM_THREADS) J.sort_idx[i] = J.rank_row[i];
  if (J.mask == nullptr) return;
  const int c1 = min(t_k, c0 + PM_COLS);
  float* row = J.mask + (int64_t)hq * t_k;
  auto value = [&](int col) { return (col < t_v || (col >= max_t_v && col < max_t_v + n16)) ? 0.f : -INFINITY; };
  if ((t_k & 3) == 0 && (reinterpret_cast<uintptr_t>(J.mask) & 15) == 0) {
    for (int col = c0 + 4 * threadIdx.x; col < c1; col += 4 * PM_THREADS)
      *reinterpret_cast<float4*>(row + col) = make_float4(value(col), value(col + 1), value(col + 2), value(col + 3));
  } else {
    for (int col = c0 + threadIdx.x; col < c1; col += PM_THREADS) row[col] = value(col);
  }
}

}  // namespace rdkv

using namespace rdkv;

static int launch_partition(const PartSet& A, const PartSet& B, int fill, cudaStream_t st) {
  const int rows = A.n_rows + B.n_rows;
  if (rows == 0) return RDKV_OK;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    g_last_cuda_error = (int)cudaGetLastError();
    return RDKV_ERR_LAUNCH;
  }
  // CTAs per row: enough to give every SM one and to keep every tile's classes (eight tiles a warp), but not
  // less than a tile a warp
  const int len = A.len > B.len ? A.len : B.len;
  int cluster = 1;
  while (cluster < PT_MAX_CLUSTER && len > cluster * PT_WARPS * 256 &&
         ((int64_t)rows * cluster < sms || len > cluster * PT_WARPS * PT_TILES * 256))
    cluster *= 2;
  if ((int64_t)rows * cluster > 0x7fffffffLL) return RDKV_ERR_TOO_LARGE;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(rows * cluster);
  cfg.blockDim = dim3(PT_THREADS);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, partition_pair_kernel, A, B, fill);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return RDKV_ERR_LAUNCH; }
  return launch_status();
}

static int part_set(PartSet& P, const void* bits, int elem_size, int64_t row_stride, int n_rows, int len, int mode,
                    int32_t* order, int32_t* counts, int32_t* rank) {
  if (n_rows < 0 || len < 0) return RDKV_ERR_BAD_ARG;
  if (n_rows > 0 && (bits == nullptr || order == nullptr || counts == nullptr)) return RDKV_ERR_BAD_ARG;
  if (elem_size != 1 && elem_size != 2 && elem_size != 4 && elem_size != 8) return RDKV_ERR_BAD_ARG;
  P.bits = bits; P.row_stride = row_stride; P.elem_size = elem_size; P.n_rows = n_rows; P.len = len; P.mode = mode;
  P.order = order; P.counts = counts; P.rank = rank;
  return RDKV_OK;
}

extern "C" int rdkv_partition_by_bits(const void* bits, int elem_size, int64_t row_stride, int n_rows, int len, int mode,
                                      int32_t* order, int32_t* counts, void* stream) {
  if (bits == nullptr || order == nullptr || counts == nullptr) return RDKV_ERR_BAD_ARG;
  if ((mode & ~4) != 0 && (mode & ~4) != 1) return RDKV_ERR_BAD_ARG;
  PartSet A, B = {};
  const int rc = part_set(A, bits, elem_size, row_stride, n_rows, len, mode & 1, order, counts, nullptr);
  if (rc != RDKV_OK) return rc;
  return launch_partition(A, B, (mode & 4) ? 0 : 1, (cudaStream_t)stream);
}

extern "C" int rdkv_partition_pair(const void* tok_bits, int tok_elem_size, int64_t tok_row_stride, int tok_rows, int tok_len,
                                   const void* ch_bits, int ch_elem_size, int64_t ch_row_stride, int ch_rows, int ch_len,
                                   int fill, int32_t* tok_order, int32_t* tok_rank, int32_t* ch_order, int32_t* counts,
                                   void* stream) {
  if (counts == nullptr || tok_rows < 0) return RDKV_ERR_BAD_ARG;
  PartSet A, B;
  int rc = part_set(A, tok_bits, tok_elem_size, tok_row_stride, tok_rows, tok_len, 0, tok_order, counts, tok_rank);
  if (rc == RDKV_OK) rc = part_set(B, ch_bits, ch_elem_size, ch_row_stride, ch_rows, ch_len, 1, ch_order, counts + 4 * (int64_t)tok_rows, nullptr);
  if (rc != RDKV_OK) return rc;
  return launch_partition(A, B, fill ? 1 : 0, (cudaStream_t)stream);
}

extern "C" int rdkv_sizeof_pack_meta_job(void) { return (int)sizeof(rdkv_pack_meta_job); }

extern "C" int rdkv_pack_meta(const rdkv_pack_meta_job* jobs, int n_jobs, int H, int gqa, void* stream) {
  if (jobs == nullptr || n_jobs < 0 || H <= 0 || gqa <= 0) return RDKV_ERR_BAD_ARG;
  if ((int64_t)H * gqa > 65535) return RDKV_ERR_TOO_LARGE;
  for (int i = 0; i < n_jobs; ++i) {
    const rdkv_pack_meta_job& J = jobs[i];
    if (J.counts == nullptr || J.seg_bounds == nullptr || J.t_eff == nullptr || J.n_v16 == nullptr || J.t_eff_k == nullptr) return RDKV_ERR_BAD_ARG;
    if (J.n_sort < 0 || (J.n_sort > 0 && (J.rank_row == nullptr || J.sort_idx == nullptr))) return RDKV_ERR_BAD_ARG;
    if (J.max_t_v < 0 || J.t_k < J.max_t_v || (reinterpret_cast<uintptr_t>(J.counts) & 15)) return RDKV_ERR_BAD_ARG;
  }
  for (int at = 0; at < n_jobs; at += PM_LAYERS) {
    const int n = n_jobs - at < PM_LAYERS ? n_jobs - at : PM_LAYERS;
    MetaJobs batch = {};
    int cols = 1;
    for (int i = 0; i < n; ++i) {
      batch.j[i] = jobs[at + i];
      const int c = jobs[at + i].mask != nullptr && jobs[at + i].t_k > jobs[at + i].n_sort ? jobs[at + i].t_k : jobs[at + i].n_sort;
      cols = c > cols ? c : cols;
    }
    pack_meta_kernel<<<dim3((cols + PM_COLS - 1) / PM_COLS, H * gqa, n), PM_THREADS, 0, (cudaStream_t)stream>>>(batch, gqa);
    const int rc = launch_status();
    if (rc != RDKV_OK) return rc;
  }
  return RDKV_OK;
}
