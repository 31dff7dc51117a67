// Packed layer -> fp16 (K, V) on the stripe token axis: the inverse of the prefill packer, for
// fallback attention through an unpacked cache and for debugging.
//
// Reference behaviour (obkv_accel/packing.py:581-709 unpack_k_mixed, :1427-1444 unpack_v_segment;
// obkv_accel/trizone_decompress.py:43-183): value = half((float(code) - float(zp)) * float(scale)),
// K scattered back to the original channel of each kept slot (evicted channels are zeros), V rows
// in head-local segment order [2-bit | 4-bit | 8-bit], zero rows up to max_T_v, then the fp16
// Zone-B rows.  The subtraction is exact (small integers), so one fp32 multiply and one rounding
// to fp16 reproduce the reference bit for bit.
#include "rdkv_common.cuh"

namespace rdkv {

constexpr int UNPACK_WARPS = 8;
constexpr int UNPACK_MAX_D = 512;

__device__ __forceinline__ uint16_t dequant_h(unsigned code, uint16_t zp_bits, uint16_t sc_bits) {
  const float d = __fsub_rn((float)code, h2f(zp_bits));
  return __half_as_ushort(__float2half_rn(__fmul_rn(d, h2f(sc_bits))));
}

// Any head dimension and alignment: grid (ceil(rows_out / UNPACK_WARPS), H_kv); one warp per stripe row.
__global__ void __launch_bounds__(UNPACK_WARPS * 32)
unpack_layer_kernel(rdkv_layer_view v, int D, const int64_t* __restrict__ k_sort_idx, int64_t k_sort_idx_head_stride,
                    const int32_t* __restrict__ k_ch_counts, int n_ch2, int n_ch4, int n_ch8,
                    uint16_t* __restrict__ k_out, uint16_t* __restrict__ v_out, int64_t out_head_stride, int rows_out) {
  __shared__ int16_t s_slot[UNPACK_MAX_D];                     // original channel -> slot in the padded order, -1: evicted
  const int h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n2p = v.n_ch2_pad, n4p = v.n_ch4_pad, n8p = v.n_ch8, d_pad = n2p + n4p + n8p;
  const int sub2 = n2p / 4, sub4 = n4p / 2;
  if (k_out != nullptr) {
    for (int c = threadIdx.x; c < D; c += blockDim.x) s_slot[c] = -1;
    __syncthreads();
    int c2 = n_ch2, c4 = n_ch4, c8 = n_ch8;
    if (k_ch_counts != nullptr) { c2 = k_ch_counts[h * 3 + 0]; c4 = k_ch_counts[h * 3 + 1]; c8 = k_ch_counts[h * 3 + 2]; }
    const int64_t* si = k_sort_idx + h * k_sort_idx_head_stride;
    for (int j = threadIdx.x; j < c2 + c4 + c8; j += blockDim.x) {
      const int slot = j < c2 ? j : j < c2 + c4 ? n2p + (j - c2) : n2p + n4p + (j - c2 - c4);
      const int64_t ch = si[j];
      if (ch >= 0 && ch < D) s_slot[ch] = (int16_t)slot;
    }
    __syncthreads();
  }
  const int row = blockIdx.x * UNPACK_WARPS + warp;
  if (row >= rows_out) return;

  if (k_out != nullptr) {
    uint16_t* dst = k_out + h * out_head_stride + (int64_t)row * D;
    const bool in_stripe = row < v.t_k && d_pad > 0;
    const uint8_t* r2 = v.k2 != nullptr ? v.k2 + h * v.k2_head_stride + (int64_t)row * sub2 : nullptr;
    const uint8_t* r4 = v.k4 != nullptr ? v.k4 + h * v.k4_head_stride + (int64_t)row * sub4 : nullptr;
    const uint8_t* r8 = v.k8 != nullptr ? v.k8 + h * v.k8_head_stride + (int64_t)row * n8p : nullptr;
    const uint16_t* sc = v.k_scale + (int64_t)h * d_pad;
    const uint16_t* zp = v.k_zp + (int64_t)h * d_pad;
    for (int c = lane; c < D; c += 32) {
      const int p = in_stripe ? s_slot[c] : -1;
      uint16_t out = 0;
      if (p >= 0) {
        unsigned code;
        if (p < n2p) code = (r2[p % sub2] >> (2 * (p / sub2))) & 3u;
        else if (p < n2p + n4p) { const int q = p - n2p; code = (r4[q % sub4] >> (4 * (q / sub4))) & 15u; }
        else code = r8[p - n2p - n4p];
        out = dequant_h(code, zp[p], sc[p]);
      }
      dst[c] = out;
    }
  }

  if (v_out != nullptr) {
    uint16_t* dst = v_out + h * out_head_stride + (int64_t)row * D;
    int n2 = v.n2, n4 = v.n4, n8 = v.n8;
    if (v.v_seg_bounds != nullptr) { n2 = v.v_seg_bounds[h * 3 + 0]; n4 = v.v_seg_bounds[h * 3 + 1]; n8 = v.v_seg_bounds[h * 3 + 2]; }
    const int t_v = n2 + n4 + n8;
    const int n16 = v.v16 == nullptr ? 0 : (v.n_v16 != nullptr ? v.n_v16[h] : v.n_v16_shared);
    if (row < t_v) {
      const int seg = row < n2 ? 0 : row < n2 + n4 ? 1 : 2;
      const int j = seg == 0 ? row : seg == 1 ? row - n2 : row - n2 - n4;
      const int sub = seg == 0 ? D / 4 : seg == 1 ? D / 2 : D;
      const uint8_t* src = seg == 0 ? v.v2 + h * v.v2_head_stride : seg == 1 ? v.v4 + h * v.v4_head_stride
                                                                             : v.v8 + h * v.v8_head_stride;
      src += (int64_t)j * sub;
      const uint16_t s = v.v_scale[h * v.v_meta_head_stride + row], z = v.v_zp[h * v.v_meta_head_stride + row];
      const int bits = seg == 0 ? 2 : seg == 1 ? 4 : 8;
      const unsigned mask = (1u << bits) - 1u;
      for (int c = lane; c < D; c += 32) {
        const unsigned code = (src[c % sub] >> (bits * (c / sub))) & mask;
        dst[c] = dequant_h(code, z, s);
      }
    } else if (row >= v.max_t_v && row < v.max_t_v + n16) {
      const uint16_t* src = v.v16 + h * v.v16_head_stride + (int64_t)(row - v.max_t_v) * D;
      for (int c = lane; c < D; c += 32) dst[c] = src[c];
    } else {
      for (int c = lane; c < D; c += 32) dst[c] = 0;
    }
  }
}

// ── 128 channels: all layers of a cache in one launch ────────────────────────
// Bound by HBM (every row costs 512 bytes of result against about 150 packed bytes).  A warp per row
// with one channel per lane and step (the general kernel above) moved 2-byte elements and spent 20
// instructions on each, two launches per layer; here:
//   * half a warp takes a row, eight neighbouring channels per lane, so that every store is 16 bytes;
//   * V: the eight codes of a lane are the same eight bytes' bits whatever the row (quarter- and
//     half-split rows), so they are one 8-byte load and two shifts;
//   * K: a CTA brings the rows' bytes (three contiguous ranges) into shared memory with whole words;
//     where a channel lies in a row (byte, shift, mask, scale, zero point) is worked out once per CTA,
//     by one thread each, and a lane keeps its eight channels' in registers;
//   * grid = (row blocks, heads, layers), K and V of a block by the same CTA; the layers' records
//     travel as launch arguments.
// 16 layers x 8 heads x 1792 rows of odd widths (165 MB): 344 us in 32 launches -> 59.5 us in one (2.8 TB/s);
// 64 rows per CTA and a lane working its channels out by itself: 117 us.
constexpr int UP_THREADS = 256;
constexpr int UP_ROWS = 128;                                 // stripe rows per CTA
constexpr int UP_JOBS = 16;                                  // layers per launch (their records are launch arguments)
struct UnpackJobs { rdkv_unpack_job j[UP_JOBS]; };
constexpr int UP_STATIC_SMEM = 128 * (2 + 4 * 4);            // s_slot, s_where, s_how, s_sc, s_zp of the kernel

// float(code) without a conversion instruction: the code in the mantissa of 2^23, exact.
__device__ __forceinline__ float code_f(uint32_t bits) { return __uint_as_float(0x4B000000u | bits) - 8388608.f; }
__device__ __forceinline__ uint32_t dequant_h2(uint32_t c0, uint32_t c1, float z0, float z1, float s0, float s1) {
  const float a = __fmul_rn(__fsub_rn(code_f(c0), z0), s0), b = __fmul_rn(__fsub_rn(code_f(c1), z1), s1);
  return (uint32_t)__half_as_ushort(__float2half_rn(a)) | (uint32_t)__half_as_ushort(__float2half_rn(b)) << 16;
}

// Bytes [src, src + n) to shared memory at dst + (src & 15), whole 16-byte blocks where they lie inside the range.
__device__ __forceinline__ void stage_bytes_of(unsigned char* dst, const uint8_t* src, int n) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(src);
  const int lead = (int)(a & 15), total = lead + n;
  for (int b = threadIdx.x; b * 16 < total; b += UP_THREADS) {
    const int lo = b * 16, hi = min(lo + 16, total);
    if (lo >= lead && lo + 16 <= total) {
      *reinterpret_cast<uint4*>(dst + lo) = __ldg(reinterpret_cast<const uint4*>(src - lead + lo));
    } else {
      for (int x = max(lo, lead); x < hi; ++x) dst[x] = __ldg(src - lead + x);
    }
  }
}

__global__ void __launch_bounds__(UP_THREADS)
unpack_layers128_kernel(const __grid_constant__ UnpackJobs jobs) {
  extern __shared__ __align__(16) unsigned char up_smem[];
  __shared__ int16_t s_slot[128];
  __shared__ __align__(16) uint32_t s_where[128];                        // a channel's shared-memory address in row 0
  __shared__ __align__(16) uint32_t s_how[128];                          // bytes per row | shift << 16 | mask << 24 (0: evicted)
  __shared__ __align__(16) float s_sc[128], s_zp[128];
  const rdkv_unpack_job& J = jobs.j[blockIdx.z];
  const rdkv_layer_view& v = J.view;
  const int h = blockIdx.y, row0 = blockIdx.x * UP_ROWS;
  if (h >= J.H_kv || row0 >= J.rows_out) return;
  const int n_rows = min(UP_ROWS, J.rows_out - row0);
  const int tid = threadIdx.x, half_id = tid >> 4, l = tid & 15;       // row within a step, lane within the row
  constexpr int STEP = UP_THREADS / 16;

  if (J.k_out != nullptr) {
    const int n2p = v.n_ch2_pad, n4p = v.n_ch4_pad, n8p = v.n_ch8;
    const int sub2 = n2p / 4, sub4 = n4p / 2;
    const int in_rows = max(0, min(n_rows, v.t_k - row0));             // rows of this block that the stripe holds
    // areas of the three streams, 16-byte aligned; a stream keeps its offset within a 16-byte block
    unsigned char* a2 = up_smem;
    unsigned char* a4 = a2 + ((UP_ROWS * sub2 + 31) & ~15);
    unsigned char* a8 = a4 + ((UP_ROWS * sub4 + 31) & ~15);
    const uint8_t* g2 = v.k2 + h * v.k2_head_stride + (int64_t)row0 * sub2;
    const uint8_t* g4 = v.k4 + h * v.k4_head_stride + (int64_t)row0 * sub4;
    const uint8_t* g8 = v.k8 + h * v.k8_head_stride + (int64_t)row0 * n8p;
    if (sub2 > 0 && in_rows > 0) stage_bytes_of(a2, g2, in_rows * sub2);
    if (sub4 > 0 && in_rows > 0) stage_bytes_of(a4, g4, in_rows * sub4);
    if (n8p > 0 && in_rows > 0) stage_bytes_of(a8, g8, in_rows * n8p);
    if (tid < 128) s_slot[tid] = -1;
    __syncthreads();
    {
      int c2 = J.n_ch2, c4 = J.n_ch4, c8 = J.n_ch8;
      if (J.k_ch_counts != nullptr) { c2 = J.k_ch_counts[h * 3]; c4 = J.k_ch_counts[h * 3 + 1]; c8 = J.k_ch_counts[h * 3 + 2]; }
      const int64_t* si = J.k_sort_idx + h * J.k_sort_idx_head_stride;
      for (int k = tid; k < c2 + c4 + c8; k += UP_THREADS) {
        const int slot = k < c2 ? k : k < c2 + c4 ? n2p + (k - c2) : n2p + n4p + (k - c2 - c4);
        const int64_t ch = si[k];
        if (ch >= 0 && ch < 128) s_slot[ch] = (int16_t)slot;
      }
    }
    __syncthreads();
    const int d_pad = n2p + n4p + n8p;
    if (tid < 128) {
      const int p = s_slot[tid];
      uint32_t where = (uint32_t)__cvta_generic_to_shared(up_smem), how = 0u;
      float sc = 0.f, zp = 0.f;
      if (p >= 0 && p < d_pad) {
        if (p < n2p) {
          where = (uint32_t)__cvta_generic_to_shared(a2) + (uint32_t)(reinterpret_cast<uintptr_t>(g2) & 15) + p % sub2;
          how = (uint32_t)sub2 | (uint32_t)(2 * (p / sub2)) << 16 | 3u << 24;
        } else if (p < n2p + n4p) {
          const int x = p - n2p;
          where = (uint32_t)__cvta_generic_to_shared(a4) + (uint32_t)(reinterpret_cast<uintptr_t>(g4) & 15) + x % sub4;
          how = (uint32_t)sub4 | (uint32_t)(4 * (x / sub4)) << 16 | 15u << 24;
        } else {
          where = (uint32_t)__cvta_generic_to_shared(a8) + (uint32_t)(reinterpret_cast<uintptr_t>(g8) & 15) + (p - n2p - n4p);
          how = (uint32_t)n8p | 255u << 24;
        }
        sc = h2f(v.k_scale[(int64_t)h * d_pad + p]);
        zp = h2f(v.k_zp[(int64_t)h * d_pad + p]);
      }
      s_where[tid] = where; s_how[tid] = how; s_sc[tid] = sc; s_zp[tid] = zp;
    }
    __syncthreads();
    uint32_t addr[8], step[8], shift[8], mask[8];
    float sc[8], zp[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const uint32_t how = s_how[8 * l + e];
      step[e] = how & 0xFFFFu; shift[e] = (how >> 16) & 0xFFu; mask[e] = how >> 24;
      addr[e] = s_where[8 * l + e] + half_id * step[e]; step[e] *= STEP;
      sc[e] = s_sc[8 * l + e]; zp[e] = s_zp[8 * l + e];
    }
    uint16_t* dst = J.k_out + h * J.out_head_stride + (int64_t)row0 * 128 + 8 * l;
#pragma unroll 2
    for (int k = half_id; k < n_rows; k += STEP) {
      uint4 w = make_uint4(0u, 0u, 0u, 0u);
      if (k < in_rows) {
        uint32_t c[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          uint32_t byte;
          asm volatile("ld.shared.u8 %0, [%1];" : "=r"(byte) : "r"(addr[e]));
          addr[e] += step[e];
          c[e] = (byte >> shift[e]) & mask[e];
        }
        w.x = dequant_h2(c[0], c[1], zp[0], zp[1], sc[0], sc[1]); w.y = dequant_h2(c[2], c[3], zp[2], zp[3], sc[2], sc[3]);
        w.z = dequant_h2(c[4], c[5], zp[4], zp[5], sc[4], sc[5]); w.w = dequant_h2(c[6], c[7], zp[6], zp[7], sc[6], sc[7]);
      }
      *reinterpret_cast<uint4*>(dst + (int64_t)k * 128) = w;
    }
  }

  if (J.v_out != nullptr) {
    int n2 = v.n2, n4 = v.n4, n8 = v.n8;
    if (v.v_seg_bounds != nullptr) { n2 = v.v_seg_bounds[h * 3]; n4 = v.v_seg_bounds[h * 3 + 1]; n8 = v.v_seg_bounds[h * 3 + 2]; }
    const int t_v = n2 + n4 + n8;
    const int n16 = v.v16 == nullptr ? 0 : (v.n_v16 != nullptr ? v.n_v16[h] : v.n_v16_shared);
    const uint8_t* p2 = v.v2 + h * v.v2_head_stride + (8 * l & 31);
    const uint8_t* p4 = v.v4 + h * v.v4_head_stride + (8 * l & 63);
    const uint8_t* p8 = v.v8 + h * v.v8_head_stride + 8 * l;
    const uint16_t* p16 = v.v16 + h * v.v16_head_stride + 8 * l;
    uint16_t* dst = J.v_out + h * J.out_head_stride + (int64_t)row0 * 128 + 8 * l;
#pragma unroll 2
    for (int k = half_id; k < n_rows; k += STEP) {
      const int row = row0 + k;
      uint4 w = make_uint4(0u, 0u, 0u, 0u);
      if (row < t_v) {
        const uint8_t* src;
        uint32_t sh, mk;
        if (row < n2) { src = p2 + (int64_t)row * 32; sh = 2 * (l >> 2); mk = 3u; }
        else if (row < n2 + n4) { src = p4 + (int64_t)(row - n2) * 64; sh = 4 * (l >> 3); mk = 15u; }
        else { src = p8 + (int64_t)(row - n2 - n4) * 128; sh = 0u; mk = 255u; }
        const uint2 b = __ldg(reinterpret_cast<const uint2*>(src));
        const float s = h2f(v.v_scale[h * v.v_meta_head_stride + row]), z = h2f(v.v_zp[h * v.v_meta_head_stride + row]);
        const uint32_t x = b.x >> sh, y = b.y >> sh;
        w.x = dequant_h2(x & mk, (x >> 8) & mk, z, z, s, s); w.y = dequant_h2((x >> 16) & mk, (x >> 24) & mk, z, z, s, s);
        w.z = dequant_h2(y & mk, (y >> 8) & mk, z, z, s, s); w.w = dequant_h2((y >> 16) & mk, (y >> 24) & mk, z, z, s, s);
      } else if (row >= v.max_t_v && row < v.max_t_v + n16) {
        w = __ldg(reinterpret_cast<const uint4*>(p16 + (int64_t)(row - v.max_t_v) * 128));
      }
      *reinterpret_cast<uint4*>(dst + (int64_t)k * 128) = w;
    }
  }
}

}  // namespace rdkv

using namespace rdkv;

static int check_unpack_job(const rdkv_unpack_job& J, int D) {
  const rdkv_layer_view& view = J.view;
  if (J.H_kv <= 0 || J.rows_out < 0 || (J.k_out == nullptr && J.v_out == nullptr)) return RDKV_ERR_BAD_ARG;
  if (J.k_out != nullptr) {
    const int d_pad = view.n_ch2_pad + view.n_ch4_pad + view.n_ch8;
    if (d_pad > 0 && (view.k_scale == nullptr || view.k_zp == nullptr || J.k_sort_idx == nullptr)) return RDKV_ERR_BAD_ARG;
    if ((view.n_ch2_pad > 0 && view.k2 == nullptr) || (view.n_ch4_pad > 0 && view.k4 == nullptr) ||
        (view.n_ch8 > 0 && view.k8 == nullptr))
      return RDKV_ERR_BAD_ARG;
    if (J.n_ch2 < 0 || J.n_ch4 < 0 || J.n_ch8 < 0 || J.n_ch2 > view.n_ch2_pad || J.n_ch4 > view.n_ch4_pad ||
        J.n_ch8 > view.n_ch8)
      return RDKV_ERR_BAD_ARG;
  }
  if (J.H_kv > 65535) return RDKV_ERR_TOO_LARGE;
  return RDKV_OK;
}

static size_t unpack_smem(const rdkv_layer_view& v) {
  return (size_t)((UP_ROWS * (v.n_ch2_pad / 4) + 31) & ~15) + ((UP_ROWS * (v.n_ch4_pad / 2) + 31) & ~15) +
         ((UP_ROWS * v.n_ch8 + 31) & ~15) + 16;
}

// The 128-channel kernel moves 8-byte words of V codes and 16-byte words of fp16 rows: bases and head
// strides on those boundaries (what this library packs always is), and K rows that fit its shared memory beside
// its tables within the 48 KB every launch may have (365 bytes a row; 128 channels take 224 at most, but a layer
// packed for larger channel targets can be wider).
static bool unpack_fast(const rdkv_unpack_job& J, int D) {
  const rdkv_layer_view& v = J.view;
  auto al = [](const void* p, int64_t stride_bytes, int a) { return ((reinterpret_cast<uintptr_t>(p) | (uintptr_t)stride_bytes) & (a - 1)) == 0; };
  return D == 128 && al(J.k_out, 2 * J.out_head_stride, 16) && al(J.v_out, 2 * J.out_head_stride, 16) &&
         al(v.v2, v.v2_head_stride, 8) && al(v.v4, v.v4_head_stride, 8) && al(v.v8, v.v8_head_stride, 8) &&
         al(v.v16, 2 * v.v16_head_stride, 16) && (J.k_out == nullptr || unpack_smem(v) + UP_STATIC_SMEM <= 48 * 1024);
}

extern "C" int rdkv_sizeof_unpack_job(void) { return (int)sizeof(rdkv_unpack_job); }

extern "C" int rdkv_unpack_layers(const rdkv_unpack_job* jobs, int n_jobs, int D, void* stream) {
  if (jobs == nullptr || n_jobs < 0 || D <= 0) return RDKV_ERR_BAD_ARG;
  if (D > UNPACK_MAX_D || (D & 3)) return RDKV_ERR_BAD_SHAPE;
  for (int i = 0; i < n_jobs; ++i) {
    const int rc = check_unpack_job(jobs[i], D);
    if (rc != RDKV_OK) return rc;
  }
  cudaStream_t st = (cudaStream_t)stream;
  UnpackJobs batch;
  int n = 0, blocks = 0, heads = 0;
  size_t smem = 0;
  auto flush = [&]() {
    if (n == 0) return (int)RDKV_OK;
    unpack_layers128_kernel<<<dim3(blocks, heads, n), UP_THREADS, smem, st>>>(batch);
    n = blocks = heads = 0; smem = 0;
    return launch_status();
  };
  for (int i = 0; i < n_jobs; ++i) {
    const rdkv_unpack_job& J = jobs[i];
    if (J.rows_out == 0) continue;
    if (unpack_fast(J, D)) {
      batch.j[n++] = J;
      blocks = max(blocks, (J.rows_out + UP_ROWS - 1) / UP_ROWS);
      heads = max(heads, J.H_kv);
      if (J.k_out != nullptr) smem = max(smem, unpack_smem(J.view));
      if (n == UP_JOBS) { const int rc = flush(); if (rc != RDKV_OK) return rc; }
    } else {
      unpack_layer_kernel<<<dim3((J.rows_out + UNPACK_WARPS - 1) / UNPACK_WARPS, J.H_kv), UNPACK_WARPS * 32, 0, st>>>(
          J.view, D, J.k_sort_idx, J.k_sort_idx_head_stride, J.k_ch_counts, J.n_ch2, J.n_ch4, J.n_ch8, J.k_out, J.v_out,
          J.out_head_stride, J.rows_out);
      const int rc = launch_status();
      if (rc != RDKV_OK) return rc;
    }
  }
  return flush();
}

extern "C" int rdkv_unpack_layer(const rdkv_layer_view* view, int H_kv, int D, const int64_t* k_sort_idx,
                                 int64_t k_sort_idx_head_stride, const int32_t* k_ch_counts, int n_ch2, int n_ch4,
                                 int n_ch8, uint16_t* k_out, uint16_t* v_out, int64_t out_head_stride, int rows_out,
                                 void* stream) {
  if (view == nullptr || H_kv <= 0 || D <= 0 || rows_out < 0 || (k_out == nullptr && v_out == nullptr))
    return RDKV_ERR_BAD_ARG;
  rdkv_unpack_job J;
  J.view = *view; J.k_sort_idx = k_sort_idx; J.k_sort_idx_head_stride = k_sort_idx_head_stride; J.k_ch_counts = k_ch_counts;
  J.n_ch2 = n_ch2; J.n_ch4 = n_ch4; J.n_ch8 = n_ch8; J.H_kv = H_kv;
  J.k_out = k_out; J.v_out = v_out; J.out_head_stride = out_head_stride; J.rows_out = rows_out; J.reserved = 0;
  return rdkv_unpack_layers(&J, 1, D, stream);
}
