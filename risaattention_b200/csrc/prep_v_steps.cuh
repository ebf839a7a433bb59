// The range step and the (tiled) code step of the V quantiser as CTA bodies, shared by their
// stand-alone kernels (prep_v.cu) and by the launches that run them next to the Q / K quantisers
// (prep_qk.cu).  Reference: csrc/kernels/quantize_v_impl.cuh:83-292.
#pragma once
#include "common.cuh"
#include <cfloat>
#include <type_traits>

namespace risa_b200 {

constexpr int kRangeChunk = 512;   // tokens per range CTA
constexpr int kRangeThreads = 256;

// What the range step of one risa_b200_quantize_v call reads and writes.
struct VRangeJob {
  const void* v;
  float2* ranges;  // [B*Hkv][chunks][head_dim] (min, max)
  int k_len, head_dim, kv_heads, batch, chunks;
  int64_t stride_b, stride_h, stride_n;
  const int32_t* perm;
  int in_dim;  // channels the input has; channels from here to head_dim are zeros (a multiple of 4)
};

// Eight channels of a row, of which the input has `have` (channels it lacks are zeros).
template <typename T>
__device__ __forceinline__ void load8(const T* p, float* v, int have) {
#pragma unroll
  for (int i = 0; i < 8; i += 4) {
    if (have > i) Load4<T>::load(p + i, v + i);
    else v[i] = v[i + 1] = v[i + 2] = v[i + 3] = 0.0f;
  }
}

// One CTA of 256 threads = one 512-token chunk of one (batch, kv head): thread = (token lane,
// 8-channel group).
template <typename T>
__device__ __forceinline__ void v_range_block(const VRangeJob& job, int chunk, int h, int b) {
  __shared__ float s_mn[256][9], s_mx[256][9];
  const int head_dim = job.head_dim, k_len = job.k_len;
  const int groups = head_dim / 8;            // 8, 16 or 32 threads per token row
  const int tokens_per_step = 256 / groups;
  const int g = threadIdx.x % groups, tl = threadIdx.x / groups;
  const int64_t bh = static_cast<int64_t>(b) * job.kv_heads + h;
  const T* in = static_cast<const T*>(job.v) + b * job.stride_b + h * job.stride_h + g * 8;
  const int32_t* row_map = job.perm ? job.perm + bh * k_len : nullptr;
  float mn[8], mx[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    mn[i] = FLT_MAX;
    mx[i] = -FLT_MAX;
  }
  const int begin = chunk * kRangeChunk;
  const int end = min(k_len, begin + kRangeChunk);
  for (int n = begin + tl; n < end; n += tokens_per_step) {
    float t[8];
    const int64_t src = row_map ? __ldg(row_map + n) : n;
    load8(in + src * job.stride_n, t, job.in_dim - 8 * g);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      mn[i] = fminf(mn[i], t[i]);
      mx[i] = fmaxf(mx[i], t[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    s_mn[threadIdx.x][i] = mn[i];
    s_mx[threadIdx.x][i] = mx[i];
  }
  __syncthreads();
  if (threadIdx.x < head_dim) {
    const int c = threadIdx.x, cg = c / 8, ci = c % 8;
    float lo = FLT_MAX, hi = -FLT_MAX;
    for (int t = 0; t < tokens_per_step; ++t) {
      lo = fminf(lo, s_mn[t * groups + cg][ci]);
      hi = fmaxf(hi, s_mx[t * groups + cg][ci]);
    }
    job.ranges[(bh * job.chunks + chunk) * head_dim + c] = make_float2(lo, hi);
  }
}

__device__ __forceinline__ int storage_position(int token) {
  // token bits {b3,b2,b1,b0} -> storage bits {b2,b0,b3,b1}: order 0,1,8,9,2,3,10,11,...
  const int w = token & 15;
  return (token & ~15) | (w & 1) | (((w >> 3) & 1) << 1) | (((w >> 1) & 1) << 2) |
         (((w >> 2) & 1) << 3);
}

// The code step, for head dims of whole 64-channel blocks: a warp takes windows of 32 tokens x 16
// channels, a lane the four tokens of one storage word (2w, 2w+1, 2w+8, 2w+9 of a 16-token group) x
// four channels.  The four code words of a lane -- one per channel -- are exchanged between the four
// lanes of a group with two shuffle steps, after which a lane holds the whole 16-byte storage group
// of one channel; neighbouring groups of a channel leave in the same store.  No shared memory and no
// barrier per window, and key lengths need not be multiples of anything: missing tokens give code 0.
// Rows are whole 16-token storage groups, not whole windows: each group's store has its own bound.
//   absmax: a CTA walks `steps` pieces of 128 tokens x 64 channels, up to four in flight per lane.
//   midpoint-affine: the residuals have an order of their own (slot t of `slots` sums tokens Lk-1-t,
//   Lk-1-t-slots, ...), so a lane keeps four residue classes of tokens modulo `slots` -- a class is
//   one slot -- and walks them from the last token down.
constexpr int kVChannels = 64, kVThreads = 512, kVPiece = 128;  // kVPiece: tokens of four windows

// What the code step of one risa_b200_quantize_v call reads and writes.
struct VCodesJob {
  const void* v;
  int8_t* out;
  float* scale_out;
  float* center_out;
  const float2* ranges;
  float* residuals;
  int k_len, padded_len, kv_heads, head_dim, batch, chunks, slots;
  int64_t stride_b, stride_h, stride_n;
  const int32_t* perm;
  int midpoint_affine;
  int in_dim;        // as in VRangeJob
  int steps, parts;  // 128-token pieces per CTA; CTAs per 64-channel block
};

// Four channels of a row as they are in memory, converted when they are used.
template <typename T> struct Raw4 {
  uint2 raw;
  __device__ __forceinline__ void load(const T* p) { raw = __ldg(reinterpret_cast<const uint2*>(p)); }
  __device__ __forceinline__ void get(float (&x)[4]) const {
    if constexpr (sizeof(T) == 2) {
      const uint32_t w[2] = {raw.x, raw.y};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if constexpr (std::is_same<T, __half>::value) {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
          x[2 * i] = f.x;
          x[2 * i + 1] = f.y;
        } else {
          x[2 * i] = __uint_as_float(w[i] << 16);
          x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
      }
    }
  }
};
template <> struct Raw4<float> {
  float4 raw;
  __device__ __forceinline__ void load(const float* p) {
    raw = __ldg(reinterpret_cast<const float4*>(p));
  }
  __device__ __forceinline__ void get(float (&x)[4]) const {
    x[0] = raw.x;
    x[1] = raw.y;
    x[2] = raw.z;
    x[3] = raw.w;
  }
};

// words[c] of lane w (of four neighbouring lanes) <-> word w of channel c: a 4 x 4 transposition.
__device__ __forceinline__ void transpose_words(uint32_t (&words)[4], int lane) {
  const bool odd = lane & 1, upper = lane & 2;
  const uint32_t a = __shfl_xor_sync(0xffffffffu, odd ? words[0] : words[1], 1);
  const uint32_t b = __shfl_xor_sync(0xffffffffu, odd ? words[2] : words[3], 1);
  if (odd) {
    words[0] = a;
    words[2] = b;
  } else {
    words[1] = a;
    words[3] = b;
  }
  const uint32_t c = __shfl_xor_sync(0xffffffffu, upper ? words[0] : words[2], 2);
  const uint32_t d = __shfl_xor_sync(0xffffffffu, upper ? words[1] : words[3], 2);
  if (upper) {
    words[0] = c;
    words[1] = d;
  } else {
    words[2] = c;
    words[3] = d;
  }
}

// CTA `part` of 64-channel block `by`, 512 threads.
template <typename T, bool AFFINE>
__device__ __forceinline__ void v_codes_block(const VCodesJob& job, int part, int by) {
  const int k_len = job.k_len, padded_len = job.padded_len, head_dim = job.head_dim;
  const int chunks = job.chunks, slots = job.slots;
  __shared__ float s_inv[kVChannels], s_center[kVChannels];
  const int d_tiles = head_dim / kVChannels;
  const int bh = by / d_tiles, d0 = (by % d_tiles) * kVChannels;
  const int h = bh % job.kv_heads, b = bh / job.kv_heads;
  const int64_t out_row = static_cast<int64_t>(bh) * head_dim + d0;

  // channel range = min / max over the per-chunk partials: spread over the whole CTA (eight chunk
  // subsets per channel) so that the loads overlap instead of forming one long dependent loop
  __shared__ float s_lo[kVThreads / kVChannels][kVChannels];
  __shared__ float s_hi[kVThreads / kVChannels][kVChannels];
  {
    const int channel = threadIdx.x % kVChannels, subset = threadIdx.x / kVChannels;
    float lo = FLT_MAX, hi = -FLT_MAX;
    const float2* r = job.ranges + static_cast<int64_t>(bh) * chunks * head_dim + d0 + channel;
    for (int c = subset; c < chunks; c += kVThreads / kVChannels) {
      const float2 x = __ldg(r + static_cast<int64_t>(c) * head_dim);
      lo = fminf(lo, x.x);
      hi = fmaxf(hi, x.y);
    }
    s_lo[subset][channel] = lo;
    s_hi[subset][channel] = hi;
  }
  __syncthreads();
  if (threadIdx.x < kVChannels) {
    float lo = FLT_MAX, hi = -FLT_MAX;
#pragma unroll
    for (int subset = 0; subset < kVThreads / kVChannels; ++subset) {
      lo = fminf(lo, s_lo[subset][threadIdx.x]);
      hi = fmaxf(hi, s_hi[subset][threadIdx.x]);
    }
    float center, radius;
    if constexpr (AFFINE) {
      center = 0.5f * (lo + hi);
      radius = 0.5f * (hi - lo);
    } else {
      center = 0.0f;
      radius = fmaxf(fabsf(lo), fabsf(hi));
    }
    const float sc = fmaxf(radius * (1.f / 127.f), 1e-12f);
    s_inv[threadIdx.x] = 1.f / sc;
    s_center[threadIdx.x] = center;
    if (part == 0) {
      job.scale_out[out_row + threadIdx.x] = sc;
      if constexpr (!AFFINE) job.center_out[out_row + threadIdx.x] = 0.0f;
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int word = lane & 3, group = (lane >> 2) & 1;          // of the window's two storage groups
  const int ch0 = (warp & 3) * 16 + (lane >> 3) * 4;           // the lane's four channels
  const int first_token = 16 * group + 2 * word;               // of the window: +0, +1, +8, +9
  float inv[4], center[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    inv[c] = s_inv[ch0 + c];
    center[c] = s_center[ch0 + c];
  }
  const bool present = d0 + ch0 < job.in_dim;
  const T* in = static_cast<const T*>(job.v) + b * job.stride_b + h * job.stride_h + d0 + ch0;
  const int32_t* row_map = job.perm ? job.perm + static_cast<int64_t>(bh) * k_len : nullptr;
  // after the exchange the lane stores channel ch0 + word of its group
  int8_t* out = job.out + (out_row + ch0 + word) * padded_len + 16 * group;
  auto load_tokens = [&](int base, int limit, Raw4<T> (&t)[4], bool (&have)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int token = base + first_token + (j & 1) + 8 * (j >> 1);
      have[j] = token < limit && present;
      if (have[j]) {
        const int64_t row = row_map ? __ldg(row_map + token) : token;
        t[j].load(in + row * job.stride_n);
      }
    }
  };
  if constexpr (!AFFINE) {
    constexpr int U = sizeof(T) == 2 ? 4 : 2;  // windows in flight
    const int end = min(padded_len, (part + 1) * job.steps * kVPiece);
    for (int base0 = part * job.steps * kVPiece + (warp >> 2) * 32; base0 < end;
         base0 += U * kVPiece) {
      Raw4<T> t[U][4];
      bool have[U][4];
#pragma unroll
      for (int u = 0; u < U; ++u)
        load_tokens(base0 + kVPiece * u, min(k_len, end), t[u], have[u]);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float x[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          t[u][j].get(x[j]);
#pragma unroll
          for (int c = 0; c < 4; ++c) x[j][c] = have[u][j] ? x[j][c] * inv[c] : 0.0f;
        }
        uint32_t words[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) words[c] = pack4_s8(x[0][c], x[1][c], x[2][c], x[3][c]);
        transpose_words(words, lane);
        if (base0 + kVPiece * u + 16 * group < end)
          *reinterpret_cast<uint4*>(out + base0 + kVPiece * u) =
              make_uint4(words[0], words[1], words[2], words[3]);
      }
    }
  } else {
    const int residue = (part * 4 + (warp >> 2)) * 32;  // first class of this warp's window
    float residual[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) residual[j][c] = 0.0f;
    const int top = (padded_len - 1) / slots * slots + residue;
#pragma unroll 2
    for (int base = top; base >= 0; base -= slots) {
      Raw4<T> t[4];
      bool have[4];
      load_tokens(base, k_len, t, have);
      uint32_t code[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float x[4];
        t[j].get(x);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          // (a channel the input lacks has centre 0, so the centre stands for its zeros too)
          const float value = have[j] ? x[c] : center[c];
          const float normalized = (value - center[c]) * inv[c];
          code[j][c] = to_s8(normalized);
          residual[j][c] += normalized - static_cast<float>(static_cast<int8_t>(code[j][c]));
        }
      }
      uint32_t words[4];
#pragma unroll
      for (int c = 0; c < 4; ++c)
        words[c] = __byte_perm(__byte_perm(code[0][c], code[1][c], 0x0040),
                               __byte_perm(code[2][c], code[3][c], 0x0040), 0x5410);
      transpose_words(words, lane);
      if (base + 16 * group < padded_len)
        *reinterpret_cast<uint4*>(out + base) = make_uint4(words[0], words[1], words[2], words[3]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int token_class = residue + first_token + (j & 1) + 8 * (j >> 1);
      const int slot = ((k_len - 1 - token_class) % slots + slots) % slots;
#pragma unroll
      for (int c = 0; c < 4; ++c) job.residuals[(out_row + ch0 + c) * slots + slot] = residual[j][c];
    }
  }
}

// Host side of the V quantiser split into its steps (prep_v.cu): v_quantize_jobs() checks the
// arguments of a risa_b200_quantize_v call and describes its range step and -- for head dims
// of whole 64-channel blocks, else codes->v stays null -- its code step, launching nothing;
// quantize_v_after_range() launches what follows the range step, without the code step if that has
// been run by somebody else.
int v_quantize_jobs(const void* v, void* v_codes, float* v_scale, float* v_center, int batch,
                    int kv_heads, int k_len, int head_dim, int padded_len, int64_t stride_b,
                    int64_t stride_h, int64_t stride_n, int dtype_code, int midpoint_affine,
                    const int32_t* perm, void* workspace, size_t workspace_bytes, VRangeJob* range,
                    VCodesJob* codes, int in_dim = 0);
int quantize_v_after_range(const void* v, void* v_codes, float* v_scale, float* v_center, int batch,
                           int kv_heads, int k_len, int head_dim, int padded_len, int64_t stride_b,
                           int64_t stride_h, int64_t stride_n, int dtype_code, int midpoint_affine,
                           const int32_t* perm, void* workspace, bool codes_done, void* stream_ptr);
// Q and K quantisation (prep_qk.cu).  With a range job the V range step runs inside the first
// launch (next to the anchor detector and the Q quantiser); with a codes job the V code step runs
// inside the second (next to the K quantiser).
int quantize_qk_with_v_steps(const void* q, void* q_codes, float* q_scale, const void* k,
                             void* k_codes, float* k_scale, int batch, int q_heads, int q_len,
                             int kv_heads, int k_len, int head_dim, int cta_k, int64_t q_stride_b,
                             int64_t q_stride_h, int64_t q_stride_n, int64_t k_stride_b,
                             int64_t k_stride_h, int64_t k_stride_n, int dtype_code,
                             int32_t* anchors, const int32_t* q_perm, const int32_t* k_perm,
                             const VRangeJob* range_job, const VCodesJob* codes_job,
                             void* stream_ptr, int in_dim = 0);

}  // namespace risa_b200
