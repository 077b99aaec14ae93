// Load-time LiquidQuant weight quantiser on the device: fp16 / bf16 / fp32 weights [N, K] -> per-row scale,
// per-group step and offset, 4-bit codes, and (optionally) the tile blob the GEMM kernels read.  Bit-exact to the
// reference's PyTorch quantiser run on the CPU (liquidgemm/quant.py:61-100), which the reference executes as about
// fifteen elementwise / reduce launches plus five host reads for its assertions (:88-92), followed by a host-side
// gather for the prepack (liquidgemm/ops.py:118-150).
//
// Rows that a CTA can hold (aligned, up to 65536 elements; float32 32768) take quantise_rows_kernel, one pass over the
// weights: 28672 x 4096 bf16 481 -> 82 us, 4096 x 14336 273 -> 51 us against the two passes below, which serve the rest:
//   pass 1  row_amax_kernel      one warp per row: s1 = max(amax, 1e-12) / 119 (IEEE division)
//   pass 2  quantise_tiles_kernel one CTA per 128 x 128 tile of the weight matrix, thread = (row, 64-wide half):
//             q    = clamp(rint(w / s1[row]), -119, 119)                       (level 1, :70-72)
//             lo/hi over the group; step = clamp(ceil((hi - lo) / 15), 1, 16)  (level 2, :75-80)
//             code = clamp(rint((q - lo) / step), 0, 15); offset = 128 + lo    (:82-85)
//           and writes the tile of the blob (one contiguous 8704-byte block, see lq_elementwise.cu), the
//           [N, K/g] step / offset arrays and, on request, the [N, K] codes (one per byte).
// The overflow invariants the packed dequant relies on (step in 1..16, code * step + offset in 0..255) are
// checked on the device into the library's status word (site 501) instead of being read back by the host.
// Groups of 64 or 128 along K (the tile holds whole groups); K % 128 == 0.
#include <stdint.h>

#include "lq_common.cuh"

namespace lq {

int settle_blob(cudaStream_t st);   // lq_elementwise.cu

namespace quantw {

constexpr int kTileBytes = 8704;

// ---- one pass: a CTA per row, the row in registers ------------------------------------------------------------
// Thread t holds the 32-element units t, t + threads, ... (NV of them): the row is read once and the row scale needs
// one block reduction.  A unit is one 16-byte chunk of the blob, and a group of 64 (128) elements is the units of two
// (four) neighbouring lanes, so a group's range takes one (two) shuffles and its step is worked out once per 32 elements.
// Bound by instruction issue (the two IEEE divisions an element that this replaces, and the group arithmetic once per
// eight elements of a first version, were most of the time).

// 32 bytes in one load (32-byte aligned).
__device__ __forceinline__ void ldg_stream_v8(const void* p, uint4& a, uint4& b) {
  asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
               : "l"(p));
}

template <typename T, int NV>
__global__ void __launch_bounds__(NV * sizeof(T) >= 16 ? 256 : 512)
quantise_rows_kernel(const T* __restrict__ w, float* __restrict__ s1, uint8_t* __restrict__ s_u8,
                     uint8_t* __restrict__ offset_a, uint8_t* __restrict__ codes, uint8_t* __restrict__ blob,
                     int* __restrict__ status, int N, int K, int group) {
  __shared__ float red[32];
  constexpr int VU = 2 * sizeof(T);   // 16-byte vectors of a unit
  const int row = blockIdx.x;
  const int units = K >> 5;
  const int lane = threadIdx.x & 31;
  uint8_t* tile = blob + (size_t)(row >> 7) * (K >> 7) * kTileBytes;   // of k-tile 0
  const int r = row & 127;
  if (row >= N) {   // padding rows of the last tile: code 0, step 1, offset 128 reconstructs to 0
    for (int u = threadIdx.x; u < units; u += blockDim.x) {
      uint8_t* t = tile + (size_t)(u >> 2) * kTileBytes;
      *reinterpret_cast<uint4*>(t + ((u & 3) * 128 + r) * 16) = make_uint4(0u, 0u, 0u, 0u);
      if ((u & 1) == 0) *reinterpret_cast<uint16_t*>(t + 8192 + r * 4 + (u & 2)) = 0x8001;
    }
    return;
  }
  const T* src = w + (size_t)row * K;
  uint4 raw[NV][VU];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int u = threadIdx.x + i * blockDim.x;
#pragma unroll
    for (int v = 0; v < VU; v += 2) {
      raw[i][v] = raw[i][v + 1] = make_uint4(0u, 0u, 0u, 0u);
      if (u < units) ldg_stream_v8(src + (size_t)u * 32 + v * (32 / VU), raw[i][v], raw[i][v + 1]);
    }
  }
  RowMax<T> rm;
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int v = 0; v < VU; ++v) rm.take(raw[i][v]);
  const float amax = block_max(rm.value(), red);
  const float scale = __fdiv_rn(fmaxf(amax, 1e-12f), 119.0f);
  const float inv = __fdiv_rn(1.0f, scale);
  if (threadIdx.x == 0) s1[row] = scale;
  const float inv_of_lane = __fdiv_rn(1.0f, (float)max(lane, 1));   // 1 / step, fetched by shuffle
  constexpr int kMagicBits = 0x4B400000;                            // kRoundMagic
  const int lanes = group >> 5;                                     // units of a group
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int u = threadIdx.x + i * blockDim.x;
    // level 1: q = clamp(rint(w / s1), -119, 119), kept as kRoundMagic + q (|w| <= amax: the fast side needs no clamp)
    float2 t[4][4];
    float mx = kRoundMagic - 128.0f, mn = kRoundMagic + 128.0f;
#pragma unroll
    for (int o = 0; o < 4; ++o) {   // octets: one 32-bit word of the blob each
      float2 x[4];
#pragma unroll
      for (int v = 0; v < VU / 4; ++v) {
        float2 e[8 / sizeof(T)];
        vec_floats<T>(raw[i][o * (VU / 4) + v], e);
#pragma unroll
        for (int j = 0; j < 8 / (int)sizeof(T); ++j) x[v * (8 / sizeof(T)) + j] = e[j];
      }
      if (!round_quotients(x, inv, t[o])) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {   // one element, nearly always
          if (!near_integer(x[j].x, inv))
            t[o][j].x = kRoundMagic + (float)max(-119, min(119, __float2int_rn(__fdiv_rn(x[j].x, scale))));
          if (!near_integer(x[j].y, inv))
            t[o][j].y = kRoundMagic + (float)max(-119, min(119, __float2int_rn(__fdiv_rn(x[j].y, scale))));
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        mx = fmaxf(fmaxf(mx, t[o][j].x), t[o][j].y);
        mn = fminf(fminf(mn, t[o][j].x), t[o][j].y);
      }
    }
    // (max, -min) of the group as two 16-bit halves
    uint32_t pk = ((uint32_t)(__float_as_int(mx) - kMagicBits) & 0xffffu) |
                  ((uint32_t)(kMagicBits - __float_as_int(mn)) << 16);
    pk = __vmaxs2(pk, __shfl_xor_sync(0xffffffffu, pk, 1));
    if (group == 128) pk = __vmaxs2(pk, __shfl_xor_sync(0xffffffffu, pk, 2));
    const int neg_lo = (int)pk >> 16;
    const int range = (int)(short)(pk & 0xffffu) + neg_lo;
    const int step = max(1, (range + 14) / 15);   // ceil(range / 15): 0 <= range <= 238, so at most 16
    const int off = 128 - neg_lo;
    // level 2: code = rint((q - lo) / step).  The product with fl(1 / step) is within 15 * 2^-24 of the quotient, the
    // nearest quotient that is not a half-integer is 1/32 away from one, and adding 1.5 * 2^13 first rounds the
    // product to a multiple of 2^-10: half-integers come out exact and the second addition resolves them to even,
    // like the division would.  No clamp: (q - lo) / step <= range / ceil(range / 15) <= 15.
    const float inv_step = __shfl_sync(0xffffffffu, inv_of_lane, step);
    const float2 minus_lo = both((float)neg_lo - kRoundMagic);
    if (u >= units) continue;
    uint32_t words[4];   // byte b of word o = code[8 o + b] | code[8 o + 4 + b] << 4
    uint32_t bytes[8];
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      uint32_t c[8];   // kMagicBits + code
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 e = add2(fma2(add2(t[o][j], minus_lo), both(inv_step), both(12288.0f)), both(kRoundMagic - 12288.0f));
        c[2 * j] = __float_as_uint(e.x);
        c[2 * j + 1] = __float_as_uint(e.y);
      }
      bytes[2 * o] = __byte_perm(__byte_perm(c[0], c[1], 0x0040), __byte_perm(c[2], c[3], 0x0040), 0x5410);
      bytes[2 * o + 1] = __byte_perm(__byte_perm(c[4], c[5], 0x0040), __byte_perm(c[6], c[7], 0x0040), 0x5410);
      words[o] = bytes[2 * o] | (bytes[2 * o + 1] << 4);
    }
    if (blob) {
      uint8_t* tk = tile + (size_t)(u >> 2) * kTileBytes;
      *reinterpret_cast<uint4*>(tk + ((u & 3) * 128 + r) * 16) = make_uint4(words[0], words[1], words[2], words[3]);
      if ((u & 1) == 0) *reinterpret_cast<uint16_t*>(tk + 8192 + r * 4 + (u & 2)) = (uint16_t)(step | (off << 8));
    }
    if ((u & (lanes - 1)) == 0) {
      const size_t g = (size_t)row * (units / lanes) + u / lanes;
      s_u8[g] = (uint8_t)step;
      offset_a[g] = (uint8_t)off;
      // The packed dequant's invariant, once per group: code * step + offset grows with q, so its largest value
      // belongs to the group's largest q (and its smallest is the offset).
      const int top = __float2int_rn(__fmul_rn((float)range, inv_step));
      if (step > 16 || off < 0 || top * step + off > 255) atomicExch(status, 501);
    }
    if (codes) {
      uint4* dst = reinterpret_cast<uint4*>(codes + (size_t)row * K + (size_t)u * 32);
      dst[0] = make_uint4(bytes[0], bytes[1], bytes[2], bytes[3]);
      dst[1] = make_uint4(bytes[4], bytes[5], bytes[6], bytes[7]);
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) row_amax_kernel(const T* __restrict__ w, float* __restrict__ s1, int N, long K) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= N) return;
  const T* wr = w + (size_t)row * K;
  constexpr int VEC = 16 / sizeof(T);
  float amax = 0.f;
  if ((reinterpret_cast<uintptr_t>(wr) & 15) == 0 && K % VEC == 0) {
    for (long k = (long)lane * VEC; k < K; k += 32 * VEC) {
      const uint4 raw = ldg_stream_v4(wr + k);
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int i = 0; i < VEC; ++i) amax = fmaxf(amax, fabsf(to_f32<T>(e[i])));
    }
  } else {
    for (long k = lane; k < K; k += 32) amax = fmaxf(amax, fabsf(to_f32<T>(wr[k])));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (lane == 0) s1[row] = __fdiv_rn(fmaxf(amax, 1e-12f), 119.0f);
}

template <typename T>
__global__ void __launch_bounds__(256)
quantise_tiles_kernel(const T* __restrict__ w, const float* __restrict__ s1, uint8_t* __restrict__ s_u8,
                      uint8_t* __restrict__ offset_a, uint8_t* __restrict__ codes, uint8_t* __restrict__ blob,
                      int* __restrict__ status, int N, long K, int group) {
  __shared__ int lohi[2][128][2];
  const int kt = blockIdx.x, nt = blockIdx.y;
  const int KT = (int)(K >> 7);
  const int r = threadIdx.x & 127, h = threadIdx.x >> 7;
  const long n = (long)nt * 128 + r;
  const bool live = n < N;
  const long k0 = (long)kt * 128 + 64 * h;

  int q[64];
  int lo = 127, hi = -127;
  if (live) {
    const float scale = s1[n];
    const T* src = w + (size_t)n * K + k0;
    constexpr int VEC = 16 / sizeof(T);
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll
      for (int v = 0; v < 64 / VEC; ++v) {
        const uint4 raw = ldg_stream_v4(src + v * VEC);
        const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          const int val = max(-119, min(119, __float2int_rn(__fdiv_rn(to_f32<T>(e[i]), scale))));
          q[v * VEC + i] = val;
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < 64; ++i) q[i] = max(-119, min(119, __float2int_rn(__fdiv_rn(to_f32<T>(src[i]), scale))));
    }
#pragma unroll
    for (int i = 0; i < 64; ++i) {
      lo = min(lo, q[i]);
      hi = max(hi, q[i]);
    }
  }
  if (group == 128) {   // the two halves of a row form one group
    lohi[h][r][0] = lo;
    lohi[h][r][1] = hi;
    __syncthreads();
    lo = min(lo, lohi[h ^ 1][r][0]);
    hi = max(hi, lohi[h ^ 1][r][1]);
  }
  int step = 1, off = 128;   // padding rows: code 0, step 1, offset 128 reconstructs to 0
  if (live) {
    step = max(1, min(16, (hi - lo + 14) / 15));   // ceil((hi - lo) / 15): exact in integers for 0 <= hi - lo <= 238
    off = 128 + lo;
  }
  const float fstep = (float)step;
  uint32_t words[8];   // word j: octet k = 8j .. 8j+7 of this half, byte b = code[8j+b] | code[8j+4+b] << 4
  bool bad = false;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    uint32_t wv = 0;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      int c = 0;
      if (live) {
        c = max(0, min(15, __float2int_rn(__fdiv_rn((float)(q[8 * j + b] - lo), fstep))));
        const int u = c * step + off;
        bad |= (u < 0) | (u > 255);
        q[8 * j + b] = c;
      }
      wv |= (uint32_t)c << (8 * (b & 3) + 4 * (b >> 2));
    }
    words[j] = wv;
  }
  if (bad || step < 1 || step > 16) atomicExch(status, 501);

  if (blob) {
    uint8_t* tile = blob + ((size_t)nt * KT + kt) * kTileBytes;
    *reinterpret_cast<uint4*>(tile + ((2 * h) * 128 + r) * 16) = make_uint4(words[0], words[1], words[2], words[3]);
    *reinterpret_cast<uint4*>(tile + ((2 * h + 1) * 128 + r) * 16) = make_uint4(words[4], words[5], words[6], words[7]);
    *reinterpret_cast<uint16_t*>(tile + 8192 + r * 4 + 2 * h) = (uint16_t)(step | (off << 8));
  }
  if (live) {
    const long G = K / group;
    if (group == 64) {
      s_u8[n * G + 2 * kt + h] = (uint8_t)step;
      offset_a[n * G + 2 * kt + h] = (uint8_t)off;
    } else if (h == 0) {
      s_u8[n * G + kt] = (uint8_t)step;
      offset_a[n * G + kt] = (uint8_t)off;
    }
    if (codes) {
      uint8_t* dst = codes + (size_t)n * K + k0;   // 16-byte aligned: K % 128 == 0 and the base is checked by the host
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        uint32_t p[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          p[i] = (uint32_t)q[16 * v + 4 * i] | ((uint32_t)q[16 * v + 4 * i + 1] << 8) |
                 ((uint32_t)q[16 * v + 4 * i + 2] << 16) | ((uint32_t)q[16 * v + 4 * i + 3] << 24);
        *reinterpret_cast<uint4*>(dst + 16 * v) = make_uint4(p[0], p[1], p[2], p[3]);
      }
    }
  }
}

template <typename T>
static int run(const void* w, int N, long K, int group, float* s1, uint8_t* s_u8, uint8_t* offset_a, uint8_t* codes,
               uint8_t* blob, cudaStream_t st) {
  int* status = status_word();
  if (!status) return LQ_ERR_CUDA;
  // One pass wherever the rows are 32-byte vectors and a CTA holds one.
  int threads = 0;
  const int nv = (reinterpret_cast<uintptr_t>(w) & 31) == 0
                     ? row_units_per_thread(N, K >> 5, 4, 256, sizeof(T) == 2 ? 512 : 256, &threads) : 0;
  if (nv) {
    const int rows = blob ? (N + 127) / 128 * 128 : N;
    auto launch = [&](auto kern) {
      kern<<<rows, threads, 0, st>>>(static_cast<const T*>(w), s1, s_u8, offset_a, codes, blob, status, N, (int)K, group);
    };
    if (nv == 1) launch(quantise_rows_kernel<T, 1>);
    else if (nv == 2) launch(quantise_rows_kernel<T, 2>);
    else launch(quantise_rows_kernel<T, 4>);
    if (int rc = check_launch("quantise_rows_kernel")) return rc;
    return blob ? settle_blob(st) : LQ_OK;
  }
  row_amax_kernel<T><<<(N + 7) / 8, 256, 0, st>>>(static_cast<const T*>(w), s1, N, K);
  if (int rc = check_launch("row_amax_kernel")) return rc;
  dim3 grid((unsigned)(K >> 7), (unsigned)((N + 127) / 128));
  quantise_tiles_kernel<T><<<grid, 256, 0, st>>>(static_cast<const T*>(w), s1, s_u8, offset_a, codes, blob, status, N, K,
                                                 group);
  if (int rc = check_launch("quantise_tiles_kernel")) return rc;
  return blob ? settle_blob(st) : LQ_OK;
}

}  // namespace quantw
}  // namespace lq

using namespace lq;

extern "C" LQ_API int lq_quantize_weight(const void* w, int w_dtype, int N, int K, int group_size, float* s1,
                                         uint8_t* s_u8, uint8_t* offset_a, uint8_t* codes, uint8_t* blob,
                                         void* stream) {
  if (!w || !s1 || !s_u8 || !offset_a || N <= 0 || K <= 0) return LQ_ERR_BAD_ARG;
  if (K % 128 || (group_size != 64 && group_size != 128)) return LQ_ERR_SHAPE;
  if ((long)((N + 127) / 128) > 65535) return LQ_ERR_SHAPE;
  if (codes && (reinterpret_cast<uintptr_t>(codes) & 15)) return LQ_ERR_BAD_ARG;
  if (blob && (reinterpret_cast<uintptr_t>(blob) & 15)) return LQ_ERR_BAD_ARG;
  cudaStream_t st = as_stream(stream);
  switch (w_dtype) {
    case LQ_DT_BF16: return quantw::run<__nv_bfloat16>(w, N, K, group_size, s1, s_u8, offset_a, codes, blob, st);
    case LQ_DT_F16: return quantw::run<__half>(w, N, K, group_size, s1, s_u8, offset_a, codes, blob, st);
    case LQ_DT_F32: return quantw::run<float>(w, N, K, group_size, s1, s_u8, offset_a, codes, blob, st);
    default: return LQ_ERR_BAD_ARG;
  }
}
