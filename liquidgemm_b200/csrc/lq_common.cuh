// Shared device/host helpers for the liquidgemm_b200 kernels (sm_100a only).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/liquidgemm_b200.h"

namespace lq {

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
void record_cuda_error(cudaError_t e, const char* where);   // lq_api.cu
int check_launch(const char* where);                        // lq_api.cu: cudaGetLastError -> code
int sm_count();                                             // lq_api.cu: cached per device
int* status_word();                                         // lq_api.cu: device address of the status word

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Launch with programmatic stream serialisation: the kernel may start while the previous kernel
// of the stream is still draining, and must execute griddepcontrol.wait (dependency_wait()) before
// it touches anything an earlier kernel may have written or may still read-modify-write.  Switched
// off with LIQUIDGEMM_PDL=0 (then this is an ordinary launch).
bool pdl_enabled();                                         // lq_api.cu
template <typename... KArgs, typename... Args>
inline cudaError_t launch_overlapped(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                     Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// ---------------------------------------------------------------------------------------------
// LQQ arithmetic
// ---------------------------------------------------------------------------------------------
// Four codes in the four byte lanes of `w` -> four int8: (code*step + a) XOR 0x80 per lane.
// code <= 15 and step <= 16 keep every product <= 240 and every sum <= 255, so no lane carries
// (reference liquidgemm/quant.py:16-22, csrc/liquid_gemm/dequant.cu:39-43).
__device__ __forceinline__ uint32_t lqq_dequant4(uint32_t codes, uint32_t step, uint32_t a_bcast) {
  return (codes * step + a_bcast) ^ 0x80808080u;
}

// The output formula of every fused epilogue: two fp32 multiplies, left to right
// (reference liquidgemm/quant.py:152, csrc/liquid_gemm/epilogue.cu:57).
__device__ __forceinline__ float lqq_scale(int acc, float a_scale, float w_scale) {
  return __fmul_rn(__fmul_rn(__int2float_rn(acc), a_scale), w_scale);
}

// Store one output element in the dtype selected by `out_dtype` (LQ_DT_*).
__device__ __forceinline__ void store_out(void* y, size_t idx, float v, int out_dtype) {
  if (out_dtype == LQ_DT_BF16) {
    reinterpret_cast<__nv_bfloat16*>(y)[idx] = __float2bfloat16_rn(v);
  } else if (out_dtype == LQ_DT_F16) {
    reinterpret_cast<__half*>(y)[idx] = __float2half_rn(v);
  } else {
    reinterpret_cast<float*>(y)[idx] = v;
  }
}

// Bias element n of a vector stored in the output dtype, as float.
__device__ __forceinline__ float load_bias(const void* b, long n, int out_dtype) {
  if (out_dtype == LQ_DT_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(b)[n]);
  if (out_dtype == LQ_DT_F16) return __half2float(reinterpret_cast<const __half*>(b)[n]);
  return reinterpret_cast<const float*>(b)[n];
}

// Store with an optional bias.  The product is first rounded to the output type and the bias is added to
// that rounded value in float32, then rounded again: exactly what PyTorch's `y + bias` computes on the
// operator's output (the reference adds its bias that way, liquidgemm/vllm_plugin.py:205-206).
__device__ __forceinline__ void store_out_bias(void* y, size_t idx, float v, float bias, bool has_bias, int out_dtype) {
  if (out_dtype == LQ_DT_BF16) {
    __nv_bfloat16 t = __float2bfloat16_rn(v);
    if (has_bias) t = __float2bfloat16_rn(__fadd_rn(__bfloat162float(t), bias));
    reinterpret_cast<__nv_bfloat16*>(y)[idx] = t;
  } else if (out_dtype == LQ_DT_F16) {
    __half t = __float2half_rn(v);
    if (has_bias) t = __float2half_rn(__fadd_rn(__half2float(t), bias));
    reinterpret_cast<__half*>(y)[idx] = t;
  } else {
    reinterpret_cast<float*>(y)[idx] = has_bias ? __fadd_rn(v, bias) : v;
  }
}

// ---------------------------------------------------------------------------------------------------------
// Epilogue of the tensor-core kernels, sixteen accumulator columns (tokens) of one channel at a time.  These
// kernels are bound by instruction issue, and an epilogue that decides the output type, the bias and the
// ragged edge per element and forms every address with 64-bit arithmetic was measured to cost the CTA-pair
// kernel 16 % on layers with K = 4096: here the decisions are made once per sixteen elements and an address
// is one 32 x 32 + 64-bit multiply-add.  kEpiI32 selects raw int32 outputs.
constexpr int kEpiI32 = 3;

template <int DT, bool BIAS>
__device__ __forceinline__ uint16_t epi_bits16(int acc, float a_scale, float w_scale, float bias) {
  const float y = lqq_scale(acc, a_scale, w_scale);
  if (DT == LQ_DT_BF16) {
    __nv_bfloat16 t = __float2bfloat16_rn(y);
    if (BIAS) t = __float2bfloat16_rn(__fadd_rn(__bfloat162float(t), bias));
    return *reinterpret_cast<uint16_t*>(&t);
  }
  __half t = __float2half_rn(y);
  if (BIAS) t = __float2half_rn(__fadd_rn(__half2float(t), bias));
  return *reinterpret_cast<uint16_t*>(&t);
}

// Straight to global memory: element j goes to out + (idx0 + j * ld) elements.
template <int DT, bool BIAS, bool FULL>
__device__ __forceinline__ void epi_store_cols_t(void* out, size_t idx0, long ld, const int (&v)[16], const float (&sc)[16],
                                                 float w_scale, float bias, int valid) {
  constexpr int ES = (DT == LQ_DT_BF16 || DT == LQ_DT_F16) ? 2 : 4;
  char* p = static_cast<char*>(out) + idx0 * ES;
  const uint32_t pitch = (uint32_t)ld * ES;   // a row pitch below 4 GB
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (FULL || j < valid) {
      char* q = p + (uint64_t)pitch * (uint32_t)j;
      if (DT == kEpiI32) *reinterpret_cast<int32_t*>(q) = v[j];
      else if (DT == LQ_DT_F32) {
        const float y = lqq_scale(v[j], sc[j], w_scale);
        *reinterpret_cast<float*>(q) = BIAS ? __fadd_rn(y, bias) : y;
      } else {
        *reinterpret_cast<uint16_t*>(q) = epi_bits16<DT, BIAS>(v[j], sc[j], w_scale, bias);
      }
    }
  }
}
template <int DT>
__device__ __forceinline__ void epi_store_cols_dt(void* out, size_t idx0, long ld, const int (&v)[16], const float (&sc)[16],
                                                  float w_scale, float bias, bool has_bias, int valid) {
  if (valid >= 16) {
    if (has_bias) epi_store_cols_t<DT, true, true>(out, idx0, ld, v, sc, w_scale, bias, valid);
    else epi_store_cols_t<DT, false, true>(out, idx0, ld, v, sc, w_scale, bias, valid);
  } else {
    if (has_bias) epi_store_cols_t<DT, true, false>(out, idx0, ld, v, sc, w_scale, bias, valid);
    else epi_store_cols_t<DT, false, false>(out, idx0, ld, v, sc, w_scale, bias, valid);
  }
}
// out_mode: LQ_DT_* or kEpiI32; `valid` of the sixteen elements exist (the ragged last token chunk).
__device__ __forceinline__ void epi_store_cols(void* out, int out_mode, size_t idx0, long ld, const int (&v)[16],
                                               const float (&sc)[16], float w_scale, float bias, bool has_bias, int valid) {
  if (out_mode == LQ_DT_BF16) epi_store_cols_dt<LQ_DT_BF16>(out, idx0, ld, v, sc, w_scale, bias, has_bias, valid);
  else if (out_mode == LQ_DT_F16) epi_store_cols_dt<LQ_DT_F16>(out, idx0, ld, v, sc, w_scale, bias, has_bias, valid);
  else if (out_mode == LQ_DT_F32) epi_store_cols_dt<LQ_DT_F32>(out, idx0, ld, v, sc, w_scale, bias, has_bias, valid);
  else epi_store_cols_dt<kEpiI32>(out, idx0, ld, v, sc, w_scale, bias, false, valid);
}

// Into a shared-memory stage of 2-byte outputs: element j goes to col[j * 128] (the thread's channel column of a
// [16 tokens][128 channels] block).  out_mode: LQ_DT_BF16 or LQ_DT_F16.
template <int DT, bool BIAS>
__device__ __forceinline__ void epi_stage_cols_t(uint16_t* col, const int (&v)[16], const float (&sc)[16], float w_scale,
                                                 float bias) {
#pragma unroll
  for (int j = 0; j < 16; ++j) col[j * 128] = epi_bits16<DT, BIAS>(v[j], sc[j], w_scale, bias);
}
__device__ __forceinline__ void epi_stage_cols(uint16_t* col, int out_mode, const int (&v)[16], const float (&sc)[16],
                                               float w_scale, float bias, bool has_bias) {
  if (out_mode == LQ_DT_BF16) {
    if (has_bias) epi_stage_cols_t<LQ_DT_BF16, true>(col, v, sc, w_scale, bias);
    else epi_stage_cols_t<LQ_DT_BF16, false>(col, v, sc, w_scale, bias);
  } else {
    if (has_bias) epi_stage_cols_t<LQ_DT_F16, true>(col, v, sc, w_scale, bias);
    else epi_stage_cols_t<LQ_DT_F16, false>(col, v, sc, w_scale, bias);
  }
}

// ---------------------------------------------------------------------------------------------
// quantisers
// ---------------------------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

__device__ __forceinline__ float block_max(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float r = lane < (blockDim.x >> 5) ? red[lane] : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
  return r;
}

// Nearest-integer quotients without a division.  Both quantisers need x / scale only to the nearest integer, with
// |x / scale| < 127.5.  With inv = fl(1 / scale) the product x * inv differs from x / scale by a relative 2^-24, and
// the IEEE quotient by another 2^-24: together less than 2^-15 here.  So wherever x * inv lies further than 2^-14
// from every half-integer its nearest integer is rint(x / scale) bit for bit.  A group (a 16-byte vector of tokens, an
// octet of weights) with an element closer than that (about one element in 8192), an infinity or a NaN takes the division:
// a token vector as a whole, an octet of weights only for such elements (all eight divided: 28672 x 4096 weights 82.5 us
// instead of 81.6, two comparisons, spread 0.6 %).
constexpr float kRoundMagic = 12582912.0f;   // 1.5 * 2^23: x + kRoundMagic has rint(x) in its low bits
constexpr float kSafeDist = 0.5f - 0x1p-14f;

// max(a, |b|, |c|); unlike fmaxf, a NaN operand gives NaN.
__device__ __forceinline__ float max_abs_nan(float a, float b, float c) {
  float d;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Two float32 operations in one instruction (the quantisers are bound by instruction issue, not by the FMA pipe).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tadd.rn.f32x2 rd, ra, rb;\n\t"
      "mov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

// t[i] = kRoundMagic + (nearest integer of x[i] * inv); false when one of them needs the division.
template <int N>
__device__ __forceinline__ bool round_quotients(const float2 (&x)[N], float inv, float2 (&t)[N]) {
  float far = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    t[i] = fma2(x[i], both(inv), both(kRoundMagic));
    const float2 r = add2(t[i], both(-kRoundMagic));     // the nearest integer, exactly
    const float2 d = fma2(x[i], both(-inv), r);          // its distance from x * inv
    far = max_abs_nan(far, d.x, d.y);
  }
  return far < kSafeDist;
}

// The same test for one element.
__device__ __forceinline__ bool near_integer(float x, float inv) {
  const float r = __fadd_rn(__fmaf_rn(x, inv, kRoundMagic), -kRoundMagic);
  return fabsf(__fmaf_rn(x, -inv, r)) < kSafeDist;
}

// Two elements of a 32-bit word (16-bit types), low half first.
template <typename T> __device__ __forceinline__ float2 unpack2(uint32_t w);
template <> __device__ __forceinline__ float2 unpack2<__half>(uint32_t w) {
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <> __device__ __forceinline__ float2 unpack2<__nv_bfloat16>(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

// Running |max| of a row, two 16-bit elements (or one float) at a time; NaN is ignored like fmaxf ignores it.
template <typename T> struct RowMax;
template <> struct RowMax<float> {
  float m = 0.f;
  __device__ __forceinline__ void take(const uint4& v) {
    const float* e = reinterpret_cast<const float*>(&v);
    m = fmaxf(fmaxf(m, fmaxf(fabsf(e[0]), fabsf(e[1]))), fmaxf(fabsf(e[2]), fabsf(e[3])));
  }
  __device__ __forceinline__ float value() const { return m; }
};
// (max.xorsign.abs: the larger magnitude in one instruction; its sign is dropped at the end)
template <> struct RowMax<__half> {
  uint32_t m = 0u;
  static __device__ __forceinline__ uint32_t mx(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("max.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
  }
  __device__ __forceinline__ void take(const uint4& v) { m = mx(m, mx(mx(v.x, v.y), mx(v.z, v.w))); }
  __device__ __forceinline__ float value() const {
    const __half2 h = __habs2(*reinterpret_cast<const __half2*>(&m));
    return fmaxf(__low2float(h), __high2float(h));
  }
};
template <> struct RowMax<__nv_bfloat16> {
  uint32_t m = 0u;
  static __device__ __forceinline__ uint32_t mx(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
  }
  __device__ __forceinline__ void take(const uint4& v) { m = mx(m, mx(mx(v.x, v.y), mx(v.z, v.w))); }
  __device__ __forceinline__ float value() const {
    return fmaxf(fabsf(__uint_as_float(m << 16)), fabsf(__uint_as_float(m & 0xffff0000u)));
  }
};

// The elements of one 16-byte vector, in pairs.
template <typename T>
__device__ __forceinline__ void vec_floats(const uint4& raw, float2 (&x)[8 / sizeof(T)]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 8 / (int)sizeof(T); ++i) {
    if constexpr (sizeof(T) == 4) x[i] = make_float2(__uint_as_float(w[2 * i]), __uint_as_float(w[2 * i + 1]));
    else x[i] = unpack2<T>(w[i]);
  }
}

// ---- activations ----
__device__ __forceinline__ int quant1(float x, float scale) {
  // IEEE division, round half to even, clamp: liquidgemm/quant.py:140 of the reference.
  int q = __float2int_rn(__fdiv_rn(x, scale));
  return max(-127, min(127, q));
}

// The scale of a token row: max(amax, 1e-12) / 127, correctly rounded.  Markstein's division step (IBM J. Res. Dev. 34,
// 1990): the exact residual of the quotient by the rounded reciprocal corrects it.  It saves the general division's 100
// cycles where a row's latency counts; infinities and NaN take the division.
__device__ __forceinline__ float token_scale(float amax) {
  const float a = fmaxf(amax, 1e-12f);
  constexpr float kInv = 1.0f / 127.0f;
  const float q = __fmul_rn(a, kInv);
  const float s = __fmaf_rn(__fmaf_rn(-127.0f, q, a), kInv, q);
  return a < 3e38f ? s : __fdiv_rn(a, 127.0f);
}

// The quantised bytes of one 16-byte vector: VEC int8 in VEC / 4 words.
template <typename T>
__device__ __forceinline__ void quant_vec(const uint4& raw, float scale, float inv, uint32_t (&out)[4 / sizeof(T)]) {
  constexpr int VEC = 16 / sizeof(T);
  float2 x[VEC / 2], t[VEC / 2];
  vec_floats<T>(raw, x);
  uint32_t q[VEC];
  const bool safe = round_quotients(x, inv, t);
#pragma unroll
  for (int i = 0; i < VEC / 2; ++i) {
    q[2 * i] = __float_as_uint(t[i].x);
    q[2 * i + 1] = __float_as_uint(t[i].y);
  }
  if (!safe) {
#pragma unroll
    for (int i = 0; i < VEC / 2; ++i) {
      q[2 * i] = (uint32_t)quant1(x[i].x, scale);
      q[2 * i + 1] = (uint32_t)quant1(x[i].y, scale);
    }
  }
#pragma unroll
  for (int i = 0; i < VEC / 4; ++i)
    out[i] = __byte_perm(__byte_perm(q[4 * i], q[4 * i + 1], 0x0040), __byte_perm(q[4 * i + 2], q[4 * i + 3], 0x0040), 0x5410);
}

// The register-held row kernels: how many units (a power of two, at most nv_max) of a row of `n` a thread holds, and the
// CTA's threads.  Few rows spread wide, so that a row's latency is short; many rows use small CTAs (down to
// `few_threads`), whose load, reduction and store phases overlap each other's.  0: the row does not fit.
inline int row_units_per_thread(long rows, long n, int nv_max, int few_threads, int max_threads, int* threads) {
  for (int nv = 1; nv <= nv_max; nv *= 2) {
    *threads = (int)((n + nv - 1) / nv + 31) / 32 * 32;
    if (*threads <= max_threads && (nv == nv_max || *threads <= few_threads || rows * *threads <= (long)sm_count() * 1280))
      return nv;
  }
  return 0;
}

// Where a kernel's outputs go: the same [M, N] block is written into up to 8 row-major matrices with
// row stride `ld` elements at column offset `col0`.  One destination with ld = N, col0 = 0 is the
// ordinary output; several destinations (this GPU's and its peers' full-width output, mapped into this
// process) make the epilogue do the all-gather of an N-sharded layer with plain stores.
struct OutSpec {
  void* ptr[8];
  int n;
  long ld, col0;
};
inline OutSpec single_out(void* out, long N) {
  OutSpec o = {};
  o.ptr[0] = out;
  o.n = 1;
  o.ld = N;
  o.col0 = 0;
  return o;
}
// Cross-GPU ordering for the gather-by-stores epilogue.  Every CTA, after its last output store, adds 1
// to word `index` of each destination rank's flag array (release, system scope); a consumer kernel
// on rank r waits until its own word reached the number of CTAs of all ranks before it reads the
// gathered data.  The flags live in memory every rank can write (symmetric memory); the host zeroes
// them, and orders the ranks once, before the first kernel of a sequence.
struct PeerSync {
  unsigned* signal[8];     // per destination rank: its flag array (null array entries = no signalling)
  int n_signal;
  int signal_index;
  const unsigned* wait;    // this rank's flag word to wait on before reading the tokens, or null
  unsigned wait_value;
};
__device__ __forceinline__ void peer_signal(const PeerSync& p) {
#pragma unroll
  for (int r = 0; r < 8; ++r)   // constant indices: see store_out_all
    if (r < p.n_signal)
      asm volatile("red.release.sys.global.add.u32 [%0], 1;" ::"l"(p.signal[r] + p.signal_index) : "memory");
}
// Bounded: gives up after `limit_ns` and returns false (the caller records a status code and goes on).
// Polls with relaxed loads and orders the following reads with one acquire fence at the end.
__device__ __forceinline__ bool peer_wait(const PeerSync& p, unsigned long long limit_ns) {
  if (!p.wait) return true;
  unsigned long long t0 = 0;
  bool ok = true;
  for (unsigned spins = 0;; ++spins) {
    unsigned v;
    asm volatile("ld.relaxed.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p.wait) : "memory");
    if (v >= p.wait_value) break;
    unsigned long long now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if (spins == 0) t0 = now;
    else if (now - t0 > limit_ns) {
      ok = false;
      break;
    }
    __nanosleep(200);
  }
  asm volatile("fence.acquire.sys;" ::: "memory");
  return ok;
}

// Kernel parameters of the gather-by-stores variants.  They travel as a separate kernel parameter that
// only the multi-destination instantiations have: measured on B200, the programmatically serialised
// decode launches cost 0.5-1 us more once their parameters exceed 256 bytes, so the ordinary
// single-output kernels keep theirs below that.
struct MultiOut {
  OutSpec out;
  PeerSync sync;
};
struct NoMultiOut {};

__device__ __forceinline__ void store_out_all(const OutSpec& o, long m, long n, float v, int out_dtype) {
  const size_t idx = (size_t)(m * o.ld + o.col0 + n);
  // Constant indices only: a run-time index into a kernel parameter makes the compiler copy the whole
  // parameter block to local memory and read every field from there (measured: +1 us per launch).
  store_out(o.ptr[0], idx, v, out_dtype);
  if (o.n > 1) {
#pragma unroll
    for (int r = 1; r < 8; ++r)
      if (r < o.n) store_out(o.ptr[r], idx, v, out_dtype);
  }
}

__device__ __forceinline__ void store_out_all(const OutSpec& o, long m, long n, float v, float bias, bool has_bias,
                                              int out_dtype) {
  const size_t idx = (size_t)(m * o.ld + o.col0 + n);
  store_out_bias(o.ptr[0], idx, v, bias, has_bias, out_dtype);   // constant indices only, as above
  if (o.n > 1) {
#pragma unroll
    for (int r = 1; r < 8; ++r)
      if (r < o.n) store_out_bias(o.ptr[r], idx, v, bias, has_bias, out_dtype);
  }
}

// ---------------------------------------------------------------------------------------------
// memory
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint4 ldg_stream_v4(const void* p) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(p));
  return r;
}

// Data that an earlier kernel of the stream may still be writing while this one is resident already (programmatic launch): a
// coherent load, for use behind dependency_wait().  ld.global.nc (which __ldg, and const __restrict__ parameters, stand for as well)
// is defined only for data that nobody writes during the kernel's life: its lines may be in the SM's L1 from a
// kernel that read the same addresses before they were written again.  Tile blobs, whose writers settle, take the one above.
__device__ __forceinline__ uint4 ld_stream_v4(const void* p) {
  uint4 r;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(p)
               : "memory");
  return r;
}

// Programmatic dependent launch, device side.  allow_dependents(): the next kernel of the stream may be
// scheduled once every CTA of this grid has executed it.  dependency_wait(): returns when all earlier
// kernels of the stream have completed and their writes are visible (no-op for an ordinary launch).
__device__ __forceinline__ void allow_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

}  // namespace lq
