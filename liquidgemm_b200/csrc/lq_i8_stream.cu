// INT8 x INT8 GEMM for decode and small mixed batches: C[M,N] = A[M,K] * B[N,K]^T, int32 sums, optionally scaled
// (the plugin's INT8-weights mode below the sizes the CTA-pair kernel takes).
//
// HBM-bound: the INT8 weights are read once and everything else is small, so the kernel is a weight stream with
// tensor cores attached.  One 128-channel x BN-token tile and one k-range per CTA, two CTAs per SM; `splits` k-ranges
// per tile so that the grid fills the SMs.  With one k-range the epilogue is fused; with several every CTA writes an
// int32 plane and the finish pass adds the planes, scales and casts (exact in any order).
//  * warp 0  producer: one thread keeps NS 128 x 128 weight boxes in flight (tensor map, 128-byte swizzle).  B may be the
//            output of the kernel just before (a quantiser, the dequantiser), so it is read after the wait for that
//            kernel; before it the first NS boxes are only hinted to L2, which changes no result whoever writes them
//            (eight linears behind quantisers, 8 tokens: 123.2 us without the hint, 122.5 with it, 115 when they were
//            read without waiting, which was wrong wherever B was fresh).
//  * warp 1  tensor memory and MMA issue: four 128 x BN x 32 tcgen05.mma kind::i8 per k-step, both operands from
//            shared memory; its commit recycles the stage.
//  * warps 2..9  two sets of 128 threads, k-steps in turn: the set that owns a k-step fetches its BN x 128-byte token
//            slice (L2 hits, requested before the wait for the stage) and stores it in the layout the 128-byte swizzle
//            gives (chunk c of row r at chunk c ^ (r & 7)).  A second tensor map for the tokens would push the kernel
//            parameters over 256 bytes, which costs a programmatically serialised launch 0.5-1 us.
//            Then the epilogue, the sets sharing the accumulator's columns.
// Every wait is bounded; the status codes are 151-155.
#include <cuda.h>

#include <mutex>

#include "lq_common.cuh"
#include "lq_tc_ptx.cuh"

namespace lq {

int launch_finish(const int32_t* acc, const float* ascale, const float* s1, const void* bias, const OutSpec& out,
                  const PeerSync* sync, int out_dtype, int planes, bool clear_planes, int M, int N, cudaStream_t st);  // lq_elementwise.cu
int make_byte_matrix_map(CUtensorMap* map, const void* ptr, long rows, long row_bytes, int box_rows,
                         int box_bytes);  // lq_gemm_tc.cu

namespace i8s {

constexpr int kWStage = 128 * 128;
constexpr int kSets = 2;
constexpr int kThreads = 64 + 128 * kSets;
constexpr uint64_t kWaitLimitNs = 2000000000ull;

struct Args {
  const int8_t* x;       // [M, K]
  const float* ascale;   // [M]
  const float* s1;       // [N]
  void* out;             // [M, N], or int32 planes [splits][M][N]
  int* status;
  int out_mode;          // LQ_DT_* or kEpiI32
  int M, N, K;
};

template <int BN, int NS>
struct Cfg {
  static constexpr int kXStage = BN * 128;
  static constexpr int kTmemCols = BN <= 32 ? 32 : BN;
  static constexpr int kBarBytes = (3 * NS + 1) * 8 + 16;
  static constexpr int kUsedBytes = 1024 /* alignment slack */ + NS * (kXStage + kWStage) + kBarBytes;
  static constexpr int kSmemBytes = kUsedBytes > 78 * 1024 ? kUsedBytes : 78 * 1024;   // never three CTAs on an SM
  static_assert(kSmemBytes <= 113 * 1024, "two CTAs per SM share the shared memory");
};

template <int BN, int NS>
__global__ void __launch_bounds__(kThreads, 2)
i8_stream_kernel(const __grid_constant__ CUtensorMap tmap_w, const Args args) {
  using C = Cfg<BN, NS>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const uint32_t xs = base;                        // NS token stages (1024-aligned)
  const uint32_t ws = xs + NS * C::kXStage;        // NS weight stages
  const uint32_t bar_full = ws + NS * kWStage;     // [NS] weight box landed
  const uint32_t bar_xready = bar_full + NS * 8;   // [NS] token slice stored
  const uint32_t bar_empty = bar_xready + NS * 8;  // [NS] the MMAs that read the stage are done
  const uint32_t bar_acc = bar_empty + NS * 8;     // accumulator final
  const uint32_t tmem_slot = bar_acc + 8;
  volatile uint32_t* tmem_slot_p = reinterpret_cast<volatile uint32_t*>(smem + (tmem_slot - base));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nt = blockIdx.x, mt = blockIdx.y, z = blockIdx.z, splits = gridDim.z;
  const int kt_total = args.K >> 7;
  const int kt_begin = (int)(((long)z * kt_total) / splits);
  const int nk = (int)(((long)(z + 1) * kt_total) / splits) - kt_begin;
  const int m0 = mt * BN;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NS; ++s) {
      ptx::mbar_init(bar_full + 8 * s, 1);
      ptx::mbar_init(bar_xready + 8 * s, 128);
      ptx::mbar_init(bar_empty + 8 * s, 1);
    }
    ptx::mbar_init(bar_acc, 1);
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&tmap_w);
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, C::kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  allow_dependents();   // the next kernel of the stream may start prefetching its weights
  const uint32_t tmem_acc = *tmem_slot_p;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (lane == 0) {
      for (int j = 0; j < nk && j < NS; ++j) ptx::tensor_prefetch_2d(&tmap_w, (kt_begin + j) * 128, nt * 128);
      dependency_wait();
      int i = 0;
      bool ok = true;
      for (; i < nk; ++i) {
        const int s = i % NS;
        if (i >= NS && !ptx::mbar_wait_bounded(bar_empty + 8 * s, ((uint32_t)(i / NS) & 1u) ^ 1u, kWaitLimitNs)) {
          atomicExch(args.status, 151);
          ok = false;
          break;
        }
        ptx::mbar_expect_tx(bar_full + 8 * s, kWStage);
        ptx::tensor_load_2d(ws + s * kWStage, &tmap_w, (kt_begin + i) * 128, nt * 128, bar_full + 8 * s);
      }
      if (!ok) {
        // copies already issued still write shared memory: let them land before the CTA exits
        for (int j = i > NS ? i - NS : 0; j < i; ++j)
          ptx::mbar_wait_bounded(bar_full + 8 * (j % NS), (uint32_t)(j / NS) & 1u, kWaitLimitNs);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issue
    // The whole warp walks the loop; one elected lane issues (see ptx::elect_one).
    const bool leader = ptx::elect_one();
    constexpr uint32_t idesc = ptx::idesc_i8(BN);
    bool ok = true;
    for (int i = 0; i < nk; ++i) {
      const int s = i % NS;
      const uint32_t ph = (uint32_t)(i / NS) & 1u;
      ok = ptx::mbar_wait_bounded(bar_full + 8 * s, ph, kWaitLimitNs);
      if (ok) ok = ptx::mbar_wait_bounded(bar_xready + 8 * s, ph, kWaitLimitNs);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (leader) atomicExch(args.status, 152);
        break;
      }
      ptx::tc_fence_after();
      if (leader) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          ptx::mma_i8_ss(tmem_acc, ptx::smem_desc_sw128(ws + s * kWStage + j * 32),
                         ptx::smem_desc_sw128(xs + s * C::kXStage + j * 32), idesc, (i > 0 || j > 0) ? 1u : 0u);
        ptx::tc_commit(bar_empty + 8 * s);
      }
    }
    if (ok && leader) ptx::tc_commit(bar_acc);
  } else {
    // ------------------------------------------------------------------ tokens, then epilogue
    const int set = (threadIdx.x - 64) >> 7;
    const int jx = (threadIdx.x - 64) & 127;
    const int quad = warp & 3;               // tensor-memory lane quadrant this warp may access
    const int row = quad * 32 + lane;        // channel inside the tile == tensor-memory lane
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const int x_row = jx >> 3;               // this thread moves 16-byte chunk (jx & 7) of rows x_row + 16 q
    const uint32_t x_off = (uint32_t)(x_row * 128 + (((jx & 7) ^ (x_row & 7)) << 4));
    const int8_t* x_src = args.x + (size_t)(m0 + x_row) * args.K + (size_t)kt_begin * 128 + (jx & 7) * 16;
    bool ok = true;
    dependency_wait();   // tokens, scales, outputs and planes belong to earlier kernels until here
    for (int i = set; i < nk; i += kSets) {
      const int s = i % NS;
      uint4 xv[BN / 16];
#pragma unroll
      for (int q = 0; q < BN / 16; ++q)
        xv[q] = (m0 + x_row + 16 * q < args.M) ? ld_stream_v4(x_src + (size_t)(16 * q) * args.K + (size_t)i * 128)
                                               : make_uint4(0u, 0u, 0u, 0u);
      if (i >= NS && !ptx::mbar_wait_bounded(bar_empty + 8 * s, ((uint32_t)(i / NS) & 1u) ^ 1u, kWaitLimitNs)) {
        atomicExch(args.status, 153);
        ok = false;
        break;
      }
#pragma unroll
      for (int q = 0; q < BN / 16; ++q)
        *reinterpret_cast<uint4*>(smem + s * C::kXStage + x_off + q * 2048) = xv[q];
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // ordinary stores, read by the tensor core
      ptx::mbar_arrive(bar_xready + 8 * s);
    }
    if (ok && !ptx::mbar_wait_bounded(bar_acc, 0u, kWaitLimitNs)) {
      atomicExch(args.status, 154);
      ok = false;
    }
    __syncwarp();
    if (ok) {
      ptx::tc_fence_after();
      const long n = (long)nt * 128 + row;
      const bool n_ok = n < args.N;
      const bool raw = args.out_mode == kEpiI32;
      const float w_scale = (n_ok && !raw) ? args.s1[n] : 0.f;
      char* out = static_cast<char*>(args.out) + (raw ? (size_t)z * args.M * args.N * 4 : 0);
#pragma unroll 1
      for (int c0 = 16 * set; c0 < BN; c0 += 16 * kSets) {   // the sets share the accumulator's columns
        if (m0 + c0 >= args.M) break;                        // uniform over the set
        int v[16];
        ptx::tmem_ld16(tmem_acc + lane_addr + c0, v);
        float sc[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) sc[j] = (!raw && m0 + c0 + j < args.M) ? args.ascale[m0 + c0 + j] : 0.f;
        ptx::tc_wait_ld();
        if (n_ok)
          epi_store_cols(out, args.out_mode, (size_t)(m0 + c0) * args.N + n, args.N, v, sc, w_scale, 0.f, false,
                         args.M - (m0 + c0));
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_acc, C::kTmemCols);
  }
}

template <int BN, int NS>
static int launch(const CUtensorMap& tw, const Args& a, int splits, cudaStream_t st) {
  using C = Cfg<BN, NS>;
  auto kern = &i8_stream_kernel<BN, NS>;
  static std::once_flag once[64];
  int dev = 0;
  cudaGetDevice(&dev);
  cudaError_t e = cudaSuccess;
  std::call_once(once[dev & 63], [&]() {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
  });
  if (e == cudaSuccess)
    e = launch_overlapped(kern, dim3((a.N + 127) / 128, (a.M + BN - 1) / BN, splits), dim3(kThreads), (size_t)C::kSmemBytes,
                          st, tw, a);
  if (e != cudaSuccess) {
    record_cuda_error(e, "i8_stream_kernel launch");
    return LQ_ERR_CUDA;
  }
  return check_launch("i8_stream_kernel");
}

static int bn_for(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128; }

}  // namespace i8s

static long i8_stream_tiles(int M, int N) {
  const int bn = i8s::bn_for(M);
  return (long)((N + 127) / 128) * ((M + bn - 1) / bn);
}

// Up to 64 tokens always; up to 255 where the tiles leave at least half of the CTA slots to k-ranges.  Measured against
// the one-CTA-per-SM persistent kernel, which takes whole tiles (so that a 4096-channel layer kept 32 SMs busy): 8 tokens
// 6144 x 4096 11.2 -> 8.2 us, 4096 x 4096 10.9 -> 6.7, 28672 x 4096 25.2 -> 22.8, 4096 x 14336 27.7 -> 14.0, 1024 x 28672 50.2 -> 10.6;
// 64 tokens 12.7 -> 10.1, 12.4 -> 9.4, 26.3 -> 25.1, 29.6 -> 16.6, 52.6 -> 12.4; 200 tokens 17.5 -> 16.8, 16.8 -> 13.6, (wide layers keep
// the persistent kernel), 39.3 -> 31.0, 66.0 -> 19.9; but 28672 x 4096 at 128 tokens 29.3 -> 32.1 and at 200 48.5 -> 52.3, and from 256
// tokens on the persistent kernel's 192-token tiles win.
bool i8_stream_serves(int M, int N, int K) {
  (void)K;
  return M <= 64 || (M < 256 && 2 * i8_stream_tiles(M, N) <= 2L * sm_count());
}

// k-ranges per tile: fill the two CTA slots of every SM, at least three k-steps each (4096 x 4096 at 8 tokens: 2 / 3 / 6 / 9
// ranges 8.3 / 7.4 / 6.7 / 6.8 us; 4096 x 14336 21.6 / 17.9 / 14.7 / 14.3).
static int i8_stream_splits(int M, int N, int K) {
  const long tiles = i8_stream_tiles(M, N);
  const int kt = K / 128;
  long S = 2L * sm_count() / (tiles > 0 ? tiles : 1);
  if (S > kt / 3) S = kt / 3;
  if (S > 16) S = 16;
  return S < 1 ? 1 : (int)S;
}

size_t i8_stream_workspace_bytes(int M, int N, int K) {
  const int S = i8_stream_splits(M, N, K);
  return S > 1 ? (size_t)S * M * N * 4 : 0;
}

// out_mode: LQ_DT_* or 3 (raw int32).  `ws`: i8_stream_workspace_bytes() of scratch.
int run_i8_stream(const int8_t* x, const int8_t* w, const float* ascale, const float* s1, void* out, int out_mode, int M,
                  int N, int K, void* ws, size_t ws_bytes, cudaStream_t st) {
  using namespace i8s;
  const int S = i8_stream_splits(M, N, K);
  if (S > 1 && (!ws || ws_bytes < i8_stream_workspace_bytes(M, N, K))) return LQ_ERR_WORKSPACE;
  CUtensorMap tw;
  if (int rc = make_byte_matrix_map(&tw, w, N, K, 128, 128)) return rc;
  Args a;
  a.x = x;
  a.ascale = ascale;
  a.s1 = s1;
  a.out = S > 1 ? ws : out;
  a.status = status_word();
  a.out_mode = S > 1 ? kEpiI32 : out_mode;
  a.M = M;
  a.N = N;
  a.K = K;
  if (!a.status) return LQ_ERR_CUDA;
  int rc;
  switch (bn_for(M)) {
    case 16: rc = launch<16, 6>(tw, a, S, st); break;
    case 32: rc = launch<32, 5>(tw, a, S, st); break;
    case 64: rc = launch<64, 4>(tw, a, S, st); break;
    default: rc = launch<128, 3>(tw, a, S, st); break;
  }
  if (rc || S <= 1) return rc;
  return launch_finish(static_cast<const int32_t*>(ws), ascale, s1, nullptr, single_out(out, N), nullptr, out_mode, S, false,
                       M, N, st);
}

}  // namespace lq
