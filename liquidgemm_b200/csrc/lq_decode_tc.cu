// W4A8 tensor-core linear for decode batches (up to 32 tokens): the weights stream from HBM once and everything else is
// small, so what a launch costs is its chain of latencies.  Replaces the reference's split-K WGMMA path for small M
// (csrc/liquid_gemm/w4a8_wgmma.cu:333-503 with the split rule at :523-534 and the finish kernel :39-56) in ONE launch.
//
//  * One 128-channel tile and one k-range per CTA; the CTAs that share a tile's K form a thread-block cluster (up to
//    eight).  320 threads, at most half of an SM, so that the next launch's CTAs become resident beside this launch's.
//  * Everything that needs only the weights happens BEFORE the wait for the previous kernel: the ring fills and the first
//    NT k-tiles are unpacked into tensor memory (the MMA's A operand).  After the wait come, one after the other, one
//    round of token loads, the MMAs, the join, the stores.
//  * warp 0  producer: one thread keeps a ring of weight tiles in flight, one contiguous 8704-byte bulk copy each.
//  * warps 2..9  two dequant sets taking alternate k-tiles; thread r of a set owns weight row r: 64 bytes of nibbles ->
//            128 INT8 (AND / SHR+AND / IMAD / XOR on 4-lane words) -> tcgen05.st into tensor-memory lane r.
//            After the wait they fetch the tokens of the CTA's whole k-range in one go (16 bytes a thread and load, L2
//            hits) and store them in the 128-byte-swizzled layout the MMA's descriptor expects.  Tokens do not come
//            through the copy engine, where they would queue behind the weights.
//            XT an activation type: the tokens are quantised here, which saves the quantiser's launch and its place in the
//            stream.  A CTA reads only its k-range of the activations; the row maxima of the cluster's CTAs meet in each
//            CTA's shared memory (st.async), and what a thread has loaded it quantises out of its registers.
//  * warp 1  MMA: the warp walks the loop, one elected lane issues four 128 x BN x 32 tcgen05.mma kind::i8 per k-tile (A from
//            tensor memory, B = tokens through a shared-memory descriptor); its commit recycles the operand stage.
//  * Join: each CTA of the cluster owns a block of the tile's channels and receives the other CTAs' int32 sums for it in
//    its shared memory (st.async, counted by an mbarrier); it adds them, scales and stores.  Integer sums are exact in any
//    order, so results do not depend on the split.  The optional bias is added to the value already rounded to the
//    output type, as PyTorch's `y + bias` after the reference's operator does (liquidgemm/vllm_plugin.py:205-206).
// Every wait is bounded; a thread whose wait expires records a site code, stops waiting and still runs the rest of its
// control flow, so the CTA reaches the exit where tensor memory is released.

#include <stdint.h>

#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "lq_common.cuh"
#include "lq_tc_ptx.cuh"

namespace lq {

namespace dtc {

// Pipeline studies (-DLQ_PIPELINE_TRACE, a build of its own): %globaltimer stamps of every CTA's milestones, read back with
// lq_debug_read_decode_trace().  The product build compiles none of it.
#ifdef LQ_PIPELINE_TRACE
__device__ long long g_trace[1024 * 8];
#define DT_STAMP(slot)                                                                      \
  do {                                                                                      \
    if (blockIdx.x < 1024u) g_trace[blockIdx.x * 8 + (slot)] = (long long)ptx::globaltimer_ns(); \
  } while (0)
#else
#define DT_STAMP(slot) ((void)0)
#endif

constexpr int kTileBytes = 8704;
constexpr int kSets = 2;                    // dequant sets of 128 threads
constexpr int kDequant = 128 * kSets;
constexpr int kThreads = 64 + kDequant;
constexpr uint64_t kWaitLimitNs = 2000000000ull;
// The wait for tokens gathered from peer GPUs gives up well before the barrier waits of the threads that
// depend on it, so that one late peer is reported once and the rest of the CTA still finishes.
constexpr uint64_t kPeerWaitLimitNs = 1000000000ull;
constexpr int kOutI32 = 3;
constexpr int kMaxRing = 12;                // weight tiles in flight
constexpr int kMaxSplits = 8;               // portable cluster size
constexpr int kTmemCols = 256;              // two CTAs per SM share 512
constexpr int kSmemLimit = 113 * 1024;      // and the shared memory

struct Args {
  const uint8_t* blob;
  const void* x;         // [M, K]: int8 tokens, or the activations themselves (kernels that quantise)
  const float* ascale;   // [M]; null with activations
  const float* s1;       // [N]
  const void* bias;      // [N] in the output dtype, or null
  void* out;             // [M, N] (single-destination kernels; the others get a MultiOut parameter)
  int* status;
  int out_mode;          // LQ_DT_* or kOutI32
  int M, N, K, splits;   // CTAs of a cluster = k-ranges of a tile
  int ring;              // weight tiles in flight
};

template <int BN>
struct Cfg {
  static constexpr int kXStage = BN * 128;
  static constexpr int kACol = BN < 32 ? 32 : BN;             // operand stages behind the accumulator, on whole stages
  static constexpr int kNT = (kTmemCols - kACol) / 32;
};
constexpr int kQuantTokens = 8;              // limit of the quantising form: a warp per row
constexpr int kQuantChunks = 2;              // chunks of sixteen activations that a lane of it holds
__host__ __device__ inline int quant_warps(int M) { return M > 4 ? 1 : 2; }   // warps of a token row
constexpr int kMaxParts = 8 * kMaxSplits;    // parts of the row maxima: one per warp and CTA of the cluster
constexpr int kNumBars = 2 * kMaxRing + 2 * 8 + 4;

// Rows of the tile that each CTA of a cluster joins: blocks of eight rows, as evenly as they go.
__host__ __device__ inline int join_first_block(int rank, int splits) { return (16 * rank + splits - 1) / splits; }
__host__ __device__ inline int join_rows_max(int splits) { return (16 + splits - 1) / splits * 8; }

// Shared memory in bytes behind the 1024-byte aligned base.
struct Layout {
  int ws, join, bars, small, total;
};
__host__ __device__ inline Layout layout(int bn, int nk_max, int ring, int splits) {
  Layout l;
  l.ws = nk_max * bn * 128;
  l.join = l.ws + ring * kTileBytes;
  l.bars = l.join + (splits > 1 ? splits * join_rows_max(splits) * bn * 4 : 0);
  l.small = l.bars + kNumBars * 8 + 16;
  l.total = l.small + (32 + 2 * 128) * 4 + kMaxParts * 16;   // token scales, channel scales, bias, parts of the row maxima
  return l;
}

// Sixteen activations: one 16-byte chunk of quantised tokens.
template <typename XT>
struct Chunk {
  uint4 r[sizeof(XT)];
  __device__ __forceinline__ void load(const XT* p) {
#pragma unroll
    for (int i = 0; i < (int)sizeof(XT); ++i) r[i] = reinterpret_cast<const uint4*>(p)[i];
  }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < (int)sizeof(XT); ++i) r[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  __device__ __forceinline__ uint4 quantised(float scale, float inv) const {
    uint32_t q[4];
#pragma unroll
    for (int i = 0; i < (int)sizeof(XT); ++i) {
      uint32_t o[4 / sizeof(XT)];
      quant_vec<XT>(r[i], scale, inv, o);
#pragma unroll
      for (int j = 0; j < 4 / (int)sizeof(XT); ++j) q[i * (4 / sizeof(XT)) + j] = o[j];
    }
    return make_uint4(q[0], q[1], q[2], q[3]);
  }
};

template <int BN, bool MULTI, typename XT>
__global__ void __launch_bounds__(kThreads, 2)
w4a8_decode_tc_kernel(const Args args, const std::conditional_t<MULTI, MultiOut, NoMultiOut> multi) {
  constexpr bool QUANT = !std::is_same_v<XT, int8_t>;
  constexpr int NT = Cfg<BN>::kNT;
  constexpr int kXStage = Cfg<BN>::kXStage;
  const int M = args.M, S = args.splits, NW = args.ring;
  const int kt_total = args.K >> 7;
  const int rank = (int)(blockIdx.x % (unsigned)S), tile = (int)(blockIdx.x / (unsigned)S);
  const int kb = rank * kt_total / S;
  const int nk = (rank + 1) * kt_total / S - kb;
  if (threadIdx.x == 0) DT_STAMP(0);   // CTA start

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw);
  const Layout lay = layout(BN, (kt_total + S - 1) / S, NW, S);
  const uint32_t xs = base;                              // token slices of the whole k-range (1024-aligned for the swizzle)
  const uint32_t ws = base + lay.ws;                     // weight ring
  const uint32_t join = base + lay.join;                 // [splits][BN / 4][join_rows_max][4] int32
  const uint32_t bar_wfull = base + lay.bars;            // [ring] weight tile landed
  const uint32_t bar_wfree = bar_wfull + kMaxRing * 8;   // [ring] a dequant set holds the tile in registers
  const uint32_t bar_aready = bar_wfree + kMaxRing * 8;  // [NT] unpacked operand in place
  const uint32_t bar_afree = bar_aready + 8 * 8;         // [NT] the MMAs that read the operand are done
  const uint32_t bar_x = bar_afree + 8 * 8;              // the tokens are in place
  const uint32_t bar_acc = bar_x + 8;                    // the accumulator is final
  const uint32_t bar_join = bar_acc + 8;                 // the cluster's sums for this CTA's rows have landed
  const uint32_t bar_amax = bar_join + 8;                // the cluster's row maxima have landed
  const uint32_t tmem_slot = bar_amax + 8;
  volatile uint32_t* tmem_slot_p = reinterpret_cast<volatile uint32_t*>(smem + (tmem_slot - base));
  float* tok_scale = reinterpret_cast<float*>(smem + lay.small);   // [32]
  float* chan_scale = tok_scale + 32;                              // [128] of the rows this CTA stores
  float* chan_bias = chan_scale + 128;
  const uint32_t parts = base + lay.small + (32 + 2 * 128) * 4;    // [M][splits * wpr] 16 bytes: bits of a part's maximum

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int fb = join_first_block(rank, S);
  const int rows_own = (join_first_block(rank + 1, S) - fb) * 8;
  const int rows_max = join_rows_max(S);
  const int groups = (M + 3) >> 2;   // of four tokens
  const bool scaled = args.out_mode != kOutI32;
  const bool has_bias = scaled && args.bias != nullptr;
  const int wpr = quant_warps(M);

  if (threadIdx.x == 0) {
    for (int s = 0; s < NW; ++s) {
      ptx::mbar_init(bar_wfull + 8 * s, 1);
      ptx::mbar_init(bar_wfree + 8 * s, 128);
    }
    for (int t = 0; t < NT; ++t) {
      ptx::mbar_init(bar_aready + 8 * t, 128);
      ptx::mbar_init(bar_afree + 8 * t, 1);
    }
    ptx::mbar_init(bar_x, kDequant);
    ptx::mbar_init(bar_acc, 1);
    ptx::mbar_init(bar_join, 1);
    ptx::mbar_init(bar_amax, 1);
    ptx::fence_mbar_init();
    ptx::mbar_expect_tx(bar_join, (uint32_t)(S * rows_own * groups * 16));
    if (QUANT) ptx::mbar_expect_tx(bar_amax, (uint32_t)(S * wpr * M * 16));
    // Weight tiles do not depend on the previous kernel of the stream, so they are requested at once.
    ptx::mbar_expect_tx(bar_wfull, kTileBytes);
    ptx::bulk_load(ws, args.blob + ((size_t)tile * kt_total + kb) * kTileBytes, kTileBytes, bar_wfull);
  }
  __syncthreads();
  allow_dependents();         // the next kernel of the stream may start prefetching its weights
  if (S > 1) ptx::cluster_sync_all();   // every CTA's barriers are initialised

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (lane == 0) {
      const uint8_t* src = args.blob + ((size_t)tile * kt_total + kb + 1) * kTileBytes;
      int s = 1, issued = 1;   // the first tile is under way
      uint32_t ph = 0;
      bool ok = true;
      for (int i = 1; i < nk; ++i, src += kTileBytes) {
        if (i >= NW && !ptx::mbar_wait_bounded(bar_wfree + 8 * s, ph ^ 1u, kWaitLimitNs)) {
          atomicExch(args.status, 401);
          ok = false;
          break;
        }
        ptx::mbar_expect_tx(bar_wfull + 8 * s, kTileBytes);
        ptx::bulk_load(ws + s * kTileBytes, src, kTileBytes, bar_wfull + 8 * s);
        ++issued;
        if (++s == NW) {
          s = 0;
          ph ^= 1u;
        }
      }
      if (!ok) {
        // Copies in flight write shared memory: they must have landed before the CTA may exit.  (On the
        // normal path the dequant sets have waited for every one of them.)
        for (int i = issued > NW ? issued - NW : 0; i < issued; ++i)
          ptx::mbar_wait_bounded(bar_wfull + 8 * (i % NW), (uint32_t)(i / NW) & 1u, kWaitLimitNs);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ tensor memory + MMA issue
    ptx::tmem_alloc(tmem_slot, kTmemCols);
    ptx::tmem_relinquish();
    ptx::tc_fence_before();
    asm volatile("bar.sync 2, %0;" ::"n"(32 + kDequant) : "memory");   // publishes the allocation to the dequant warps
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot_p;
    {
      // The whole warp walks the loop; one elected lane issues (see ptx::elect_one).
      const bool leader = ptx::elect_one();
      constexpr uint32_t idesc = ptx::idesc_i8(BN);
      bool ok = true;
      // Scales and bias of the CTA's channels, in the MMA warp's registers (the dequant threads have none to spare).  Read only
      // behind the wait, since the kernel before may be their writer (a copy that made them contiguous, a linear whose output
      // is this one's bias).  (A hint to L2 ahead of the wait cost 1 %: 70B layers in eight shards at 8 tokens 148 -> 150 us.)
      float w_scale[4], w_bias[4];
      const long n0 = (long)tile * 128 + fb * 8 + lane;
      auto chan_ok = [&](int q) { return scaled && lane + 32 * q < rows_own && n0 + 32 * q < args.N; };
      dependency_wait();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        w_scale[q] = chan_ok(q) ? args.s1[n0 + 32 * q] : 0.f;
        w_bias[q] = (chan_ok(q) && has_bias) ? load_bias(args.bias, n0 + 32 * q, args.out_mode) : 0.f;
      }
      // The operands that were unpacked ahead of the tokens: once the tokens are there their MMAs go out back to back.
      // (With a wait and a commit around each k-tile's four MMAs a k-tile takes the issuing warp 350 cycles instead of
      // about 110.)
      const int pre = min(nk, NT);
      for (int t = 0; t < pre; ++t) ok = ok && ptx::mbar_wait_bounded(bar_aready + 8 * t, 0u, kWaitLimitNs);
      ok = ok && ptx::mbar_wait_bounded(bar_x, 0u, kWaitLimitNs);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok && leader) atomicExch(args.status, 402);
      ptx::tc_fence_after();
      if (leader) {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          if (t < pre) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              ptx::mma_i8_ts(tmem_base, tmem_base + Cfg<BN>::kACol + t * 32 + j * 8,
                             ptx::smem_desc_sw128(xs + t * kXStage + j * 32), idesc, (t > 0 || j > 0) ? 1u : 0u);
            if (t + NT < nk) ptx::tc_commit(bar_afree + 8 * t);   // a later k-tile takes this stage
          }
        }
      }
      __syncwarp();
      int t = 0;
      uint32_t ph = 1;
      for (int i = NT; i < nk; ++i) {
        if (ok && !ptx::mbar_wait_bounded(bar_aready + 8 * t, ph, kWaitLimitNs)) {
          if (leader) atomicExch(args.status, 403);
          ok = false;
        }
        __syncwarp();
        ptx::tc_fence_after();
        if (leader) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            ptx::mma_i8_ts(tmem_base, tmem_base + Cfg<BN>::kACol + t * 32 + j * 8,
                           ptx::smem_desc_sw128(xs + i * kXStage + j * 32), idesc, 1u);
          if (i + NT < nk) ptx::tc_commit(bar_afree + 8 * t);
        }
        if (++t == NT) {
          t = 0;
          ph ^= 1u;
        }
      }
      if (leader) ptx::tc_commit(bar_acc);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (lane + 32 * q >= rows_own) continue;
        chan_scale[lane + 32 * q] = w_scale[q];
        chan_bias[lane + 32 * q] = w_bias[q];
      }
    }
    __syncwarp();
    asm volatile("bar.arrive 5, %0;" ::"n"(32 + kDequant) : "memory");
    // Tensor memory is released as soon as the accumulator has been read, ahead of the join.
    asm volatile("bar.sync 4, %0;" ::"n"(32 + kDequant) : "memory");
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, kTmemCols);
  } else {
    // ------------------------------------------------------------------ dequant sets: unpack, tokens, join
    const int d = threadIdx.x - 64;
    const int set = d >> 7;                   // takes k-tiles set, set + 2, ...
    const int quad = warp & 3;                // tensor-memory lane quadrant this warp may access
    const int row = quad * 32 + lane;         // weight row inside the tile == tensor-memory lane
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    auto all_sets = []() { asm volatile("bar.sync 3, %0;" ::"n"(kDequant) : "memory"); };
    // Token rows past M are zero.
    if (M < BN) {
      const int chunks = (BN - M) * 8;
      for (int i = d; i < nk * chunks; i += kDequant)
        *reinterpret_cast<uint4*>(smem + (i / chunks) * kXStage + M * 128 + (i % chunks) * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
    asm volatile("bar.sync 2, %0;" ::"n"(32 + kDequant) : "memory");
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot_p;
    const uint32_t tmem_a = tmem_base + Cfg<BN>::kACol + lane_addr;
    bool ok = true;
    int i = set;                                  // k-tile
    uint32_t stage = (uint32_t)(set % NW), ph = (uint32_t)(set / NW) & 1u;   // its ring stage and the pass over the ring
    uint32_t t = (uint32_t)set, tph = 1u;         // its operand stage
    const uint8_t* const my_row = smem + lay.ws + row * 16;
    const uint8_t* const my_meta = smem + lay.ws + 8192 + row * 4;
    // One k-tile of this thread's weight row: nibbles and (step, offset) -> 128 INT8 ...
    uint32_t v[32];
    auto unpack = [&]() {
      if (ok && !ptx::mbar_wait_bounded(bar_wfull + 8 * stage, ph, kWaitLimitNs)) {
        atomicExch(args.status, 404);
        ok = false;
      }
      const uint8_t* p = my_row + stage * kTileBytes;
      uint4 ch[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) ch[c] = *reinterpret_cast<const uint4*>(p + c * 2048);
      const uint32_t meta = *reinterpret_cast<const uint32_t*>(my_meta + stage * kTileBytes);
      if (i + NW < nk) ptx::mbar_arrive_reader(bar_wfree + 8 * stage);   // the tile is in registers: its stage is refilled
      stage += kSets;
      if (stage >= (uint32_t)NW) {
        stage -= (uint32_t)NW;
        ph ^= 1u;
      }
      const uint32_t step0 = meta & 0xffu, a0 = __byte_perm(meta, 0u, 0x1111);
      const uint32_t step1 = __byte_perm(meta, 0u, 0x4442), a1 = __byte_perm(meta, 0u, 0x3333);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t st = c < 2 ? step0 : step1;
        const uint32_t ab = c < 2 ? a0 : a1;
        const uint32_t pk[4] = {ch[c].x, ch[c].y, ch[c].z, ch[c].w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          v[8 * c + 2 * h] = lqq_dequant4(pk[h] & 0x0F0F0F0Fu, st, ab);
          v[8 * c + 2 * h + 1] = lqq_dequant4((pk[h] >> 4) & 0x0F0F0F0Fu, st, ab);
        }
      }
    };
    // ... -> tensor memory: the operand of k-tile i.
    auto store_operand = [&]() {
      if (i >= NT && ok && !ptx::mbar_wait_bounded(bar_afree + 8 * t, tph, kWaitLimitNs)) {
        atomicExch(args.status, 406);
        ok = false;
      }
      __syncwarp();
      if (i >= NT) ptx::tc_fence_after();
      ptx::tmem_st32(tmem_a + t * 32, v);
      ptx::tc_wait_st();
      ptx::tc_fence_before();
      ptx::mbar_arrive(bar_aready + 8 * t);
      i += kSets;
      t += kSets;
      if (t >= (uint32_t)NT) {
        t -= NT;
        tph ^= 1u;
      }
    };

    // ---- before the wait for the previous kernel: operands of the first NT k-tiles, and one more in the set's registers
#pragma unroll 1
    while (i < min(nk, NT)) {
      unpack();
      store_operand();
    }
    if (i < nk) unpack();

    // ---- the previous kernel is done: the tokens of the whole k-range
    if (d == 0) DT_STAMP(1);   // operands of the first stages done
    dependency_wait();   // tokens, scales, bias and outputs belong to earlier kernels until here
    if (d == 0) DT_STAMP(2);
    if constexpr (MULTI) {
      // tokens gathered from peer GPUs: one thread waits for their flags on behalf of the others
      if (d == 0 && !peer_wait(multi.sync, kPeerWaitLimitNs)) atomicExch(args.status, 409);
      all_sets();
    }
    // In the 128-byte swizzle chunk c (16 bytes) of token row r sits at chunk c ^ (r & 7) of that row.
    if constexpr (!QUANT) {
      const int jx = d & 127;
      const int x_row = jx >> 3;
      const uint32_t x_off = (uint32_t)(x_row * 128 + (((jx & 7) ^ (x_row & 7)) << 4));
      const int8_t* src = static_cast<const int8_t*>(args.x) + (size_t)x_row * args.K + (size_t)kb * 128 + (jx & 7) * 16;
      if (d < M) tok_scale[d] = scaled ? args.ascale[d] : 0.f;
      constexpr int Q = BN / 16, U = Q == 1 ? 8 : 4;
#pragma unroll 1
      for (int j0 = set; j0 < nk; j0 += kSets * U) {
        uint4 xv[U][Q];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int q = 0; q < Q; ++q)
            if (j0 + kSets * u < nk && x_row + 16 * q < M)
              xv[u][q] = ld_stream_v4(src + (size_t)(16 * q) * args.K + (size_t)(j0 + kSets * u) * 128);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int q = 0; q < Q; ++q)
            if (j0 + kSets * u < nk && x_row + 16 * q < M)
              *reinterpret_cast<uint4*>(smem + (j0 + kSets * u) * kXStage + x_off + q * 2048) = xv[u][q];
      }
    } else {
      // Up to eight tokens, one or two warps a row (wpr); a lane holds every 32 * wpr-th chunk of sixteen activations of
      // the CTA's k-range in registers until the row's scale is known (decode_tc_quantises() keeps them to H).
      constexpr int H = kQuantChunks;
      const int m = (d >> 5) / wpr, part = (d >> 5) % wpr;
      const int c0 = part * 32 + lane, cstep = 32 * wpr, nch = m < M ? nk * 8 : 0;
      const XT* x = static_cast<const XT*>(args.x) + (size_t)m * args.K + (size_t)kb * 128;
      Chunk<XT> held[H];
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const int c = c0 + h * cstep;
        if (c < nch) held[h].load(x + (size_t)c * 16);
        else held[h].clear();
      }
      RowMax<XT> rm;
#pragma unroll
      for (int h = 0; h < H; ++h)
#pragma unroll
        for (int k = 0; k < (int)sizeof(XT); ++k) rm.take(held[h].r[k]);
      // The maxima of the row's parts (warps of all CTAs of the cluster) go to every CTA; non-negative floats are ordered
      // like their bits.
      const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(rm.value()));
      const int np = S * wpr;
      if (m < M && lane < S) {
        const uint32_t slot = parts + (uint32_t)((m * np + rank * wpr + part) * 16);
        if (S == 1) asm volatile("st.shared.b32 [%0], %1;" ::"r"(slot), "r"(top) : "memory");
        else ptx::st_async_v4(ptx::map_to_cta(slot, (uint32_t)lane), (int)top, 0, 0, 0, ptx::map_to_cta(bar_amax, (uint32_t)lane));
      }
      if (S == 1) {
        all_sets();
      } else if (ok && !ptx::mbar_wait_bounded_cluster(bar_amax, 0u, kWaitLimitNs)) {
        atomicExch(args.status, 407);
        ok = false;
      }
      if (m < M) {   // uniform over the warp
        uint32_t mine = 0u;
        for (int k = lane; k < np; k += 32) {
          uint32_t t;
          asm volatile("ld.shared.b32 %0, [%1];" : "=r"(t) : "r"(parts + (uint32_t)((m * np + k) * 16)) : "memory");
          mine = max(mine, t);
        }
        const float scale = token_scale(__uint_as_float(__reduce_max_sync(0xffffffffu, mine)));
        const float inv = __frcp_rn(scale);
        if (c0 == 0) tok_scale[m] = scale;
        uint8_t* dst = smem + m * 128;
        auto put = [&](int c, uint4 q) {
          *reinterpret_cast<uint4*>(dst + (c >> 3) * kXStage + (((c & 7) ^ (m & 7)) << 4)) = q;
        };
#pragma unroll
        for (int h = 0; h < H; ++h)
          if (c0 + h * cstep < nch) put(c0 + h * cstep, held[h].quantised(scale, inv));
      }
    }
    // written with ordinary stores: make the tokens visible to the tensor core's reads
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    ptx::mbar_arrive(bar_x);
    if (d == 0) DT_STAMP(3);   // tokens in place
#pragma unroll 1
    while (i < nk) {
      store_operand();
      if (i < nk) unpack();
    }
    // token scales (and everything above), channel scales and bias before the epilogue of any thread
    asm volatile("bar.sync 5, %0;" ::"n"(32 + kDequant) : "memory");

    // ---- epilogue: a set takes every other eight columns (tokens)
    const int units = rows_own * groups;       // (four tokens, channel) sums that this CTA joins
    int g = d / rows_own, r = d - g * rows_own;
    const int owner = ((row >> 3) * S) >> 4;   // the CTA that joins this thread's channel
    const uint32_t peer_bar = ptx::map_to_cta(bar_join, (uint32_t)owner);
    const uint32_t peer_row = ptx::map_to_cta(join, (uint32_t)owner) +
                              (uint32_t)((rank * (BN / 4) * rows_max + row - 8 * join_first_block(owner, S)) * 16);
    if (ok && !ptx::mbar_wait_bounded(bar_acc, 0u, kWaitLimitNs)) {
      atomicExch(args.status, 405);
      ok = false;
    }
    __syncwarp();
    ptx::tc_fence_after();
    if (d == 0) DT_STAMP(4);   // accumulator final
    // One channel of four consecutive tokens: scale (or not) and store.
    auto emit4 = [&](int r, int m0, int4 sum) {
      const long n = (long)tile * 128 + fb * 8 + r;
      if (n >= args.N) return;
      const float w_scale = chan_scale[r], bias = chan_bias[r];
      const int v[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (m0 + j >= M) break;
        if (!scaled) {
          reinterpret_cast<int32_t*>(args.out)[(size_t)(m0 + j) * args.N + n] = v[j];
        } else {
          const float y = lqq_scale(v[j], tok_scale[m0 + j], w_scale);
          if constexpr (MULTI) store_out_all(multi.out, m0 + j, n, y, bias, has_bias, args.out_mode);
          else store_out_bias(args.out, (size_t)(m0 + j) * args.N + n, y, bias, has_bias, args.out_mode);
        }
      }
    };
#pragma unroll 1
    for (int c0 = 8 * set; c0 < BN; c0 += 8 * kSets) {
      if (c0 >= M) break;   // uniform over the set
      int v[8];
      __syncwarp();
      ptx::tmem_ld8(tmem_base + lane_addr + c0, v);
      ptx::tc_wait_ld();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (c0 + 4 * h >= M) break;
        if (S == 1) emit4(row, c0 + 4 * h, make_int4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]));
        else
          ptx::st_async_v4(peer_row + (uint32_t)((c0 / 4 + h) * rows_max * 16), v[4 * h], v[4 * h + 1], v[4 * h + 2],
                           v[4 * h + 3], peer_bar);
      }
    }
    __syncwarp();
    ptx::tc_fence_before();
    asm volatile("bar.arrive 4, %0;" ::"n"(32 + kDequant) : "memory");
    if (S > 1) {
      if (ok && !ptx::mbar_wait_bounded_cluster(bar_join, 0u, kWaitLimitNs)) {
        atomicExch(args.status, 408);
        ok = false;
      }
      if (d == 0) DT_STAMP(5);   // sums landed
      for (int u = d; u < units; u += kDequant) {
        if (u != d) {
          g = u / rows_own;
          r = u - g * rows_own;
        }
        const int4* p = reinterpret_cast<const int4*>(smem + lay.join) + g * rows_max + r;
        int4 sum = p[0];
#pragma unroll 4
        for (int k = 1; k < S; ++k) {
          const int4 w = p[k * (BN / 4) * rows_max];
          sum.x += w.x; sum.y += w.y; sum.z += w.z; sum.w += w.w;
        }
        emit4(r, 4 * g, sum);
      }
    }
    if constexpr (MULTI) {
      // Every output store of this CTA, including those into peer memory, is ordered before the flags:
      // the barrier makes the other threads' stores visible to thread 0 (CTA scope), and the release of
      // its system-scope reduction is cumulative over them.
      all_sets();
      if (d == 0) peer_signal(multi.sync);   // red.release.sys: ordered after everything the barrier made visible
    }
    if (d == 0) DT_STAMP(6);   // outputs stored
    // Whoever has waited for the cluster's sums has nothing of its shared memory accessed any more and may exit.  A thread
    // whose wait expired stays until the other CTAs' threads have done the same or exited.
    if (S > 1 && !ok) {
      ptx::cluster_arrive();
      ptx::cluster_wait();
    }
  }
}

struct Plan {
  int tiles, splits, nk, ring, smem;   // ring 0: not a shape for this kernel
};
// Which shapes the kernel takes and how it cuts them.  Two launches should fit the machine side by side (one CTA of each
// per SM), or the second loses the head start that the design lives from: up to 74 tiles at most one CTA per SM, and at most
// 130 where clusters of three and more leave slots of a GPC empty (6144 x 4096 at 8 tokens: 2 / 3 / 4 / 6 k-ranges a tile
// = 96 / 144 / 192 / 288 CTAs 6.0 / 6.8 / 6.5 / 10.4 us).  Within that as many k-ranges as there is room for (4096 x 4096: 3 / 4 ranges
// 4.8 / 4.4; 2048 x 8192: 4 / 5 / 8 6.0 / 5.4 / 4.9).  A k-range is at most 16 k-tiles (8 above 16 tokens): the tokens of the
// range stay in shared memory, and k-tiles beyond those unpacked ahead cost 0.2 us each behind the tokens (4096 x 14336 in 28s:
// 9.8 us against the tile kernel's 9.9 with its finish pass; 7168 x 8192 in 32s 12.2 against 9.7).
// From 75 tiles on a k longer than that is cut in two all the same, with two CTAs on most SMs (here and below in us with the
// quantiser at 8 tokens, weights from HBM, this kernel / the tile kernel: 9728 x 4096 9.3 / 10.0, 12800 x 4096 10.1 / 11.7, 17408 x
// 4096 12.1 / 12.7).  With a tile on nearly every SM only one range of 9..16 k-tiles is left (148 tiles: K = 512 5.6 / 4.8, 1024 6.1 /
// 6.0, 2048 8.8 / 10.3, 4096 in two 13.8 / 13.3).  Above 16 tokens the tile kernel's whole tiles are ahead on short
// k and on many tiles (24 tokens: 4096 x 512 and its like 5.2 / 5.0, 12800 x 1024 6.1 / 5.9, 16384 x 1024 6.4 / 6.0; 8192 x 1024
// 6.0 / 6.6, 9728 x 1024 6.2 / 6.4).
static Plan plan_for(int M, int N, int K) {
  const int bn = M <= 16 ? 16 : 32;
  const int kt = K / 128;
  Plan p = {};
  p.tiles = (N + 127) / 128;
  const int sms = sm_count();
  int S = sms / p.tiles;
  if (S >= 3) S = (sms - sms / 8) / p.tiles > 2 ? (sms - sms / 8) / p.tiles : 2;
  if (S > kMaxSplits) S = kMaxSplits;
  if (S > kt / 4) S = kt / 4 > 1 ? kt / 4 : 1;
  if (S == 1 && kt > 16 && p.tiles <= sms && bn == 16) S = 2;
  if (S < 1) return p;
  if (p.tiles > sms - sms / 16 && (kt <= 8 || S > 1)) return p;
  if (bn == 32 && (kt < 8 || p.tiles > sms * 5 / 8)) return p;
  p.splits = S;
  p.nk = (kt + S - 1) / S;
  if (p.nk > (bn == 16 ? 16 : 8)) return p;
  // The ring holds the whole k-range, or an even number of stages: a stage then always belongs to the same dequant set.
  // (Otherwise a set could meet a stage whose previous tile, the other set's, has not landed yet, and the parity of
  // the pass before would let it through.)
  for (int ring = p.nk <= kMaxRing ? p.nk : kMaxRing; ring >= 1; --ring) {
    if (ring < p.nk && (ring & 1)) continue;
    p.smem = layout(bn, p.nk, ring, S).total + 1024;
    if (p.smem <= kSmemLimit) {
      p.ring = ring;
      break;
    }
  }
  // more than a third of the SM's shared memory, so that never three CTAs (of this and of the next kernels, under
  // programmatic dependent launch) share an SM: the third would wait for tensor memory
  if (p.smem < 78 * 1024) p.smem = 78 * 1024;
  return p;
}

template <int BN, bool MULTI, typename XT>
static int launch(const Args& a, const MultiOut* multi, const Plan& p, cudaStream_t st) {
  auto kern = &w4a8_decode_tc_kernel<BN, MULTI, XT>;
  static std::once_flag once[64];
  int dev = 0;
  cudaGetDevice(&dev);
  cudaError_t e = cudaSuccess;
  std::call_once(once[dev & 63], [&]() {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
  });
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.tiles * p.splits);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (p.splits > 1) {
      attr[n].id = cudaLaunchAttributeClusterDimension;
      attr[n].val.clusterDim.x = p.splits;
      attr[n].val.clusterDim.y = 1;
      attr[n++].val.clusterDim.z = 1;
    }
    if (pdl_enabled()) {
      attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    if constexpr (MULTI) e = cudaLaunchKernelEx(&cfg, kern, a, *multi);
    else e = cudaLaunchKernelEx(&cfg, kern, a, NoMultiOut{});
  }
  if (e != cudaSuccess) {
    record_cuda_error(e, "w4a8_decode_tc_kernel launch");
    return LQ_ERR_CUDA;
  }
  return check_launch("w4a8_decode_tc_kernel");
}

}  // namespace dtc

bool decode_tc_serves(int M, int N, int K) {
  return M >= 1 && M <= 32 && N >= 1 && K >= 128 && K % 128 == 0 && dtc::plan_for(M, N, K).ring > 0;
}

// Whether it also quantises its tokens: three to eight, one CTA per SM at most.  Below, the quantising GEMV is ahead (two
// tokens 1280 x 8192 5.0 against 5.1 us, 6144 x 4096 6.8 against 6.8, one token 4096 x 4096 4.8 against 5.2); above, the pass over the
// activations costs more than the quantiser's launch (4096 x 4096 at 16 tokens 6.2 us behind the quantiser, 7.6 here), and so it does
// where two CTAs share an SM (12800 x 2560 at eight tokens 8.1 and 9.0).  A lane holds two chunks of activations: with two warps a
// row (up to four tokens) any range that the plan cuts, with one up to eight k-tiles.  Four chunks a lane spilled registers and
// lengthened every such launch by 8 to 11 %, and ranges above eight k-tiles at five to eight tokens lost to the quantiser's launch
// (6144 x 4096 at eight tokens 9.6 us against 8.2).  us at four and eight tokens, weights from HBM, in the kernel / behind the
// quantiser: 1024 x 4096 4.1 / 5.2 and 4.3 / 5.4; 1280 x 8192 4.9 / 6.2 and 5.6 / 6.6; 6144 x 2048 4.8 / 5.6 and 5.4 / 5.7; 4096 x 4096
// 5.3 / 6.2 and 6.0 / 6.3; 6144 x 4096 7.4 / 7.9 at four.
bool decode_tc_quantises(int M, int N, int K) {
  if (M < 3 || M > dtc::kQuantTokens || !decode_tc_serves(M, N, K)) return false;
  const dtc::Plan p = dtc::plan_for(M, N, K);
  return p.tiles * p.splits <= sm_count() && p.nk * 8 <= dtc::kQuantChunks * 32 * dtc::quant_warps(M);
}

// What callers are told to bring for this kernel: nothing, since the join stays inside the cluster.  Only where a kernel that
// joined through global memory served before (up to 16 tokens on matrices up to 32 M weights) the all-zero buffer that
// callers were told of, and without which the call is refused, is kept; it is not touched.
size_t decode_tc_workspace_bytes(int M, int N, int K) {
  return M <= 16 && (long)N * K <= (1L << 25) ? (size_t)(2 * sm_count()) * (size_t)(16 * 128 * 8) : 0;
}
bool decode_tc_workspace_ok(int M, int N, int K, const void* ws, size_t ws_bytes) {
  const size_t need = decode_tc_workspace_bytes(M, N, K);
  return need == 0 || (ws && ws_bytes >= need);
}

// Ranges of more than eight k-tiles on wide matrices (at most four ranges a tile; 6144 x 4096, 4096 x 7680): more than half of a
// launch lies behind the wait, and on a part of the SMs only.
bool decode_tc_long_ranges(int M, int N, int K) {
  const dtc::Plan p = dtc::plan_for(M, N, K);
  return p.ring > 0 && p.nk > 8 && p.splits <= 4;
}

// CTAs a launch of this shape uses: what a consumer of the gather-by-stores epilogue must see arrive
// from every rank.
int decode_tc_grid(int M, int N, int K) {
  const dtc::Plan p = dtc::plan_for(M, N, K);
  return p.tiles * p.splits;
}

// x_dtype: LQ_DT_* of activations to quantise, or -1 for int8 tokens with their scales.  out_mode: LQ_DT_* or 3 (raw int32).
int run_decode_tc(const void* x, int x_dtype, const uint8_t* blob, const float* ascale, const float* s1, const void* bias,
                  const OutSpec& out, const PeerSync* sync, int out_mode, int M, int N, int K, void* ws, size_t ws_bytes,
                  cudaStream_t st) {
  using namespace dtc;
  if (M < 1 || M > 32 || (x_dtype >= 0 && !decode_tc_quantises(M, N, K))) return LQ_ERR_SHAPE;
  if (!decode_tc_workspace_ok(M, N, K, ws, ws_bytes)) return LQ_ERR_WORKSPACE;
  const Plan plan = plan_for(M, N, K);
  if (plan.ring == 0) return LQ_ERR_SHAPE;
  Args a;
  a.blob = blob;
  a.x = x;
  a.ascale = ascale;
  a.s1 = s1;
  a.bias = bias;
  // one plain destination with nothing to signal or wait for: the small-parameter kernels
  const bool multi = out.n != 1 || out.ld != N || out.col0 != 0 || (sync && (sync->n_signal > 0 || sync->wait));
  if (multi && (out_mode == kOutI32 || x_dtype >= 0)) return LQ_ERR_BAD_ARG;
  a.out = out.ptr[0];
  a.status = status_word();
  a.out_mode = out_mode;
  a.M = M;
  a.N = N;
  a.K = K;
  a.splits = plan.splits;
  a.ring = plan.ring;
  if (!a.status) return LQ_ERR_CUDA;
  if (x_dtype == LQ_DT_BF16) return launch<16, false, __nv_bfloat16>(a, nullptr, plan, st);
  if (x_dtype == LQ_DT_F16) return launch<16, false, __half>(a, nullptr, plan, st);
  if (x_dtype == LQ_DT_F32) return launch<16, false, float>(a, nullptr, plan, st);
  if (!multi) {
    if (M <= 16) return launch<16, false, int8_t>(a, nullptr, plan, st);
    return launch<32, false, int8_t>(a, nullptr, plan, st);
  }
  MultiOut mo;
  mo.out = out;
  mo.sync = sync ? *sync : PeerSync{};
  if (M <= 16) return launch<16, true, int8_t>(a, &mo, plan, st);
  return launch<32, true, int8_t>(a, &mo, plan, st);
}

}  // namespace lq

#ifdef LQ_PIPELINE_TRACE
// Copies the per-CTA stamps of the last launch (1024 CTAs x 8 slots of int64) to host memory.
extern "C" LQ_API int lq_debug_read_decode_trace(long long* host_dst) {
  return cudaMemcpyFromSymbol(host_dst, lq::dtc::g_trace, sizeof(long long) * 1024 * 8) == cudaSuccess ? 0 : -4;
}
#endif
