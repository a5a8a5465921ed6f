// gi_mlp_tc.cu -- fused reconstruction on the 5th-generation tensor cores: the
// 32 features of each pixel and the 32 -> 64 -> 64 -> 64 -> 3 network in one
// persistent kernel, with tcgen05.mma (BF16 operands from shared memory, FP32
// accumulators in tensor memory) and no intermediate buffer in HBM.
//
// One CTA per SM = 5 groups of 4 warps sharing one shared-memory copy of the
// weights and the SM's 512 tensor-memory columns; each group works on its own
// 128-pixel tile with its own staging buffer, mbarriers, named barrier and 96
// columns, so the groups' feature gathers and MMA rounds overlap.  In a group,
// thread i owns pixel i of the tile, which is row i of every layer's A operand and
// lane i of the accumulator, so each warp reads back and writes exactly its own 32
// lanes.  Per tile:
//   features (registers) -> A [128 x 32] -> MMA with W1 (+ the bias MMA) ->
//   tcgen05.ld, ReLU, bf16 -> A [128 x 64] -> MMA with W2 -> ... -> MMA with W4
//   (N = 16, columns 3-15 unused) -> softmax blend of the candidate estimates,
//   x exposure scale -> out.
// The A operands are in tensor memory (bf16 pairs, written by tcgen05.st beside the
// accumulator).  With A in shared memory the kernel was bound by that memory's
// bandwidth: an MMA of N = 64 reads twice as many bytes of A as of B, and every
// layer's rows were stored there first (tensor-core and load/store accesses each kept it
// 47 % busy; now 32 and 21 %).  1920 x 1080: 124.5 -> 116.5 us; what is left is the
// latency of a tile's chain, of which tensor memory holds five at once.  Loading the next
// tile's taps during the MMA rounds spilled (140 us).
// A tile is 128 consecutive pixels, so its own depth moments, normals, albedo,
// few-ray light and direct light are five contiguous byte ranges: one thread of
// the group copies them into the group's staging buffer with bulk asynchronous
// copies (TMA, cp.async.bulk, completion counted in bytes on an mbarrier) for
// the NEXT tile while the current tile runs its MMA rounds; the neighbourhood
// and mip taps are read from global memory.  (Inputs not 16-byte aligned, and a
// last partial tile, read everything from global memory.)
// One thread of a group issues the MMAs of a layer and commits them to the group's
// mbarrier, and every thread waits on it, and for the staging copies (bounded: after a
// wait that runs out the group stops at its next barrier and records an error; the CTA
// then waits for its copies in flight, frees its tensor memory and returns).  So a layer
// takes one hardware barrier of the group, before its MMAs (1920 x 1080: 127.5 -> 124.5
// us against one waiting thread and a second barrier).
//
// Layout of the operands in shared memory: core matrices of 8 rows x 16 bytes, stored as
// 128 contiguous bytes, without swizzle.  Weights are stored as they lie in memory,
// inputs x outputs, a core matrix 8 inputs by 8 consecutive outputs: K runs along the rows
// (MN-major), core matrices adjacent along the outputs are 128 bytes apart (the
// descriptor's stride byte offset) and those adjacent along K outputs * 16 bytes (its
// leading byte offset), and 16-byte accesses stage them.  The bias operand is K-major.
// One MMA consumes K = 16.
#include <cuda_bf16.h>

#include <mutex>

#include "gi_features.cuh"
#include "gi_internal.h"
#include "gi_mlp.h"
#include "gi_mlp_layout.h"

namespace gi {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kRows = 128;  // pixels per tile = MMA M = accumulator lanes
constexpr int kGroups = 5;  // tiles in flight per CTA (one CTA per SM)
constexpr int kTcThreads = 128 * kGroups;
// Tensor-memory columns: per group a 128 x 64 FP32 accumulator and a 128 x 64 bf16 A
// operand, then the four layers' constant "ones" operands (128 x 16 bf16 each).
constexpr uint32_t cA = 64, kGroupCols = cA + kHid / 2, cOnes = kGroupCols * kGroups, kOnesCols = 8, kTmemCols = 512;
static_assert(cOnes + 4 * kOnesCols <= kTmemCols, "tensor memory");

// Shared memory (bytes).  B operands: the weights, inputs x outputs and read MN-major
// (kBRows); the bias operand alone is K-major.
constexpr int tB1 = 0;                            // 32 x 64 (inputs x outputs)
constexpr int tB2 = tB1 + kHid * kIn * 2;         // 64 x 64
constexpr int tB3 = tB2 + kHid * kHid * 2;        // 64 x 64
constexpr int tB4 = tB3 + kHid * kHid * 2;        // 64 x 16 (outputs 3-15 zero)
// Biases enter the accumulators through one extra MMA per layer: A = a constant
// "ones" operand, B = the bias operand.  Bias row n holds, at k = 2L and 2L + 1,
// the bf16 high and low parts of layer L's bias b_L[n] (b - hi rounded again), so
// the MMA adds hi + lo, b to about 2^-16 relative.  Layer L's ones operand has
// 1 at k = 2L, 2L + 1 in every row and 0 elsewhere; k = 8-15 read the bias rows again.
constexpr int tBB = tB4 + kHid * kOutPad * 2;     // 64 rows x 8 k (16 bytes a row)
// Staging of a tile's own inputs: normal, albedo, few-ray light, direct light, filtered
// few-ray light (16 bytes a pixel each) and depth moments (8).
constexpr int sNormal = 0, sAlbedo = 2048, sLight = 4096, sDirect = 6144, sFiltered = 8192, sMoments = 10240;
constexpr int kStageBytes = 11264;
constexpr int tStage = tBB + kHid * 16;
constexpr int tBar = tStage + kGroups * kStageBytes;  // per group: MMA mbarrier, staging mbarrier
constexpr int tPattern = tBar + 16 * kGroups;         // features 29 and 30 of an interleave pattern's pixels
constexpr int tTmem = tPattern + 2 * 64 * 4;
constexpr int kSmemTc = tTmem + 8;
static_assert(tStage % 128 == 0 && kStageBytes % 128 == 0, "bulk copy destinations");
static_assert(tBB % 128 == 0 && tBar % 8 == 0, "alignment");

__device__ int g_tc_errors;  // waits that ran out (kept across launches)
constexpr long long kWaitCycles = 1ll << 31;  // ~1 s of SM clocks
// Bound of the first MMA-completion wait of each tile group (training: of each CTA) in a
// launch; kWaitCycles unless the test hook gi_debug_tensor_core_wait_limit shortened it (so that the
// wait runs out and the error path runs).  Every other wait keeps kWaitCycles.
__device__ long long g_tc_first_wait_cycles = kWaitCycles;

// Byte offset of element (r, k) of an R x K operand in the K-major core-matrix layout.
__device__ __forceinline__ int cm_off(int r, int k, int K) {
  return (r >> 3) * (K * 16) + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor: start address, leading and stride byte
// offsets (each stored >> 4), the fixed version bits 46-48 = 0b001, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo & 0x3FFFFu) >> 4) << 16) |
         ((uint64_t)((sbo & 0x3FFFFu) >> 4) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator (bits 4-5 = 1), BF16 A
// (bits 7-9 = 1) and B (bits 10-12 = 1), N >> 3 at bit 17, M >> 4 at bit 24; K-major
// operands, or MN-major ones with the flags below.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// K runs along the rows of A's, of B's core matrices.
constexpr uint32_t kARows = 1u << 15, kBRows = 1u << 16;

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

// The same with A in tensor memory (lane = row, a column = two consecutive k).
__device__ __forceinline__ void mma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Waits for the phase with the given parity to complete, for at most `limit` SM
// cycles (by default ~2^31, about a second); false if it did not.  The first look does
// not suspend the thread, so that a limit of a few cycles runs out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, long long limit = kWaitCycles) {
  const long long t0 = clock64();
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  while (!done) {
    if (clock64() - t0 > limit) return false;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
  }
  return true;
}

// One arrival that also expects `bytes` of asynchronous copies on the barrier.
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Bulk asynchronous copy global -> shared (TMA, no tensor map), completing
// `bytes` on the mbarrier; both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// The .sync.aligned instructions below are executed by a whole warp together.  A warp
// that waited lane by lane (mbar_wait) or left one lane's branch need not have come
// together again, so each has a __syncwarp directly before it.

// 16 consecutive FP32 columns of this thread's accumulator lane; the load and
// its completion wait are one asm statement, so no use can be scheduled between.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// 32 consecutive FP32 columns of this thread's accumulator lane (one load, one wait).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// 32-bit columns of this thread's lane written to tensor memory; tmem_st_wait before the
// barrier that precedes the MMA that reads them.
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  __syncwarp();
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  __syncwarp();
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(
          taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  __syncwarp();
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// `cols` columns of tensor memory for this CTA, by one warp: their start is stored at
// `slot` (shared memory); the CTA allocates once.
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t cols) {
  __syncwarp();
  asm volatile(
      "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n\t"
      "tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::"r"(slot),
      "r"(cols)
      : "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t start, uint32_t cols) {
  __syncwarp();
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(start), "r"(cols) : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const bf16 x = __float2bfloat16_rn(a), y = __float2bfloat16_rn(b);
  return (uint32_t)__bfloat16_as_ushort(x) | ((uint32_t)__bfloat16_as_ushort(y) << 16);
}

// ReLU of two FP32 values rounded to bf16 and packed (a in the low half), one cvt.
__device__ __forceinline__ uint32_t pack_relu_bf16(float a, float b) {
  uint32_t r;
  asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}

__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// A K x N weight matrix (bf16, row-major, N columns) as core matrices of 8 rows x 8 columns.
template <int K, int N, int THREADS>
__device__ __forceinline__ void stage_weights(uint32_t dst, const bf16* __restrict__ w) {
#pragma unroll
  for (int i = threadIdx.x; i < K * N / 8; i += THREADS) {
    const int k = i / (N / 8), c = i % (N / 8);
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(w) + i);
    st_shared_v4(dst + cm_off(k, 8 * c, N), q.x, q.y, q.z, q.w);
  }
}

// Barrier of one group's 128 threads (named barrier 1 + group); whether any of them
// passed true.
__device__ __forceinline__ bool group_any(int group, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %3, 0;\n\t"
      "barrier.cta.red.or.pred q, %1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"(1 + group), "r"(kRows), "r"((uint32_t)v)
      : "memory");
  return r != 0;
}

// Makes this group's A operand (its columns of tensor memory, written by every thread)
// visible to the tensor cores, issues the layer's bias MMA and its K/16 MMAs from the
// group's first thread and waits for them; the fence after the wait orders their
// completion before the accumulator reads.  `bad` is set on a thread whose wait runs
// out; returns false (on every thread of the group) if an earlier one did.
// `first` runs on the issuing thread after the barrier, before the MMAs.
template <int K, int N, int L, typename First>
__device__ __forceinline__ bool run_layer(uint32_t sbase, uint32_t ones, int b_off, uint32_t tmem, uint32_t bar,
                                          uint32_t& phase, int group, bool& bad, First first,
                                          long long limit = kWaitCycles) {
  tmem_st_wait();
  fence_before();
  if (group_any(group, bad)) return false;
  fence_after();
  if ((threadIdx.x & (kRows - 1)) == 0) {
    first();
    constexpr uint32_t idesc = idesc_bf16(kRows, N);
    mma_bf16_ts(tmem, ones + kOnesCols * L, smem_desc(sbase + tBB, 0, 128), idesc, 0u);
#pragma unroll
    for (int j = 0; j < K / 16; j++)
      mma_bf16_ts(tmem, tmem + cA + 8 * j, smem_desc(sbase + b_off + j * N * 32, N * 16, 128), idesc | kBRows, 1u);
    mma_commit(bar);
  }
  if (!mbar_wait(bar, phase, limit)) bad = true;
  phase ^= 1u;
  fence_after();
  return true;
}

// Hidden-layer epilogue: accumulator lane (bias included) -> ReLU -> bf16 row
// of the next A operand (K = 64).
__device__ __forceinline__ void hidden_epilogue(uint32_t lane_addr) {
#pragma unroll
  for (int c = 0; c < kHid; c += 32) {
    float v[32];
    tmem_ld32(lane_addr + c, v);
    uint32_t r[16];
#pragma unroll
    for (int k = 0; k < 16; k++) r[k] = pack_relu_bf16(v[2 * k], v[2 * k + 1]);
    tmem_st16(lane_addr + cA + c / 2, r);
  }
}

// Issues the staging copies of tile t (a full tile) into the group's buffer.
__device__ __forceinline__ void stage_tile(const FeatureArgs& a, int t, uint32_t buf, uint32_t bar) {
  const size_t p0 = (size_t)t * kRows;
  fence_async_smem();  // the group's reads of the previous tile's staging come first
  mbar_expect_tx(bar, kStageBytes);
  bulk_g2s(buf + sNormal, a.normal + 4 * p0, 16 * kRows, bar);
  bulk_g2s(buf + sAlbedo, a.albedo + 4 * p0, 16 * kRows, bar);
  bulk_g2s(buf + sLight, a.indirect[0] + 4 * p0, 16 * kRows, bar);
  bulk_g2s(buf + sDirect, a.direct + 4 * p0, 16 * kRows, bar);
  bulk_g2s(buf + sFiltered, a.filtered + 4 * p0, 16 * kRows, bar);
  bulk_g2s(buf + sMoments, a.moments + 2 * p0, 8 * kRows, bar);
}

// ROWS: the network on given feature rows (a.rows, a.row_scale; a.width = rows,
// a.height = 1) instead of the fused feature builder -- the same MMA rounds,
// epilogues and head.
template <bool ROWS>
__global__ void __launch_bounds__(kTcThreads, 1) mlp_reconstruct_kernel(const __grid_constant__ FeatureArgs a,
                                                                     const bf16* __restrict__ wb,
                                                                     const float* __restrict__ params,
                                                                     float* __restrict__ out, int staged) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5;
  const int group = tid / kRows, gtid = tid % kRows;
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar = sbase + tBar + 16 * group;  // MMA completion
  const uint32_t sbar = bar + 8;                   // staging copies
  const uint32_t stage = sbase + tStage + group * kStageBytes;
  const unsigned char* stage_p = smem + tStage + group * kStageBytes;

  stage_weights<kIn, kHid, kTcThreads>(sbase + tB1, wb + qW1);
  stage_weights<kHid, kHid, kTcThreads>(sbase + tB2, wb + qW2);
  stage_weights<kHid, kHid, kTcThreads>(sbase + tB3, wb + qW3);
  stage_weights<kHid, kOutPad, kTcThreads>(sbase + tB4, wb + qW4);
  // Bias operand: row n, k = 2L / 2L + 1 = high / low bf16 part of b_L[n].
  for (int i = tid; i < kHid * 8; i += kTcThreads) {
    const int n = i >> 3, k = i & 7, L = k >> 1;
    float b = 0.0f;
    if (L == 0) b = params[ob1 + n];
    else if (L == 1) b = params[ob2 + n];
    else if (L == 2) b = params[ob3 + n];
    else if (n < kOut) b = params[ob4 + n];
    const bf16 hi = __float2bfloat16_rn(b);
    const bf16 v = (k & 1) ? __float2bfloat16_rn(b - __bfloat162float(hi)) : hi;
    *reinterpret_cast<bf16*>(smem + tBB + n * 16 + k * 2) = v;
  }
  float* pattern = reinterpret_cast<float*>(smem + tPattern);
  if (!ROWS && tid < a.pattern * a.pattern) pattern_features(tid, a.pattern, pattern[tid], pattern[64 + tid]);
  if (gtid == 0) {
    mbar_init(bar, 1);
    mbar_init(sbar, 1);
  }
  if (warp == 0) tmem_alloc(sbase + tTmem, kTmemCols);
  fence_async_smem();  // the staged operands, for the tensor cores
  fence_before();
  __syncthreads();
  fence_after();
  // The ones operands, by the first group; the others' first MMAs wait for them.
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem + tTmem);
  const uint32_t warp_lanes = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t ones = tmem_base + cOnes;
  if (group == 0) {
#pragma unroll
    for (int L = 0; L < 4; L++) {
      uint32_t r[8];
#pragma unroll
      for (int k = 0; k < 8; k++) r[k] = k == L ? 0x3F803F80u : 0u;
      tmem_st8(ones + kOnesCols * L + warp_lanes, r);
    }
    tmem_st_wait();
  }
  fence_before();
  __syncthreads();
  fence_after();
  // This group's columns; this warp's 32 lanes of them.
  const uint32_t tmem = tmem_base + kGroupCols * group;
  const uint32_t lane_addr = tmem + warp_lanes;

  const int W = a.width, n = a.width * a.height;
  const int tiles = (n + kRows - 1) / kRows;
  const int full_tiles = n / kRows;
  const int stride = gridDim.x * kGroups;
  uint32_t phase = 0, sphase = 0;
  bool bad = false, failed = false;  // a wait of this thread, of the group ran out
  int t = blockIdx.x * kGroups + group;
  const int first_tile = t;
  bool pending = staged && t < full_tiles;  // a staging copy of tile t in flight
  if (pending && gtid == 0) stage_tile(a, t, stage, sbar);
  // The pixel's place, advanced by whole strides instead of divided anew.
  int x = (t * kRows + gtid) % W, y = (t * kRows + gtid) / W;
  const int step_x = stride * kRows % W, step_y = stride * kRows / W;
  for (; t < tiles && !failed; t += stride) {
    const int p = t * kRows + gtid;
    const int px = x, py = y;
    x += step_x;
    y += step_y;
    if (x >= W) {
      x -= W;
      y++;
    }
    float f[kIn];
    float scale = 1.0f;
    if (ROWS) {  // the row's bf16 features (exact in float) and its scale
      if (p < n) {
        const uint4* src = reinterpret_cast<const uint4*>(a.rows + (size_t)p * kIn);
#pragma unroll
        for (int c = 0; c < kIn / 8; c++) {
          const uint4 q = __ldg(src + c);
          const uint32_t w4[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int h = 0; h < 4; h++) {
            f[8 * c + 2 * h] = __uint_as_float(w4[h] << 16);
            f[8 * c + 2 * h + 1] = __uint_as_float(w4[h] & 0xFFFF0000u);
          }
        }
        if (a.row_scale) scale = __ldg(a.row_scale + p);
      } else {
#pragma unroll
        for (int i = 0; i < kIn; i++) f[i] = 0.0f;
      }
    } else if (pending) {
      if (!mbar_wait(sbar, sphase)) bad = true;
      sphase ^= 1u;
      pending = false;
      const float depth = reinterpret_cast<const float*>(stage_p + sMoments)[2 * gtid];
      const float4 n4 = reinterpret_cast<const float4*>(stage_p + sNormal)[gtid];
      const float4 al = reinterpret_cast<const float4*>(stage_p + sAlbedo)[gtid];
      const float4 li = reinterpret_cast<const float4*>(stage_p + sLight)[gtid];
      const float4 dl = reinterpret_cast<const float4*>(stage_p + sDirect)[gtid];
      const float4 fl = reinterpret_cast<const float4*>(stage_p + sFiltered)[gtid];
      pixel_features_from(a, px, py, depth, n4, al, li, dl, fl, pattern, f, scale);
    } else if (p < n) {
      pixel_features(a, px, py, pattern, f, scale);
    } else {
#pragma unroll
      for (int i = 0; i < kIn; i++) f[i] = 0.0f;
    }
    // The staging buffer takes the group's next tile once every thread has its
    // features: issued after the first layer's barrier.
    const bool prefetch = staged && t + stride < full_tiles;
    {
      uint32_t r[kIn / 2];
#pragma unroll
      for (int k = 0; k < kIn / 2; k++) r[k] = pack_bf16(f[2 * k], f[2 * k + 1]);
      tmem_st16(lane_addr + cA, r);
    }
    // The head blends candidate estimates as the network saw them (bf16).
    float cand[3][3];
#pragma unroll
    for (int ch = 0; ch < 3; ch++) {
      cand[0][ch] = __bfloat162float(__float2bfloat16_rn(f[kCand0 + ch]));
      cand[1][ch] = __bfloat162float(__float2bfloat16_rn(f[kCand1 + ch]));
      cand[2][ch] = __bfloat162float(__float2bfloat16_rn(f[kCand2 + ch]));
    }

    const int tn = t + stride;
    auto issue_next = [&] {
      if (prefetch) stage_tile(a, tn, stage, sbar);
    };
    auto nothing = [] {};
    const long long first_limit = t == first_tile ? g_tc_first_wait_cycles : kWaitCycles;
    if (!run_layer<kIn, kHid, 0>(sbase, ones, tB1, tmem, bar, phase, group, bad, issue_next, first_limit)) {
      failed = true;
      break;
    }
    pending = prefetch;
    hidden_epilogue(lane_addr);
    if (!run_layer<kHid, kHid, 1>(sbase, ones, tB2, tmem, bar, phase, group, bad, nothing)) { failed = true; break; }
    hidden_epilogue(lane_addr);
    if (!run_layer<kHid, kHid, 2>(sbase, ones, tB3, tmem, bar, phase, group, bad, nothing)) { failed = true; break; }
    hidden_epilogue(lane_addr);
    if (!run_layer<kHid, kOutPad, 3>(sbase, ones, tB4, tmem, bar, phase, group, bad, nothing)) {
      failed = true;
      break;
    }
    float v[16];
    tmem_ld16(lane_addr, v);
    if (p < n && !bad) {
      const float lo[3] = {v[0], v[1], v[2]};
      float w[3], y[3];
      head_forward(lo, cand, w, y);
      reinterpret_cast<float4*>(out)[p] = make_float4(y[0] * scale, y[1] * scale, y[2] * scale, 1.0f);
    }
  }
  failed = group_any(group, bad) || failed;
  if (failed && gtid == 0) {
    atomicAdd(&g_tc_errors, 1);
    (void)mbar_wait(bar, phase ^ 1u);    // the group's MMAs in flight, bounded
    (void)mbar_wait(sbar, sphase ^ 1u);  // and a staging copy whose wait ran out
  }
  if (pending && gtid == 0) (void)mbar_wait(sbar, sphase);  // a staging copy in flight, bounded
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0) tmem_free(tmem_base, kTmemCols);
}

// ---- Training on the tensor cores -----------------------------------------
//
// mlp_train_tc_kernel: forward with saved activations, the head's loss gradient,
// backward through every layer and the weight gradients, for 128-pixel tiles
// (persistent: one CTA of 256 threads per SM walks the batch's tiles).  Threads i
// and i + 128 own pixel i of a tile -- row i of every layer's operand and lane i of
// the accumulators -- and half of its columns each.  Products of a tile (D in tensor
// memory, M = 128):
//   forward   Z = A_l W_l             A = X / H1 / H2 / H3 (pixels x features)
//   backward  dH = dZ_l W_l^T         A = dZ (pixels x outputs)
//   gradient  dW_l += H_{l-1}^T dZ_l  the pixels are the reduction, and dW
//                                     accumulates over every tile of the CTA in
//                                     tensor memory (M = 128: rows past the layer's
//                                     inputs read the next bytes and are never read
//                                     back)
//             db_l += 1^T dZ_l        a constant operand of ones
// Every operand is stored once, as 8 x 8 core matrices of rows (pixels, or a weight's
// inputs) by 8 consecutive columns, and the descriptors name its K axis: along the
// columns (K-major: forward and backward A, backward B) or along the rows (MN-major:
// forward B, both gradient operands).
// Epilogues (two threads per pixel): bias and ReLU to bf16 (forward), the head's loss
// gradient (layer 4), the ReLU mask of the backward (dZ = dH where H > 0).  A layer's
// gradient products run behind the next epilogue: only the layer's accumulator is
// waited for, and each layer has its own dZ.  At the end each CTA adds its gradient
// sums to `grads` (16-byte reductions) and its loss.
// Arithmetic: bf16 operands (inputs, weights, hidden activations, the logits'
// gradient and the masked hidden gradients), FP32 accumulation, FP32 bias and
// head; the sums run in the tensor cores' order.
//
// Bound by latency: a tile is a chain of 8 products and epilogues, and batches to
// 19 456 pixels are one tile per SM.  16 384 rows: 71.7 -> 18.5 us against 128 threads a tile, transposed
// copies of every operand, column sums in a loop and one addition per value.
constexpr int kTrThreads = 256;
constexpr int uW1 = 0;                             // weights, inputs x outputs
constexpr int uW2 = uW1 + kHid * kIn * 2;
constexpr int uW3 = uW2 + kHid * kHid * 2;
constexpr int uW4 = uW3 + kHid * kHid * 2;         // 64 x 16 (outputs 3-15 zero)
constexpr int uX = uW4 + kHid * kOutPad * 2;       // 128 x 32
constexpr int uH1 = uX + kRows * kIn * 2;          // 128 x 64 each
constexpr int uH2 = uH1 + kRows * kHid * 2;
constexpr int uH3 = uH2 + kRows * kHid * 2;
constexpr int uDY = uH3 + kRows * kHid * 2;        // 128 x 16 (outputs 3-15 zero)
constexpr int uZ1 = uDY + kRows * kOutPad * 2;     // 128 x 64 each: dZ
constexpr int uZ2 = uZ1 + kRows * kHid * 2;
constexpr int uZ3 = uZ2 + kRows * kHid * 2;
constexpr int uOne = uZ3 + kRows * kHid * 2;       // one core matrix of ones
constexpr int uBias = uOne + 128;                  // b1, b2, b3 (64 floats each), b4
constexpr int uBar = uBias + (3 * kHid + 4) * 4;   // two mbarriers: the layer's accumulator; a tile's gradients
constexpr int uFail = uBar + 16;
constexpr int uTmem = uFail + 4;
constexpr int kSmemTrainTc = uTmem + 4;
// A gradient operand of M = 128 rows reads 16 core matrices (2 KB) from each of its
// pixel groups' starts.
static_assert(uH3 + kRows * kHid * 2 + 2048 <= kSmemTrainTc, "gradient operand reads stay in shared memory");
static_assert(uX % 128 == 0 && uDY % 128 == 0 && uZ1 % 128 == 0 && uOne % 128 == 0 && uBias % 16 == 0 &&
                  uBar % 8 == 0,
              "alignment");
static_assert(ob1 % 4 == 0 && oW2 % 4 == 0 && ob2 % 4 == 0 && oW3 % 4 == 0 && ob3 % 4 == 0 && oW4 % 4 == 0,
              "16-byte reductions");
// Tensor-memory columns: the layer accumulator, the weight-gradient sums and the
// bias-gradient sums (every row the same).
constexpr uint32_t cZ = 0, cW1 = 64, cW2 = 128, cW3 = 192, cW4 = 256, cB3 = 288, cB2 = 352, cB1 = 416, cB4 = 480,
                   kTrTmemCols = 512;

// An operand in shared memory: its start, the distances of core matrices adjacent along
// K and along M (or N), and whether K runs along the rows (MN-major).  An MMA consumes
// two core matrices along K.
struct Operand {
  uint32_t at, k, mn;
  bool rows;
};
template <int W> __device__ __forceinline__ Operand along_columns(uint32_t at) { return Operand{at, 128, W * 16, false}; }
template <int W> __device__ __forceinline__ Operand along_rows(uint32_t at) { return Operand{at, W * 16, 128, true}; }

// K/16 MMAs of A (M = 128 x K) and B (N x K) into D; `first` clears D.
template <int K, int N>
__device__ __forceinline__ void mma_chain(uint32_t d, const Operand& a, const Operand& b, bool first) {
  const uint32_t idesc = idesc_bf16(kRows, N) | (a.rows ? kARows : 0u) | (b.rows ? kBRows : 0u);
#pragma unroll
  for (int j = 0; j < K / 16; j++)
    mma_bf16(d, smem_desc(a.at + 2 * j * a.k, a.k, a.mn), smem_desc(b.at + 2 * j * b.k, b.k, b.mn), idesc,
             (first && j == 0) ? 0u : 1u);
}

__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 q;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w)
               : "r"(addr)
               : "memory");
  return q;
}

// *p += v for four consecutive floats (16-byte aligned), one reduction.
__device__ __forceinline__ void red_add4(float* p, float a, float b, float c, float d) {
  asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
               : "memory");
}
__device__ __forceinline__ void red_add32(float* p, const float (&v)[32]) {
#pragma unroll
  for (int j = 0; j < 32; j += 4) red_add4(p + j, v[j], v[j + 1], v[j + 2], v[j + 3]);
}

__global__ void __launch_bounds__(kTrThreads, 1) mlp_train_tc_kernel(const bf16* __restrict__ feats,
                                                                   const float* __restrict__ targets,
                                                                   const float* __restrict__ scale, int n,
                                                                   const bf16* __restrict__ wb,
                                                                   const float* __restrict__ params,
                                                                   float* __restrict__ grads,
                                                                   float* __restrict__ loss, int* __restrict__ failed_ctas,
                                                                   int loss_kind) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t sbase = smem_u32(smem);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int row = tid & (kRows - 1), half = tid >> 7;  // the thread's pixel, and its half of the columns
  const uint32_t layer_bar = sbase + uBar, grad_bar = layer_bar + 8;
  volatile int* fail = reinterpret_cast<volatile int*>(smem + uFail);
  const float* bias = reinterpret_cast<const float*>(smem + uBias);
  const long long first_limit = g_tc_first_wait_cycles;

  stage_weights<kIn, kHid, kTrThreads>(sbase + uW1, wb + qW1);
  stage_weights<kHid, kHid, kTrThreads>(sbase + uW2, wb + qW2);
  stage_weights<kHid, kHid, kTrThreads>(sbase + uW3, wb + qW3);
  stage_weights<kHid, kOutPad, kTrThreads>(sbase + uW4, wb + qW4);
  if (tid < 3 * kHid + kOut) {
    const int l = tid >> 6, at = tid & (kHid - 1);
    const int from = (l == 0 ? ob1 : l == 1 ? ob2 : l == 2 ? ob3 : ob4) + at;
    reinterpret_cast<float*>(smem + uBias)[tid] = __ldg(params + from);
  }
  if (tid < 64) reinterpret_cast<bf16*>(smem + uOne)[tid] = __float2bfloat16_rn(1.0f);
  if (tid == 0) {
    mbar_init(layer_bar, 1);
    mbar_init(grad_bar, 1);
    *fail = 0;
  }
  if (warp == 0) tmem_alloc(sbase + uTmem, kTrTmemCols);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + uTmem);
  const uint32_t lane = tmem + ((uint32_t)((warp & 3) * 32) << 16);  // this warp's 32 accumulator lanes
  const uint32_t mine = lane + 32 * half;                            // and its columns of a 64-column accumulator
  uint32_t layer_phase = 0, grad_phase = 0;
  bool first = true;
  float lsum = 0.0f;

  // A bounded wait of every thread.  One that runs out is recorded and the tile goes on
  // (with values that are not used), so that the threads stay together; the later
  // waits then return at once.
  auto wait = [&](uint32_t bar, uint32_t& phase, long long limit = kWaitCycles) {
    if (!*fail && !mbar_wait(bar, phase, limit)) *fail = 1;
    phase ^= 1u;
  };
  // Shared-memory writes -> the tensor cores -> `layer` (the layer's accumulator) and
  // `grad` (left running) on thread 0 -> wait for the accumulator.
  auto mma_round = [&](auto layer, auto grad, long long limit = kWaitCycles) {
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
    if (tid == 0) {
      layer();
      mma_commit(layer_bar);
      grad();
    }
    wait(layer_bar, layer_phase, limit);
    fence_after();
  };
  auto nothing = [] {};
  // Layer accumulator -> + bias -> ReLU -> bf16 row of the next operand.
  auto forward_epilogue = [&](int buf, const float* b) {
    float v[32];
    tmem_ld32(mine + cZ, v);
#pragma unroll
    for (int c = 0; c < 32; c += 8) {
      const float4 b0 = *reinterpret_cast<const float4*>(b + 32 * half + c);
      const float4 b1 = *reinterpret_cast<const float4*>(b + 32 * half + c + 4);
      st_shared_v4(sbase + buf + cm_off(row, 32 * half + c, kHid), pack_relu_bf16(v[c] + b0.x, v[c + 1] + b0.y),
                   pack_relu_bf16(v[c + 2] + b0.z, v[c + 3] + b0.w),
                   pack_relu_bf16(v[c + 4] + b1.x, v[c + 5] + b1.y),
                   pack_relu_bf16(v[c + 6] + b1.z, v[c + 7] + b1.w));
    }
  };
  // dH (accumulator) masked by the ReLU of the layer's output H (its bf16 row) -> dZ.
  auto backward_epilogue = [&](int h_buf, int z_buf) {
    float v[32];
    tmem_ld32(mine + cZ, v);
#pragma unroll
    for (int c = 0; c < 32; c += 8) {
      const int at = cm_off(row, 32 * half + c, kHid);
      const uint4 q = ld_shared_v4(sbase + h_buf + at);
      const uint32_t h[4] = {q.x, q.y, q.z, q.w};
      uint32_t z[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const float g0 = (h[k] & 0xFFFFu) && !(h[k] & 0x8000u) ? v[c + 2 * k] : 0.0f;  // bf16 > 0
        const float g1 = (h[k] >> 16) && !(h[k] & 0x80000000u) ? v[c + 2 * k + 1] : 0.0f;
        z[k] = pack_bf16(g0, g1);
      }
      st_shared_v4(sbase + z_buf + at, z[0], z[1], z[2], z[3]);
    }
  };
  const Operand ones{sbase + uOne, 0, 0, false};

  const int tiles = (n + kRows - 1) / kRows;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int p = t * kRows + row;
    const bool valid = p < n;
    // Half the feature row each; the targets, divided by the exposure scale, of the
    // threads that evaluate the head.
    uint4 x[2];
    float T[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int c = 0; c < 2; c++)
      x[c] = valid ? __ldg(reinterpret_cast<const uint4*>(feats + (size_t)p * kIn) + 2 * half + c)
                   : make_uint4(0u, 0u, 0u, 0u);
    if (valid && half == 0) {
      const float sc = scale ? __ldg(scale + p) : 1.0f;
      const float4 q = __ldg(reinterpret_cast<const float4*>(targets) + p);
      T[0] = scale ? q.x / sc : q.x;
      T[1] = scale ? q.y / sc : q.y;
      T[2] = scale ? q.z / sc : q.z;
      T[3] = q.w;
    }
    if (!first) wait(grad_bar, grad_phase);  // the previous tile's operands are free
#pragma unroll
    for (int c = 0; c < 2; c++)
      st_shared_v4(sbase + uX + cm_off(row, 16 * half + 8 * c, kIn), x[c].x, x[c].y, x[c].z, x[c].w);

    mma_round([&] { mma_chain<kIn, kHid>(tmem + cZ, along_columns<kIn>(sbase + uX), along_rows<kHid>(sbase + uW1), true); },
              nothing, first ? first_limit : kWaitCycles);
    forward_epilogue(uH1, bias);
    mma_round([&] { mma_chain<kHid, kHid>(tmem + cZ, along_columns<kHid>(sbase + uH1), along_rows<kHid>(sbase + uW2), true); },
              nothing);
    forward_epilogue(uH2, bias + kHid);
    mma_round([&] { mma_chain<kHid, kHid>(tmem + cZ, along_columns<kHid>(sbase + uH2), along_rows<kHid>(sbase + uW3), true); },
              nothing);
    forward_epilogue(uH3, bias + 2 * kHid);
    mma_round(
        [&] { mma_chain<kHid, kOutPad>(tmem + cZ, along_columns<kHid>(sbase + uH3), along_rows<kOutPad>(sbase + uW4), true); },
        nothing);
    // Head: the loss gradient at the logits -> dY.
    if (half == 0) {
      float z[16];
      tmem_ld16(lane + cZ, z);
      const float lo[3] = {z[0] + bias[3 * kHid], z[1] + bias[3 * kHid + 1], z[2] + bias[3 * kHid + 2]};
      float c[3][3], d[3] = {0.0f, 0.0f, 0.0f};
      auto xval = [&](int k) {
        return __bfloat162float(*reinterpret_cast<const bf16*>(smem + uX + cm_off(row, k, kIn)));
      };
#pragma unroll
      for (int ch = 0; ch < 3; ch++) {
        c[0][ch] = xval(kCand0 + ch);
        c[1][ch] = xval(kCand1 + ch);
        c[2][ch] = xval(kCand2 + ch);
      }
      const float l = head_loss_grad_logits(lo, c, T, d, loss_kind);
      if (valid) lsum += l;
      else d[0] = d[1] = d[2] = 0.0f;
      st_shared_v4(sbase + uDY + cm_off(row, 0, kOutPad), pack_bf16(d[0], d[1]), pack_bf16(d[2], 0.0f), 0u, 0u);
      st_shared_v4(sbase + uDY + cm_off(row, 8, kOutPad), 0u, 0u, 0u, 0u);
    }
    // Layer 4: dH3 = dY W4^T; dW4 += H3^T dY.
    mma_round(
        [&] { mma_chain<kOutPad, kHid>(tmem + cZ, along_columns<kOutPad>(sbase + uDY), along_columns<kOutPad>(sbase + uW4), true); },
        [&] {
          mma_chain<kRows, kOutPad>(tmem + cW4, along_rows<kHid>(sbase + uH3), along_rows<kOutPad>(sbase + uDY), first);
          mma_chain<kRows, kOutPad>(tmem + cB4, ones, along_rows<kOutPad>(sbase + uDY), first);
        });
    backward_epilogue(uH3, uZ3);
    // Layer 3: dH2 = dZ3 W3^T; dW3 += H2^T dZ3.
    mma_round(
        [&] { mma_chain<kHid, kHid>(tmem + cZ, along_columns<kHid>(sbase + uZ3), along_columns<kHid>(sbase + uW3), true); },
        [&] {
          mma_chain<kRows, kHid>(tmem + cW3, along_rows<kHid>(sbase + uH2), along_rows<kHid>(sbase + uZ3), first);
          mma_chain<kRows, kHid>(tmem + cB3, ones, along_rows<kHid>(sbase + uZ3), first);
        });
    backward_epilogue(uH2, uZ2);
    // Layer 2: dH1 = dZ2 W2^T; dW2 += H1^T dZ2.
    mma_round(
        [&] { mma_chain<kHid, kHid>(tmem + cZ, along_columns<kHid>(sbase + uZ2), along_columns<kHid>(sbase + uW2), true); },
        [&] {
          mma_chain<kRows, kHid>(tmem + cW2, along_rows<kHid>(sbase + uH1), along_rows<kHid>(sbase + uZ2), first);
          mma_chain<kRows, kHid>(tmem + cB2, ones, along_rows<kHid>(sbase + uZ2), first);
        });
    backward_epilogue(uH1, uZ1);
    // Layer 1: dW1 += X^T dZ1.  The tile's last products: the next tile waits for them.
    fence_async_smem();
    fence_before();
    const bool stop = __syncthreads_or(*fail) != 0;
    fence_after();
    if (tid == 0) {
      mma_chain<kRows, kHid>(tmem + cW1, along_rows<kIn>(sbase + uX), along_rows<kHid>(sbase + uZ1), first);
      mma_chain<kRows, kHid>(tmem + cB1, ones, along_rows<kHid>(sbase + uZ1), first);
      mma_commit(grad_bar);
    }
    first = false;
    if (stop) break;
  }
  // Every product in flight, bounded: a tile's commit covers all before it.  After a wait
  // that ran out the previous tile's may still be open, and is waited for first.
  if (!first && *fail) (void)mbar_wait(grad_bar, grad_phase ^ 1u);
  if (!first && !mbar_wait(grad_bar, grad_phase)) *fail = 1;
  fence_before();
  __syncthreads();
  fence_after();
  const bool failed = *fail != 0;
  if (failed && tid == 0) {  // its sums are left out: the batch is reported as failed
    atomicAdd(&g_tc_errors, 1);
    atomicAdd(failed_ctas, 1);
  }
  if (!failed && !first) {
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    if (half == 0 && (tid & 31) == 0) atomicAdd(loss, lsum);
    float v[32];
    if ((warp & 3) < 2) {  // weight-gradient rows: lane r of the accumulators = input feature r
      if ((warp & 1) == 0) {
        tmem_ld32(mine + cW1, v);
        red_add32(grads + oW1 + row * kHid + 32 * half, v);
      }
      tmem_ld32(mine + cW2, v);
      red_add32(grads + oW2 + row * kHid + 32 * half, v);
      tmem_ld32(mine + cW3, v);
      red_add32(grads + oW3 + row * kHid + 32 * half, v);
    } else if ((warp & 3) == 2) {  // bias gradients: any row
      tmem_ld32(mine + cB1, v);
      if ((tid & 31) == 0) red_add32(grads + ob1 + 32 * half, v);
      tmem_ld32(mine + cB2, v);
      if ((tid & 31) == 0) red_add32(grads + ob2 + 32 * half, v);
      tmem_ld32(mine + cB3, v);
      if ((tid & 31) == 0) red_add32(grads + ob3 + 32 * half, v);
    }
    float u[16];
    if (half == 0 && (warp & 3) < 2) {
      tmem_ld16(lane + cW4, u);
      for (int j = 0; j < kOut; j++) atomicAdd(grads + oW4 + row * kOut + j, u[j]);
    } else if (half == 0 && (warp & 3) == 2) {
      tmem_ld16(lane + cB4, u);
      if ((tid & 31) == 0)
        for (int j = 0; j < kOut; j++) atomicAdd(grads + ob4 + j, u[j]);
    }
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0) tmem_free(tmem, kTrTmemCols);
}

std::mutex g_tc_mutex;
int g_tc_grid[64] = {0};  // persistent grid per device (0 = not set up)

}  // namespace

// The reconstruction kernels' shared-memory attributes, set once per device, and
// their persistent grid: one CTA per SM (each allocates all 512 tensor-memory columns).
static int reconstruct_grid_cap(int* cap) {
  int dev = 0;
  int e = check_cuda(cudaGetDevice(&dev), "reconstruct: device");
  if (e) return e;
  std::lock_guard<std::mutex> lock(g_tc_mutex);
  if (dev >= 64) return fail(GI_ERR_UNSUPPORTED, "reconstruct: device index");
  if (!g_tc_grid[dev]) {
    int sms = 0, optin = 0, per_sm = kSmemTc + 1024;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    if (optin < kSmemTc) return fail(GI_ERR_UNSUPPORTED, "reconstruct: not enough shared memory per block");
    for (auto kernel : {mlp_reconstruct_kernel<false>, mlp_reconstruct_kernel<true>}) {
      e = check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemTc),
                     "reconstruct: smem attribute");
      if (e) return e;
      // Shared memory for the one CTA; the rest of the SM's storage is L1 for the taps.
      e = check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                          (kSmemTc + 1024) * 100 / per_sm + 1),
                     "reconstruct: carveout");
      if (e) return e;
    }
    g_tc_grid[dev] = sms;
  }
  *cap = g_tc_grid[dev];
  return GI_OK;
}

int launch_reconstruct(const FeatureArgs& a, const __nv_bfloat16* wb, const float* params, float* out,
                       cudaStream_t stream) {
  int grid_cap = 0;
  int e = reconstruct_grid_cap(&grid_cap);
  if (e) return e;
  const int n = a.width * a.height;
  const int tiles = (n + kRows - 1) / kRows;
  const int ctas = (tiles + kGroups - 1) / kGroups;
  const int grid = ctas < grid_cap ? ctas : grid_cap;
  if (grid <= 0) return GI_OK;
  // The staging copies need 16-byte aligned sources.
  const int staged = aligned16(a.normal) && aligned16(a.albedo) && aligned16(a.indirect[0]) && aligned16(a.direct) &&
                     aligned16(a.moments) && aligned16(a.filtered);
  mlp_reconstruct_kernel<false><<<grid, kTcThreads, kSmemTc, stream>>>(a, wb, params, out, staged);
  GI_CHECK_LAUNCH("mlp_reconstruct_kernel");
  count_launches(1);
  return GI_OK;
}

int launch_forward_tc(const __nv_bfloat16* rows, const float* scale, int n, const __nv_bfloat16* wb,
                      const float* params, float* out, cudaStream_t stream) {
  if (n <= 0) return GI_OK;
  int grid_cap = 0;
  int e = reconstruct_grid_cap(&grid_cap);
  if (e) return e;
  FeatureArgs a{};
  a.width = n;
  a.height = 1;
  a.pattern = 1;
  a.rows = rows;
  a.row_scale = scale;
  const int tiles = (n + kRows - 1) / kRows;
  const int ctas = (tiles + kGroups - 1) / kGroups;
  const int grid = ctas < grid_cap ? ctas : grid_cap;
  mlp_reconstruct_kernel<true><<<grid, kTcThreads, kSmemTc, stream>>>(a, wb, params, out, 0);
  GI_CHECK_LAUNCH("mlp_reconstruct_kernel (rows)");
  count_launches(1);
  return GI_OK;
}

int launch_train_tc(const __nv_bfloat16* feats, const float* targets, const float* scale, int n,
                    const __nv_bfloat16* wb, const float* params, float* grads, float* loss, int* failed_ctas,
                    int loss_kind, cudaStream_t stream) {
  int dev = 0;
  int e = check_cuda(cudaGetDevice(&dev), "train: device");
  if (e) return e;
  static bool attr_set[64] = {};
  int sms = 0;
  {
    std::lock_guard<std::mutex> lock(g_tc_mutex);
    if (dev >= 64) return fail(GI_ERR_UNSUPPORTED, "train: device index");
    if (!attr_set[dev]) {
      int optin = 0;
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
      if (optin < kSmemTrainTc) return fail(GI_ERR_UNSUPPORTED, "train: not enough shared memory per block");
      e = check_cuda(cudaFuncSetAttribute(mlp_train_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          kSmemTrainTc),
                     "train: smem attribute");
      if (e) return e;
      attr_set[dev] = true;
    }
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  const int tiles = (n + kRows - 1) / kRows;
  const int grid = tiles < sms ? tiles : sms;  // one CTA per SM: all 512 tensor-memory columns
  if (grid <= 0) return GI_OK;
  mlp_train_tc_kernel<<<grid, kTrThreads, kSmemTrainTc, stream>>>(feats, targets, scale, n, wb, params, grads,
                                                                   loss, failed_ctas, loss_kind);
  GI_CHECK_LAUNCH("mlp_train_tc_kernel");
  count_launches(1);
  return GI_OK;
}

int reconstruct_wait_limit(long long cycles) {
  const long long v = cycles > 0 ? cycles : kWaitCycles;
  return check_cuda(cudaMemcpyToSymbol(g_tc_first_wait_cycles, &v, sizeof(v)), "reconstruct: wait limit");
}

int reconstruct_errors(int* count) {
  return check_cuda(cudaMemcpyFromSymbol(count, g_tc_errors, sizeof(int)), "reconstruct: error count");
}

}  // namespace gi
