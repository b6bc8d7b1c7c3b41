// Block-cooperative tensor-core GEMMs (decode steps, prompts):
//     Y[m, n] = sum_k X[m, k] * W[n, k]          W row-major with k contiguous, like every weight of the reference
//
//   * FP8:  W and X are OCP E4M3 bytes with per-tensor scales (the reference's FP8MatMul, custom_ops/matmul_fp8.cpp:885-1091,
//           in the E4M3 form): tcgen05.mma kind::f8f6f4, fp32 accumulation in tensor memory, scales applied in the epilogue.
//   * FP16: W and X fp16, tcgen05.mma kind::f16, with the bias, GELU, residual, squared-ReLU and SwiGLU epilogues: the same kernel
//           with 64 elements of k per 128-byte operand row.
//   * BF16: W and X bfloat16, tcgen05.mma kind::f16, bf16 or fp32 output with the epilogues of dense_out.cuh: the same kernel as FP8
//           with 64 elements of k per 128-byte operand row.  Grouped: every tile of activation rows names its weight matrix.
//   * INT4: W is packed nibbles with fp16 group scales (utils/param_handler/precision_strategy.py:24-42,56-60).  Transform
//           warps turn every staged tile into fp16(q) * scale - one fp16 rounding per weight, exactly the reference's
//           Int4ToHalf (custom_ops/int4_to_half_codelets.cpp:18-38) - in tensor memory, where the MMA takes its A operand from;
//           tcgen05.mma kind::f16 multiplies it with the fp16 activations, fp32 accumulation.
//
// The weights are the big operand, so they take the 128-row M side of the instruction and the activation rows the N side
// (16 .. 256 columns): the kernel computes Y^T tiles, D[128 weight rows, mb activation rows] in tensor memory.
// One CTA per (128 weight rows, k-slice).  Weights of a model are tiled once at load time (pt_gemm_repack) so that the tile of
// every stage is one contiguous run in global memory, already in the shared-memory image the tensor core wants: the producer
// fetches it with a single bulk copy (measured on B200: a 2-D TMA box of 128 strided rows costs about 0.65 us per box whatever
// the row width, which caps an SM near 25 GB/s; contiguous bulk copies stream at the HBM rate).  The activations (few rows) and
// the row-major weights of the plain FP8MatMul op come through tiled TMA (cp.async.bulk.tensor; this GPU's memory only, no
// multicast).  One thread issues the MMAs and hands stages back with tcgen05.commit; the other warps convert (INT4: a deep ring
// of raw nibble tiles feeds a few slots of fp16 weights in tensor memory) and run the epilogue (tcgen05.ld, scale, fp16, coalesced
// stores along n).  k-slices of one tile are the blocks of a cluster, which sum them in slice order (deterministic).
// Every wait on an mbarrier is bounded: on a time-out the CTA raises the error flag, skips its remaining waits, stays until nothing is on its way to its shared
// memory any more, and frees its tensor memory.  Waits for tensor memory and for the blocks of a cluster have no limit and end by construction (gemm_plan.h).
#include <cuda.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "dense_out.cuh"
#include "fp16_out.cuh"
#include "gemm_plan.h"
#include "mbarrier.cuh"

namespace pt {
namespace few {   // gemm_few.cu: small products of few activation rows
bool takes(const pt_gemm_args &a);
cudaError_t run(const pt_gemm_args &a, int out_ld, cudaStream_t st);
}  // namespace few
namespace tc {

// What becomes of a finished sum of the kernels with fp16 output (FP8, INT4, FP16).
struct Fp16Out {
  __half *out;
  const __half *residual, *bias, *gate;
  int out_ld, N, epilogue, halve;
  float scale;
};
constexpr int MAX_PARTS = 3;
// How the sums of a tile's k-slices come together, if it has any.  (Instantiations for both, since a kernel with both is slower for either; none for whole tiles: products
// that follow one another in a step are sliced or not, and found each other's code no longer in the instruction cache, ChatGLM2 at 8 rows 2.45 -> 2.48 ms.)
enum Sums { SENT, FETCHED };

// (A launch's parameters come from memory: what every block reads first lies together, and the outputs, of which it reads one set, at the end.)
struct GemmParams {
  int M, N, K;
  int mb;                 // activation rows per CTA (multiple of 16, at most 256)
  int group;              // INT4 scale group along k
  int kb_per_split, n_kb; // k blocks (of 128 bytes of operand row) per k-slice / in total
  int ksplit, stages, raw_stages;
  int tmem_columns;       // tensor memory of a CTA
  int w_tiled;            // weights tiled by pt_gemm_repack (one contiguous tile per stage) instead of row-major
  int pdl;                // programmatic dependent launch (tiled weights): they are fetched before the producer of x has finished
  int x_warps;            // few activation rows: warps fetch them, not TMA
  int sum_offset;         // where in a block's shared memory the slices of its share of a tile arrive (0: in place of the operands)
  int n_tiles;            // tiles of 128 weight rows
  int n_parts, part_tile[MAX_PARTS];   // FP16: products that share a launch, part s from tile part_tile[s] on with activation rows s M ..
  const unsigned char *w; // tiled weights (w_tiled)
  const unsigned char *x; // activations, rows of x_pitch bytes
  size_t x_pitch;
  const __half *scales;   // INT4: [N][K / group]
  int *error_flag;
  const int *group_of;    // BF16, grouped: the weight matrix of every tile of mb rows (negative: none)
  const int *group_used;  // ... and how many of its rows are in use (null: all)
  size_t group_stride;    // bytes between weight matrices
  DenseOut dense;         // BF16: what becomes of a finished sum
  Fp16Out o[MAX_PARTS];   // the others: of every part
};

// ------------------------------------------------------------------------------------------ PTX
__device__ __forceinline__ uint32_t sa(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// One lane of the (whole) warp.  The single-thread roles go by it: the compiler then knows that one lane runs, and gives the instructions
// that take uniform registers (bulk copies, MMAs, commits) their operands without a loop over the lanes.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst), "l"(map),
               "r"(bar), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// D[tmem] (+)= A[smem desc] * B[smem desc]
template <bool F8>
__device__ __forceinline__ void umma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  if (F8)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(d_tmem),
                 "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u)
                 : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(d_tmem),
                 "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u)
                 : "memory");
}
// The same with A in tensor memory (lane = row, a column holds two consecutive k), fp16.
__device__ __forceinline__ void umma_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(d_tmem),
               "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u)
               : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
               "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
               "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
               "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]),
               "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Distributed shared memory of a cluster: a local address in block `rank`, a store there that arrives at that block's barrier, and all threads of all
// its blocks meeting.
__device__ __forceinline__ uint32_t in_block(uint32_t local, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  return a;
}
__device__ __forceinline__ void send4(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1,%2,%3,%4}, [%5];" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar) : "memory");
}
// (The aligned forms want whole warps: lanes that leave a loop at different times are brought together first.)
__device__ __forceinline__ void cluster_arrive() { __syncwarp(); asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { __syncwarp(); asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Ordinary stores to shared memory come before what the tensor core and TMA read and write there.
__device__ __forceinline__ void fence_operands() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// The mbarrier gets one arrival once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                 "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(taddr)
               : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
               "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                 "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
                 "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
                 "=r"(v[31])
               : "r"(taddr)
               : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor of a K-major operand tile stored as rows of 128 bytes with the 128-byte swizzle (the layout
// TMA writes with CU_TENSOR_MAP_SWIZZLE_128B and the transform warps reproduce): 8-row groups are 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);   // start address, 16-byte units
  d |= (uint64_t)1 << 16;                    // leading byte offset (unused for swizzled K-major operands)
  d |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;                    // descriptor version of this architecture
  d |= (uint64_t)2 << 61;                    // 128-byte swizzle
  return d;
}
// Instruction descriptor: fp32 accumulator, both operands K-major, M = 128, N = n.
__host__ __device__ inline uint32_t instr_desc(bool bf16, int n) {
  uint32_t d = 0;
  d |= 1u << 4;                 // D format: fp32
  d |= (bf16 ? 1u : 0u) << 7;   // A format: E4M3 (f8f6f4) / F16 or BF16 (f16)
  d |= (bf16 ? 1u : 0u) << 10;  // B format: the same
  d |= (uint32_t)(n >> 3) << 17;
  d |= (uint32_t)(BM >> 4) << 24;
  return d;
}

struct SharedCtl {
  uint64_t full[8], empty[8], accum, sums;
  uint64_t raw_full[24], raw_empty[24];
  uint32_t tmem_base;
  volatile int abort;
};

// What every role does when one of its waits runs out.
__device__ __forceinline__ void give_up(SharedCtl &ctl, int *error_flag, int code) {
  if (!ctl.abort && error_flag) atomicCAS(error_flag, 0, code);
  ctl.abort = 1;
}

// A wait inside a hot loop: the first look is inline, the rest a call.  It looks MORE times before it lets itself be suspended: from that it would wake
// 250 cycles late (measured on B200).  (Not in the INT4 kernel, whose transform wants the issue slots.)
__device__ __noinline__ bool wait_on(uint32_t bar, uint32_t parity, volatile int *abort_flag, int more) {
  for (int i = 0; i < more; ++i)
    if (mbar_test(bar, parity)) return true;
  return mbar_wait(bar, parity, abort_flag);
}
__device__ __noinline__ bool wait_plain(uint32_t bar, uint32_t parity, volatile int *abort_flag) { return mbar_wait(bar, parity, abort_flag); }
template <int MORE = 64> __device__ __forceinline__ bool wait_fast(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  return mbar_test(bar, parity) || (MORE ? wait_on(bar, parity, abort_flag, MORE) : wait_plain(bar, parity, abort_flag));
}
// The same for a whole warp: every lane gets the same answer.
template <int MORE = 64> __device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  return __all_sync(0xffffffffu, wait_fast<MORE>(bar, parity, abort_flag));
}

__device__ __forceinline__ __half relu2_h(__half y) {
  const __half r = __hgt(y, __float2half_rn(0.f)) ? y : __float2half_rn(0.f);
  return h_mul(r, r);
}
// Sums of the gate row n (n % 16 < 8) and of the up row n + 8.
__device__ __forceinline__ __half swiglu_h(const Fp16Out &p, float gate, float up) {
  return h_mul(__float2half_rn(up * p.scale), swish_h(__float2half_rn(gate * p.scale)));
}
// The first `rows` of R rows m .. m + R - 1 of a warp's 32 weight rows (lane = n), fp16.
// PAIRS: all n are inside the output and neighbours on 4-byte boundaries: neighbouring lanes trade values so that a lane writes two
// consecutive n.  SWIGLU trades between lanes n and n + 8, and each computes every other row of the pair's feature.
struct Ahead2 { __half2 res[2], gate[2]; };     // residual and gate of four rows of a pair of outputs: every other row is a lane's
template <int EPI, bool PAIRS, int R> __device__ __forceinline__ void fp16_rows(const Fp16Out &p, const float (&sum)[R], int m, int rows, int n, int lane, const Ahead2 *got = nullptr) {
  constexpr bool GATED = EPI == PT_EPI_GATED_RESIDUAL, RES = EPI == PT_EPI_RESIDUAL || EPI == PT_EPI_BIAS_RESIDUAL || GATED, BIAS = EPI == PT_EPI_BIAS || EPI == PT_EPI_BIAS_GELU || EPI == PT_EPI_BIAS_RESIDUAL;
  if constexpr (EPI == PT_EPI_SWIGLU) {
    const bool up = lane & 8, in = PAIRS || n < p.N;
    __half *to = p.out + (size_t)(m + (up ? 1 : 0)) * p.out_ld + n / 16 * 8 + n % 8;
#pragma unroll
    for (int j = 0; j < R; j += 2) {
      const float t = __shfl_xor_sync(0xffffffffu, up ? sum[j] : sum[j + 1], 8);
      if (in && j + (up ? 1 : 0) < rows) *to = up ? swiglu_h(p, t, sum[j + 1]) : swiglu_h(p, sum[j], t);
      to += 2 * (size_t)p.out_ld;
    }
  } else if constexpr (PAIRS) {
    const int odd = lane & 1;
    __half2 *to = reinterpret_cast<__half2 *>(p.out + (size_t)(m + odd) * p.out_ld + (n - odd));
    __half2 res[RES ? R / 2 : 1], gate[GATED ? R / 2 : 1], bias = __half2half2(__half(0));
    if constexpr (RES) {
#pragma unroll
      for (int j = 0; j < R / 2; ++j) {
        const size_t at = (size_t)(m + odd + 2 * j) * p.N + (n - odd);
        if (R == 4 && got) {
          res[j] = got->res[j & 1];
          if constexpr (GATED) gate[j] = got->gate[j & 1];
        } else if (2 * j + odd < rows) {
          res[j] = __ldcg(reinterpret_cast<const __half2 *>(p.residual + at));
          if constexpr (GATED) gate[j] = __ldcg(reinterpret_cast<const __half2 *>(p.gate + at));
        }
      }
    }
    if constexpr (BIAS) bias = *reinterpret_cast<const __half2 *>(p.bias + (n - odd));
#pragma unroll
    for (int j = 0; j < R; j += 2) {
      const float t = __shfl_xor_sync(0xffffffffu, odd ? sum[j] : sum[j + 1], 1);   // even lane: row j of n + 1; odd lane: row j + 1 of n - 1
      __half2 y = odd ? __floats2half2_rn(t * p.scale, sum[j + 1] * p.scale) : __floats2half2_rn(sum[j] * p.scale, t * p.scale);
      if constexpr (BIAS) y = __hadd2_rn(y, bias);
      if constexpr (EPI == PT_EPI_RELU2) y = __halves2half2(relu2_h(__low2half(y)), relu2_h(__high2half(y)));
      if constexpr (EPI == PT_EPI_BIAS_GELU) y = __halves2half2(gelu_h(__low2half(y)), gelu_h(__high2half(y)));
      if constexpr (GATED) y = __halves2half2(h_mul(sigmoid_h(__low2half(gate[j / 2])), __low2half(y)), h_mul(sigmoid_h(__high2half(gate[j / 2])), __high2half(y)));
      if constexpr (RES) y = __hadd2_rn(res[j / 2], y);
      if constexpr (GATED) { if (p.halve) y = __hmul2_rn(y, __float2half2_rn(0.5f)); }
      if (j + odd < rows) *to = y;
      to += p.out_ld;   // (two rows, in units of two)
    }
  } else if (n < p.N) {
    __half *to = p.out + (size_t)m * p.out_ld + n;
    const __half bias = BIAS ? p.bias[n] : __half(0);
#pragma unroll
    for (int j = 0; j < R; ++j) {
      if (j >= rows) break;
      __half y = __float2half_rn(sum[j] * p.scale);
      if constexpr (BIAS) y = h_add(y, bias);
      if constexpr (EPI == PT_EPI_RELU2) y = relu2_h(y);
      if constexpr (EPI == PT_EPI_BIAS_GELU) y = gelu_h(y);
      if constexpr (GATED) y = h_mul(sigmoid_h(__ldcg(p.gate + (size_t)(m + j) * p.N + n)), y);
      if constexpr (RES) y = h_add(__ldcg(p.residual + (size_t)(m + j) * p.N + n), y);
      if constexpr (GATED) { if (p.halve) y = h_mul(y, __float2half_rn(0.5f)); }
      *to = y;
      to += p.out_ld;
    }
  }
}
// ALL: the FP16 kernel's epilogues too (the others' code stays short).
template <bool ALL, bool PAIRS, int R> __device__ __forceinline__ void fp16_rows_by(const Fp16Out &p, const float (&sum)[R], int m, int rows, int n, int lane, const Ahead2 *got = nullptr) {
  if (p.epilogue == PT_EPI_SWIGLU) fp16_rows<PT_EPI_SWIGLU, PAIRS, R>(p, sum, m, rows, n, lane, got);
  else if (p.epilogue == PT_EPI_RESIDUAL) fp16_rows<PT_EPI_RESIDUAL, PAIRS, R>(p, sum, m, rows, n, lane, got);
  else if (p.epilogue == PT_EPI_BIAS) fp16_rows<PT_EPI_BIAS, PAIRS, R>(p, sum, m, rows, n, lane, got);
  else if (ALL && p.epilogue == PT_EPI_BIAS_GELU) fp16_rows<PT_EPI_BIAS_GELU, PAIRS, R>(p, sum, m, rows, n, lane, got);
  else if (ALL && p.epilogue == PT_EPI_GATED_RESIDUAL) fp16_rows<PT_EPI_GATED_RESIDUAL, PAIRS, R>(p, sum, m, rows, n, lane, got);
  else if (ALL && p.epilogue == PT_EPI_RELU2) fp16_rows<PT_EPI_RELU2, PAIRS, R>(p, sum, m, rows, n, lane, got);
  else if (ALL && p.epilogue == PT_EPI_BIAS_RESIDUAL) fp16_rows<PT_EPI_BIAS_RESIDUAL, PAIRS, R>(p, sum, m, rows, n, lane, got);
  else fp16_rows<PT_EPI_STORE, PAIRS, R>(p, sum, m, rows, n, lane, got);
}
// Whether the rows of the 32 weight rows from nq on can leave in pairs.
__device__ __forceinline__ bool fp16_pairs(const Fp16Out &p, int nq) {
  return nq + 32 <= p.N && p.out_ld % 2 == 0 && ((uintptr_t)p.out & 3) == 0 && (!p.residual || (p.N % 2 == 0 && ((uintptr_t)p.residual & 3) == 0)) &&
         (!p.bias || ((uintptr_t)p.bias & 3) == 0) && (!p.gate || ((uintptr_t)p.gate & 3) == 0);
}
// The epilogue of a tile without k-slices, fp16 outputs: `part` of `parts` warps share a quarter of the rows and take alternate 16 columns.
// (Measured on B200, FP8 10304 x 2048, whose last tile is half empty, at 256 rows: 12.9 us; element by element over all branches, empty
// quarters included, 18.9.  2048 x 128 at 12 rows, a step of 16 in part: 3.1 and 4.7.)
template <bool ALL> __device__ __forceinline__ void epilogue_fp16(const GemmParams &p, const Fp16Out &o, uint32_t tmem, int q, int lane, int part, int parts, int n0, int m0) {
  const int nq = n0 + q * 32, n = nq + lane, rows = min(p.mb, p.M - m0);
  if (nq >= o.N) return;          // (uniform over the warp, as is `pairs`)
  const bool pairs = fp16_pairs(o, nq);
  for (int c0 = part * 16; c0 < rows; c0 += 16 * parts) {
    uint32_t v[16];
    float sum[16];
    tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
    for (int j = 0; j < 16; ++j) sum[j] = __uint_as_float(v[j]);
    if (pairs) fp16_rows_by<ALL, true>(o, sum, m0 + c0, rows - c0, n, lane);
    else fp16_rows_by<ALL, false>(o, sum, m0 + c0, rows - c0, n, lane);
  }
}
// R rows of one weight row per lane, gated: lanes n and n + 8 hold a feature's two sums.
template <int GLU, bool EXT, int R> __device__ __forceinline__ void glu_rows(const GemmParams &p, const float (&sum)[R], int m, int m_end, int n, int lane) {
  const DenseOut &d = p.dense;
  const bool store = n < p.N && (lane & 8) == 0;
  const float bg = store && d.bias ? __ldg(d.bias + n) : 0.f, bu = store && d.bias ? __ldg(d.bias + n + 8) : 0.f;
  const int f = n / 16 * 8 + n % 8;
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const float up = __shfl_xor_sync(0xffffffffu, sum[j], 8);
    if (!store || m + j >= m_end) continue;
    const float s = dense_factor<EXT>(d, m + j);
    dense_put(d, m + j, f, glu_unit<true, GLU>(fmaf(sum[j], s, bg), fmaf(up, s, bu), d.limit));
  }
}

// Rows m .. m + R - 1 of the BF16 kernel's 32 weight rows from nq on: any sizes and alignment.
template <bool EXT, int R> __device__ __forceinline__ void bf16_rows(const GemmParams &p, const float (&sum)[R], int m, int m_end, int nq, int lane) {
  const int n = nq + lane;
  if (p.dense.epilogue == PT_EPI_GLU && nq < p.dense.split_n) {   // (uniform over the warp)
    if (EXT && p.dense.glu == PT_GLU_SILU) glu_rows<PT_GLU_SILU, EXT>(p, sum, m, m_end, n, lane);
    else if (EXT && p.dense.glu == PT_GLU_GELU) glu_rows<PT_GLU_GELU, EXT>(p, sum, m, m_end, n, lane);
    else glu_rows<PT_GLU_CLAMPED, EXT>(p, sum, m, m_end, n, lane);
  } else if (n < p.N) {
#pragma unroll
    for (int j = 0; j < R; ++j) {
      if (m + j >= m_end) break;
      dense_store<EXT>(p.dense, m + j, n, sum[j]);
    }
  }
}
// Four rows of a warp's 32 weight rows (lane = n): four lanes trade their values, so that each has one row of their four weight rows and leaves them at once.
// (Element by element: 1600 x 1600 at 24 rows in seven slices 4.65 us, so 4.3.)
template <bool EXT> __device__ __forceinline__ void bf16_rows4(const GemmParams &p, const float (&sum)[4], int m, int m_end, int nq, int lane) {
  const bool odd = lane & 1, high = lane & 2;
  const float a = __shfl_xor_sync(0xffffffffu, odd ? sum[0] : sum[1], 1), b = __shfl_xor_sync(0xffffffffu, odd ? sum[2] : sum[3], 1);
  // rows odd and odd + 2 of two neighbours, then row (lane & 3) of all four
  const float r0 = odd ? a : sum[0], r1 = odd ? sum[1] : a, s0 = odd ? b : sum[2], s1 = odd ? sum[3] : b;
  const float c = __shfl_xor_sync(0xffffffffu, high ? r0 : s0, 2), d = __shfl_xor_sync(0xffffffffu, high ? r1 : s1, 2);
  const float4 v = high ? make_float4(c, d, s0, s1) : make_float4(r0, r1, c, d);
  const int row = m + (lane & 3), n = nq + (lane & ~3);
  if (p.dense.epilogue == PT_EPI_GLU && nq < p.dense.split_n) {   // (uniform over the warp; gate rows n % 16 < 8, their up rows eight further)
    float4 up;
    up.x = __shfl_xor_sync(0xffffffffu, v.x, 8); up.y = __shfl_xor_sync(0xffffffffu, v.y, 8);
    up.z = __shfl_xor_sync(0xffffffffu, v.z, 8); up.w = __shfl_xor_sync(0xffffffffu, v.w, 8);
    if (row < m_end && n < p.N && !(lane & 8)) dense_store_glu4<EXT>(p.dense, row, n, v, up);
  } else if (row < m_end && n + 4 <= p.N) {
    dense_store4<EXT>(p.dense, row, n, v);
  } else if (row < m_end && n < p.N) {
    dense_store<EXT>(p.dense, row, n, v.x);
    if (n + 1 < p.N) dense_store<EXT>(p.dense, row, n + 1, v.y);
    if (n + 2 < p.N) dense_store<EXT>(p.dense, row, n + 2, v.z);
  }
}
// The BF16 kernel's general epilogue: 16 columns a step.
template <bool EXT>
__device__ __forceinline__ void epilogue_any(const GemmParams &p, uint32_t tmem, int q, int lane, int n0, int m0, int m_end, int c_first) {
  for (int c0 = c_first; c0 < min(p.mb, m_end - m0); c0 += 16) {
    uint32_t v[16];
    float sum[16];
    tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
    for (int j = 0; j < 16; ++j) sum[j] = __uint_as_float(v[j]);
    bf16_rows<EXT>(p, sum, m0 + c0, m_end, n0 + q * 32, lane);
  }
}

// The BF16 kernel's epilogue of a whole 32-column group without k-slices: uniform branches outside the element loop, pointer
// increments instead of index arithmetic (the general form above costs as much as the products of a 2048-deep tile).
// bf16 output: neighbouring lanes (n, n + 1) trade values of two columns, so every store writes 4 bytes per lane.
// Gated features: lanes n and n + 8 trade likewise, and each computes one column of the pair's feature.
enum { OUT_F32 = 0, OUT_BF16 = 1, OUT_GLU = 2, OUT_GELU_MUL = 3 };
enum { ACT_NONE = 0, ACT_RELU2 = 1, ACT_SOFTCAP = 2, ACT_XIELU = 3, ACT_SCALED = 16 };   // OUT_GLU: the kind of unit, plus ACT_SCALED with a factor per row
template <int KIND, int ACT>
__device__ __forceinline__ void epilogue_rows32(const DenseOut &d, void *out, int ld, const uint32_t (&v)[32], int n, int m, int lane) {
  const float b = d.bias ? __ldg(d.bias + n + (KIND == OUT_F32 && out == d.out2 ? d.split_n : 0)) : 0.f;
  auto fin = [&](uint32_t x) {
    float y = fmaf(__uint_as_float(x), d.alpha, b);
    if (ACT == ACT_RELU2) { y = fmaxf(y, 0.f); y *= y; }
    if (ACT == ACT_SOFTCAP) y = softcap_fast(y, d.limit);
    if (ACT == ACT_XIELU) y = xielu_f<false>(y, d.pos, d.neg);
    return y;
  };
  if (KIND == OUT_F32) {
    float *o = reinterpret_cast<float *>(out) + (size_t)m * ld + n;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      *o = fin(v[j]);
      o += ld;
    }
  } else if (KIND == OUT_BF16 || KIND == OUT_GELU_MUL) {
    float w[KIND == OUT_GELU_MUL ? 32 : 1];     // the factors of this lane's column, requested together
    if (KIND == OUT_GELU_MUL) {
      const __nv_bfloat16 *mul = reinterpret_cast<const __nv_bfloat16 *>(d.mul) + n;
#pragma unroll
      for (int j = 0; j < 32; ++j) w[j] = __bfloat162float(mul[(size_t)__ldg(d.mul_ids + m + j) * d.mul_ld]);
    }
    const int odd = lane & 1;
    __nv_bfloat16 *o = reinterpret_cast<__nv_bfloat16 *>(out) + (size_t)(m + odd) * ld + (n - odd);
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      float a = fin(v[j]), c = fin(v[j + 1]);
      if (KIND == OUT_GELU_MUL) {
        a = gelu_tanh_fast(a) * w[KIND == OUT_GELU_MUL ? j : 0];
        c = gelu_tanh_fast(c) * w[KIND == OUT_GELU_MUL ? j + 1 : 0];
      }
      const float t = __shfl_xor_sync(0xffffffffu, odd ? a : c, 1);     // even lane: column j of n + 1; odd lane: column j + 1 of n - 1
      *reinterpret_cast<__nv_bfloat162 *>(o) = odd ? __floats2bfloat162_rn(t, c) : __floats2bfloat162_rn(a, t);
      o += 2 * (size_t)ld;
    }
  } else {
    const bool up = lane & 8;
    __nv_bfloat16 *o = reinterpret_cast<__nv_bfloat16 *>(out) + (size_t)(m + (up ? 1 : 0)) * ld + n / 16 * 8 + n % 8;
    const float mine = (ACT & ACT_SCALED) ? d.alpha * __ldcg(d.row_scale + m + lane) : d.alpha;     // lane j: the factor of row m + j
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const float s0 = (ACT & ACT_SCALED) ? __shfl_sync(0xffffffffu, mine, j) : mine, s1 = (ACT & ACT_SCALED) ? __shfl_sync(0xffffffffu, mine, j + 1) : mine;
      const float a = fmaf(__uint_as_float(v[j]), s0, b), c = fmaf(__uint_as_float(v[j + 1]), s1, b);
      const float t = __shfl_xor_sync(0xffffffffu, up ? a : c, 8);      // gate lane: the up value of column j; up lane: the gate value of j + 1
      *o = __float2bfloat16_rn(up ? glu_unit<true, ACT & 15>(t, c, d.limit) : glu_unit<true, ACT & 15>(a, t, d.limit));
      o += 2 * (size_t)ld;
    }
  }
}
template <bool EXT> __device__ __forceinline__ void epilogue_bf16(const GemmParams &p, uint32_t tmem, int q, int lane, int n0, int m0, int m_end) {
  const DenseOut &d = p.dense;
  const int nq = n0 + q * 32, n = nq + lane;
  // (warp-uniform) where this warp's 32 outputs go
  const bool second = nq >= d.split_n, glu = d.epilogue == PT_EPI_GLU && !second, f32 = second || d.out_dt == PT_DT_F32;
  // whole columns of 32 rows inside the output; 4-byte aligned pairs for bf16
  const bool fast = nq + 32 <= p.N && !(!second && d.epilogue == PT_EPI_GELU_MUL && f32) && !(glu && f32) && (!EXT || ((!d.row_scale || (glu && d.glu == PT_GLU_SILU)) && (second || (f32 ? d.epilogue != PT_EPI_XIELU : d.epilogue != PT_EPI_SOFTCAP)))) &&
                    (f32 || glu || (d.out_ld % 2 == 0 && ((uintptr_t)d.out & 3) == 0));
  const int rows = min(p.mb, m_end - m0), whole = fast ? rows & ~31 : 0;
  for (int c0 = 0; c0 < whole; c0 += 32) {
    uint32_t v[32];
    tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v);
    if (second) {
      epilogue_rows32<OUT_F32, ACT_NONE>(d, d.out2, d.out2_ld, v, n - d.split_n, m0 + c0, lane);
    } else if (glu) {
      if (EXT && d.glu == PT_GLU_SILU && d.row_scale) epilogue_rows32<OUT_GLU, PT_GLU_SILU | ACT_SCALED>(d, d.out, d.out_ld, v, n, m0 + c0, lane);
      else if (EXT && d.glu == PT_GLU_GELU) epilogue_rows32<OUT_GLU, PT_GLU_GELU>(d, d.out, d.out_ld, v, n, m0 + c0, lane);
      else if (EXT && d.glu == PT_GLU_SILU) epilogue_rows32<OUT_GLU, PT_GLU_SILU>(d, d.out, d.out_ld, v, n, m0 + c0, lane);
      else epilogue_rows32<OUT_GLU, PT_GLU_CLAMPED>(d, d.out, d.out_ld, v, n, m0 + c0, lane);
    } else if (f32) {
      if (d.epilogue == PT_EPI_RELU2) epilogue_rows32<OUT_F32, ACT_RELU2>(d, d.out, d.out_ld, v, n, m0 + c0, lane);
      else if (EXT && d.epilogue == PT_EPI_SOFTCAP) epilogue_rows32<OUT_F32, ACT_SOFTCAP>(d, d.out, d.out_ld, v, n, m0 + c0, lane);
      else epilogue_rows32<OUT_F32, ACT_NONE>(d, d.out, d.out_ld, v, n, m0 + c0, lane);
    } else {
      if (d.epilogue == PT_EPI_GELU_MUL) epilogue_rows32<OUT_GELU_MUL, ACT_NONE>(d, d.out, d.out_ld, v, n, m0 + c0, lane);
      else if (d.epilogue == PT_EPI_RELU2) epilogue_rows32<OUT_BF16, ACT_RELU2>(d, d.out, d.out_ld, v, n, m0 + c0, lane);
      else if (EXT && d.epilogue == PT_EPI_XIELU) epilogue_rows32<OUT_BF16, ACT_XIELU>(d, d.out, d.out_ld, v, n, m0 + c0, lane);
      else epilogue_rows32<OUT_BF16, ACT_NONE>(d, d.out, d.out_ld, v, n, m0 + c0, lane);
    }
  }
  if (whole < rows) epilogue_any<EXT>(p, tmem, q, lane, n0, m0, m_end, whole);
}

// k-slices of a tile: the blocks of a cluster, slice = rank.  The tile's activation rows in groups of four are dealt out to the blocks; every block sends each
// group to the block that writes it, as [group][slice][weight row][4], by stores that arrive at a barrier there, and that block sums the slices in
// order (deterministic).  That is for tiles of few rows (gemm_plan.h has the rule).  (Blocks that left their sums at home, met, fetched what they needed and met again before their shared memory
// went took longer: 1600 x 1600 at 16 rows in seven slices 4.8 us a launch in a row of launches, so 3.9; 1600 x 6400 7.7 and 7.0; 2048 x 2048 at 32 rows 5.3 and
// 4.7; B200.)
__device__ __forceinline__ int own_groups(int groups, int ksplit, int rank) { return rank < groups ? (groups - rank + ksplit - 1) / ksplit : 0; }
__device__ __forceinline__ int row_groups(const GemmParams &p, int m0, int m_end) { return (min(p.mb, m_end - m0) + 3) >> 2; }
__device__ __forceinline__ void expect_sums(const GemmParams &p, SharedCtl &ctl, int rank, int m0, int m_end) {
  mbar_init(sa(&ctl.sums), 1);
  const int own = own_groups(row_groups(p, m0, m_end), p.ksplit, rank);
  if (own) mbar_expect_tx(sa(&ctl.sums), own * p.ksplit * BM * 16);
}
// The warps that sum have asked for what they need before their products are there: residual and gate of the first group of rows a warp writes, and
// (the parameters of a launch are in no cache at first) the fields that the outputs go by.
struct SumAhead { Ahead2 v; bool pairs, got; };
template <bool BF16> __device__ __forceinline__ SumAhead sums_ahead(const GemmParams &p, const Fp16Out &o, int rank, int part, int n0, int m0, int m_end, int q, int lane) {
  SumAhead a;
  a.pairs = !BF16 && fp16_pairs(o, n0 + q * 32);
  a.got = a.pairs && o.residual;
  if constexpr (BF16) asm volatile("" ::"r"(p.dense.epilogue), "r"(p.dense.out_ld), "f"(p.dense.limit), "r"(p.dense.glu), "l"(p.dense.out), "l"(p.dense.bias));
  if (a.got) {
    const int odd = lane & 1, m = m0 + 4 * (part * p.ksplit + rank);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const size_t at = (size_t)(m + odd + 2 * j) * o.N + (n0 + q * 32 + lane - odd);
      const bool in = m + odd + 2 * j < m_end;
      a.v.res[j] = in ? __ldcg(reinterpret_cast<const __half2 *>(o.residual + at)) : __half2half2(__half(0));
      a.v.gate[j] = in && o.gate ? __ldcg(reinterpret_cast<const __half2 *>(o.gate + at)) : __half2half2(__half(0));
    }
  }
  return a;
}
// Larger tiles leave the sums at home: every block in its own shared memory as [mb][128] floats (the operand ring, which nobody reads any more), the blocks meet,
// each sums its share of the tile over all of them in slice order, all its threads at once, and they meet again before their shared memory goes.  Sent and summed by four
// warps, a group of rows after the other, they take longer: us sent / fetched, 4096 x 4096 at 128 rows (two slices of 64-row tiles) fp16 18.3 / 15.3, bf16 19.5 / 15.5;
// 4608 x 4096 at 256 rows fp8 18.1 / 15.5; 4096 x 4096 at 200 rows int4 13.7 / 12.0.
__device__ __forceinline__ void leave_sums(const GemmParams &p, uint32_t tmem, int q, int lane, int part, int parts, float *dst) {
  for (int c0 = part * 16; c0 < p.mb; c0 += 16 * parts) {
    uint32_t v[16];
    tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
    for (int j = 0; j < 16; ++j) dst[(c0 + j) * BM + q * 32 + lane] = __uint_as_float(v[j]);
  }
}
__device__ __forceinline__ float4 load_cluster4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
template <bool BF16, bool EXT, bool ALL = false>
__device__ __forceinline__ void fetch_sums(const GemmParams &p, const Fp16Out &o, const SharedCtl &ctl, uint32_t part, int rank, int n0, int m0, int m_end, int threads) {
  cluster_arrive();
  cluster_wait();
  if (!ctl.abort) {
    const int N = BF16 ? p.N : o.N, units = min(p.mb, m_end - m0) * (BM / 4), share = (units + p.ksplit - 1) / p.ksplit, last = min(units, (rank + 1) * share);
    const bool rows_of_4 = !BF16 && N % 4 == 0, res_whole = rows_of_4 && ((uintptr_t)o.residual & 7) == 0, gate_whole = rows_of_4 && ((uintptr_t)o.gate & 7) == 0;
    for (int i = rank * share + (int)threadIdx.x; i < last; i += threads) {
      const int m = m0 + i / (BM / 4), n = n0 + (i % (BM / 4)) * 4;
      if (n >= N) continue;
      Half4 res{}, gate{}, bias{};
      if constexpr (!BF16) {
        if (o.residual) res = load4(o.residual + (size_t)m * N + n, n, N, res_whole);
        if (ALL && o.gate) gate = load4(o.gate + (size_t)m * N + n, n, N, gate_whole);
        if (o.bias) bias = load4(o.bias + n, n, N, n + 4 <= N && ((uintptr_t)o.bias & 7) == 0);
      }
      auto sum4 = [&](int unit) {
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (int s0 = 0; s0 < p.ksplit; s0 += 4) {   // four loads in flight
          float4 v[4];
#pragma unroll
          for (int s = 0; s < 4; ++s) v[s] = s0 + s < p.ksplit ? load_cluster4(in_block(part + unit * 16, s0 + s)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int s = 0; s < 4; ++s) { acc.x += v[s].x; acc.y += v[s].y; acc.z += v[s].z; acc.w += v[s].w; }
        }
        return acc;
      };
      const bool glu = BF16 ? p.dense.epilogue == PT_EPI_GLU && n < p.dense.split_n : o.epilogue == PT_EPI_SWIGLU;
      if (glu) {   // gate rows n % 16 < 8, their up rows eight further
        if (n & 8) continue;
        const float4 g = sum4(i), u = sum4(i + 2);
        if constexpr (BF16) {
          dense_store_glu4<EXT>(p.dense, m, n, g, u);
        } else {
          const int f = n / 16 * 8 + n % 8;
          const Half4 y = {swiglu_h(o, g.x, u.x), swiglu_h(o, g.y, u.y), swiglu_h(o, g.z, u.z), swiglu_h(o, g.w, u.w)};
          store4(o.out + (size_t)m * o.out_ld + f, y, f, N / 2);
        }
        continue;
      }
      float4 acc = sum4(i);
      if constexpr (!BF16) {
        acc.x *= o.scale; acc.y *= o.scale; acc.z *= o.scale; acc.w *= o.scale;
        store4(o.out + (size_t)m * o.out_ld + n, finish4<ALL>(o.epilogue, acc, res, bias, gate, o.halve), n, N);
      } else if (n + 4 <= N) {
        dense_store4<EXT>(p.dense, m, n, acc);
      } else {
        dense_store<EXT>(p.dense, m, n, acc.x);
        if (n + 1 < N) dense_store<EXT>(p.dense, m, n + 1, acc.y);
        if (n + 2 < N) dense_store<EXT>(p.dense, m, n + 2, acc.z);
      }
    }
  }
  cluster_arrive();
  cluster_wait();
}
// The warps that have a tile's quarters q (`parts` times four of them, each part every parts-th step of 16 rows); the other threads of the block call it too.
template <bool BF16, bool EXT, bool ALL = false>
__device__ __forceinline__ void sum_cluster(const GemmParams &p, const Fp16Out &o, SharedCtl &ctl, uint32_t tmem, unsigned char *smem, int rank, int n0, int m0, int m_end, int part, int parts, int q, int lane, const SumAhead &ahead) {
  if (p.sum_offset == 0) {    // where the sums take the place of the operands, nobody reads these any more
    cluster_arrive();
    cluster_wait();
  }
  if (part < 0) return;
  const int groups = row_groups(p, m0, m_end), ks = p.ksplit;
  const uint32_t mine = sa(smem + p.sum_offset) + (q * 32 + lane) * 16, bar = sa(&ctl.sums);
  // (After a failure what there is goes out all the same: the others' waits end, and the error flag is up.)
  int to = part * 4 % ks, slot = part * 4 / ks * ks + rank;
  for (int g0 = part * 4; g0 < groups; g0 += 4 * parts) {
    uint32_t v[16];
    tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(4 * g0), v);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if (g0 + t < groups) send4(in_block(mine + slot * (BM * 16), to), v[4 * t], v[4 * t + 1], v[4 * t + 2], v[4 * t + 3], in_block(bar, to));
      if (++to == ks) { to = 0; slot += ks; }
    }
    for (int skip = 4 * (parts - 1); skip > 0; --skip)
      if (++to == ks) { to = 0; slot += ks; }
  }
  const int own = own_groups(groups, ks, rank);
  if (!own) return;
  if (!warp_wait(bar, 0, &ctl.abort)) give_up(ctl, p.error_flag, 27);
  if (ctl.abort) return;
  const int nq = n0 + q * 32, n = nq + lane;
  if (nq >= (BF16 ? p.N : o.N)) return;
  for (int i = part; i < own; i += parts) {
    float4 v[MAX_CLUSTER];
#pragma unroll
    for (int s = 0; s < MAX_CLUSTER; ++s)
      v[s] = s < ks ? *reinterpret_cast<const float4 *>(smem + p.sum_offset + ((size_t)(i * ks + s) * BM + q * 32 + lane) * 16) : make_float4(0.f, 0.f, 0.f, 0.f);
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < MAX_CLUSTER; ++s) { sum[0] += v[s].x; sum[1] += v[s].y; sum[2] += v[s].z; sum[3] += v[s].w; }
    const int m = m0 + 4 * (i * ks + rank);
    if constexpr (BF16) bf16_rows4<EXT>(p, sum, m, m_end, nq, lane);
    else if (ahead.pairs) fp16_rows_by<ALL, true>(o, sum, m, m_end - m, n, lane, ahead.got && i == part ? &ahead.v : nullptr);
    else fp16_rows_by<ALL, false>(o, sum, m, m_end - m, n, lane);
  }
}

// Up to 32 activation rows: four warps fetch a k block in turn, a lane 16 bytes of every fourth row, the next block's loads under way while one is stored
// in the image that TMA would have written.  (One thread gets a TMA box of 128 bytes a row on its way every 280 cycles, whatever the rows: of four boxes the
// last arrived 1700 cycles after the kernel in front had ended, B200.)  A wait tells only odd from even uses of a slot, so at least four slots.
__device__ __forceinline__ void fetch_rows(const GemmParams &p, SharedCtl &ctl, unsigned char *b0, uint32_t stage_bytes, int kb0, int n_it, int m0, int rows, int w, int lane) {
  const int r0 = lane >> 3, c = lane & 7;
  const unsigned char *src = p.x + (size_t)(m0 + r0) * p.x_pitch + (size_t)kb0 * BKB + c * 16;
  const uint32_t full0 = sa(&ctl.full[0]), empty0 = sa(&ctl.empty[0]);
  uint4 v[8];
  auto get = [&](int it) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (4 * i + r0 < rows) v[i] = __ldcg(reinterpret_cast<const uint4 *>(src + (size_t)(4 * i) * p.x_pitch + (size_t)it * BKB));
  };
  int s = w;
  uint32_t par = 1;
  if (w < n_it) get(w);
  for (int it = w; it < n_it; it += 4) {
    if (it >= p.stages && !warp_wait(empty0 + s * 8, par, &ctl.abort)) { give_up(ctl, p.error_flag, 25); break; }
    unsigned char *to = b0 + (size_t)s * stage_bytes + r0 * BKB;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (4 * i + r0 < rows) *reinterpret_cast<uint4 *>(to + 4 * i * BKB + ((c ^ (((i & 1) << 2) + r0)) << 4)) = v[i];
    if (it + 4 < n_it) get(it + 4);
    fence_operands();
    __syncwarp();
    if (lane == 0) mbar_arrive(full0 + s * 8);
    s += 4;
    while (s >= p.stages) { s -= p.stages; par ^= 1u; }
  }
}

// The end of a block that gave up, all threads: what it has asked for has landed (`full0` and `issued` of the thread that asked), its MMAs are done with
// shared and tensor memory, and nobody sends it sums any more.
__device__ __noinline__ void end_after_failure(SharedCtl &ctl, uint32_t full0, int issued, int stages, int warp, int ksplit) {
  if (issued) mbar_wait_ring(full0, issued, stages);
  if (warp == 1) mbar_wait_ring(sa(&ctl.accum), 1, 1);
  if (ksplit > 1) stay_for_cluster();
  __syncthreads();
}

// ------------------------------------------------------------------------------------------ FP8, FP16 and BF16
// Dynamic shared memory: [stage][NA A tiles of 16 KB | B tile mb * 128 B], every tile 1024-byte aligned.  NA = 2: a CTA takes 256 weight
// rows (two accumulators), which fetches a third less per product than NA = 1; without k-slices.  With up to 128 activation rows two such CTAs share an
// SM, so their registers have to allow it (96 a thread): a Pivavik of width 2048 takes four prompts of 2048 tokens, whose experts have tiles of 128
// rows, in 20.4 ms so and in 24.5 with the 168 registers that one CTA of 320 threads per SM may have (measured on B200).
template <int FMT, int NA, bool EXT, Sums SUMS>
__global__ void __launch_bounds__(64 + 128 * NA, 2) gemm_dense_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                                   const GemmParams p) {
  constexpr bool BF16 = FMT == PT_W_BF16, F8 = FMT == PT_W_FP8;
  constexpr int KX = F8 ? BKB : BKB / 2;     // elements of k per stage
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ SharedCtl ctl;
  unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  int part = 0;
  if (FMT == PT_W_FP16)
    while (part + 1 < p.n_parts && (int)blockIdx.x >= p.part_tile[part + 1]) ++part;
  // (FP16: a copy.  Which part it is the compiler does not know, and read where it is used 128 x 128 at 128 rows takes 3.7 us instead of 3.0.)
  const std::conditional_t<FMT == PT_W_FP16, Fp16Out, const Fp16Out &> o = p.o[FMT == PT_W_FP16 ? part : 0];
  const int n0 = (blockIdx.x - (FMT == PT_W_FP16 ? p.part_tile[part] : 0)) * (BM * NA), m0 = blockIdx.z * p.mb, x0 = part * p.M + m0, ks = blockIdx.y;     // (x0: the first activation row)
  const int kb0 = ks * p.kb_per_split, kb1 = min(p.n_kb, kb0 + p.kb_per_split);
  const int n_it = kb1 - kb0, na = NA == 1 ? 1 : min(NA, p.n_tiles - (int)blockIdx.x * NA);
  const uint32_t b_bytes = (uint32_t)p.mb * BKB;
  const uint32_t stage_bytes = NA * A_TILE + ((b_bytes + 1023u) & ~1023u);
  const uint32_t smem_s = sa(smem);
  const bool sent = SUMS == SENT && NA == 1 && p.ksplit > 1, fetched = SUMS == FETCHED && NA == 1 && p.ksplit > 1;
  int m_end = min(p.M, m0 + p.mb), mma_n = p.mb;
  size_t w_base = 0;
  if constexpr (BF16) {
    if (p.group_of) {
      if (p.pdl) wait_for_prerequisites();     // the router may be among the kernels before
      const int grp = p.group_of[blockIdx.z];
      if (grp < 0) return;                     // a tile without rows: nothing is initialised yet
      w_base = (size_t)grp * p.group_stride;
      if (p.group_used) {
        m_end = m0 + min(p.mb, p.group_used[blockIdx.z]);
        mma_n = max(16, (m_end - m0 + 15) & ~15);
      }
    }
  }
  const uint32_t tmem_cols = p.tmem_columns, acc_cols = tmem_cols / NA;

  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(sa(&ctl.full[s]), p.x_warps ? 2 : 1);
      mbar_init(sa(&ctl.empty[s]), 1);
    }
    mbar_init(sa(&ctl.accum), 1);
    if (sent) expect_sums(p, ctl, ks, m0, m_end);
    ctl.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (sent) cluster_arrive();
  if (warp == 1) tmem_alloc(sa(&ctl.tmem_base), tmem_cols);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = ctl.tmem_base;
  // Not before: a CTA of the next GEMM that found the tensor memory free would keep it while it waits for this kernel to end.
  if (p.pdl) launch_dependents();
  SumAhead ahead{};
  int issued = 0;     // stages that this thread has asked for

  if (warp == 0) {
    if (elect_one()) {
      // (ring positions and parities are carried as counters: this thread's instruction count per stage is what limits a CTA)
      const unsigned char *wt = p.w + w_base + ((size_t)blockIdx.x * NA * p.n_kb + kb0) * A_TILE;
      const size_t next_tile = (size_t)p.n_kb * A_TILE;
      const uint32_t tx = na * A_TILE + (p.x_warps ? 0 : b_bytes), full0 = sa(&ctl.full[0]), empty0 = sa(&ctl.empty[0]);
      const bool tiled = p.w_tiled != 0;     // (always, if p.pdl: the early loads below do not move kx on)
      int s = 0, kx = kb0 * KX;
      uint32_t par = 1;   // parity of the `empty` phase that must have completed before slot s is refilled (none in the first round)
      bool first_round = true;
      auto load_w = [&](uint32_t st, uint32_t fb) {
        if (tiled) {
          bulk_g2s(st, wt, A_TILE, fb);
          if (NA == 2 && na == 2) bulk_g2s(st + A_TILE, wt + next_tile, A_TILE, fb);
        } else {
          tma_load_2d(st, &map_w, kx, n0, fb);
        }
        wt += A_TILE;
      };
      int early = 0;                         // stages whose weights are already on their way
      if (p.pdl) {
        for (; early < min(p.stages, n_it); ++early) {
          mbar_expect_tx(full0 + early * 8, tx);
          load_w(smem_s + early * stage_bytes, full0 + early * 8);
        }
        wait_for_prerequisites();
      }
      for (int it = 0; it < n_it; ++it) {
        if (!first_round && !wait_fast(empty0 + s * 8, par, &ctl.abort)) { give_up(ctl, p.error_flag, 21); break; }
        issued = it + 1;
        const uint32_t st = smem_s + s * stage_bytes, fb = full0 + s * 8;
        if (it >= early) {
          mbar_expect_tx(fb, tx);
          load_w(st, fb);
        }
        if (!p.x_warps) tma_load_2d(st + NA * A_TILE, &map_x, kx, x0, fb);
        kx += KX;
        if (++s == p.stages) { s = 0; par ^= 1u; first_round = false; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      // One thread issues every MMA of the CTA, so its loop is kept to a few dozen instructions per stage: descriptors are one
      // 64-bit add away from the stage-0 descriptors (the start-address field counts 16-byte units), ring position and parity
      // are counters.  (Measured: with divisions and descriptor rebuilds in this loop a stage took 0.6 us whatever its size.)
      const uint32_t idesc = instr_desc(BF16, mma_n);
      const uint64_t adesc0 = smem_desc_sw128(smem_s), bdesc0 = smem_desc_sw128(smem_s + NA * A_TILE);
      const uint32_t full0 = sa(&ctl.full[0]), empty0 = sa(&ctl.empty[0]), stage16 = stage_bytes >> 4;
      int s = 0;
      uint32_t par = 0, acc = 0;
      for (int it = 0; it < n_it; ++it) {
        if (!wait_fast(full0 + s * 8, par, &ctl.abort)) { give_up(ctl, p.error_flag, 22); break; }
        fence_after();
        const uint64_t adesc = adesc0 + (uint64_t)(s * stage16), bdesc = bdesc0 + (uint64_t)(s * stage16);
        umma<F8>(tmem, adesc, bdesc, idesc, acc);   // four MMAs of 32 bytes of k each; inside the swizzle atom the start address moves by 32 bytes
        umma<F8>(tmem, adesc + 2, bdesc + 2, idesc, 1u);
        umma<F8>(tmem, adesc + 4, bdesc + 4, idesc, 1u);
        umma<F8>(tmem, adesc + 6, bdesc + 6, idesc, 1u);
        if (NA == 2 && na == 2) {
          const uint64_t a2 = adesc + (A_TILE >> 4);
          umma<F8>(tmem + acc_cols, a2, bdesc, idesc, acc);
          umma<F8>(tmem + acc_cols, a2 + 2, bdesc + 2, idesc, 1u);
          umma<F8>(tmem + acc_cols, a2 + 4, bdesc + 4, idesc, 1u);
          umma<F8>(tmem + acc_cols, a2 + 6, bdesc + 6, idesc, 1u);
        }
        umma_commit(empty0 + s * 8);
        acc = 1u;
        if (++s == p.stages) { s = 0; par ^= 1u; }
      }
      umma_commit(sa(&ctl.accum));   // fires when every MMA above has completed
    }
  } else {
    if (NA == 1 && p.x_warps) {
      if (p.pdl) wait_for_prerequisites();
      fetch_rows(p, ctl, smem + A_TILE, stage_bytes, kb0, n_it, x0, m_end - m0, warp - 2, lane);
    }
    if (sent) {
      if (p.pdl) wait_for_prerequisites();
      ahead = sums_ahead<BF16>(p, o, ks, 0, n0, m0, m_end, warp & 3, lane);
      cluster_wait();             // everybody's barrier is there
    }
    if (p.pdl) wait_for_prerequisites();                // the residual and the output are others' until here
    const bool done = warp_wait(sa(&ctl.accum), 0, &ctl.abort);
    if (!done) give_up(ctl, p.error_flag, 24);
    fence_after();
    if (done && fetched) leave_sums(p, tmem, warp & 3, lane, 0, 1, reinterpret_cast<float *>(smem));
    if (done && !sent && !fetched) {
      if constexpr (BF16) {
        const int a = (warp - 2) >> 2;    // (each accumulator has four warps: nothing else runs on the SM while a tile of 256 x 256 leaves)
        if (a < na) epilogue_bf16<EXT>(p, tmem + a * acc_cols, warp & 3, lane, n0 + a * BM, m0, m_end);
      } else {
        epilogue_fp16<FMT == PT_W_FP16>(p, o, tmem, warp & 3, lane, 0, 1, n0, m0);
      }
    }
  }
  if (sent) {
    if (warp < 2) cluster_wait();
    if (p.pdl) wait_for_prerequisites();
    sum_cluster<BF16, EXT, FMT == PT_W_FP16>(p, o, ctl, tmem, smem, ks, n0, m0, m_end, warp < 2 ? -1 : 0, 1, warp & 3, lane, ahead);
  } else if (fetched) {
    if (p.pdl) wait_for_prerequisites();
    fetch_sums<BF16, EXT, FMT == PT_W_FP16>(p, o, ctl, smem_s, ks, n0, m0, m_end, 64 + 128);
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (ctl.abort) end_after_failure(ctl, sa(&ctl.full[0]), issued, p.stages, warp, sent || fetched ? p.ksplit : 1);
  if (warp == 1) tmem_dealloc(tmem, tmem_cols);
}

// ------------------------------------------------------------------------------------------ INT4
// Weights go through the tensor memory: a transform warp turns a thread's row of a raw tile (128 nibbles) into 64 registers of fp16 pairs and
// stores them to 64 tensor-memory columns, where the MMA reads its A operand (lane = weight row); shared memory holds only the raw ring
// and the activations.  NG groups of four transform warps (one warp per quarter of the lanes) take the steps of 128 k in turn, so that the
// chain of a step - raw tile, nibbles, slot free, tensor memory, MMA - overlaps with that of its neighbours.
// What bounds it: up to about 100 activation rows the instructions of the single-thread roles and of the transform, beyond it the MMAs
// (8 x mb / 2 cycles a step).  A wait costs a single thread a hundred cycles or more even when nothing is left to wait for, so a step has ONE
// barrier in front of the MMAs (activations and weights arrive on the same one) and is 128 k deep.  The form before this one (64 k a
// step, fp16 tiles through shared memory, eight warps in step) took 1500 cycles per 64 k whatever the number of rows.  Measured on B200,
// 12288 x 4096 / 4096 x 11008, before and after: 16 rows 35 / 39 and 14.5 / 13 us, 511 rows 105 / 164 and 44.5 / 41 us (1150 TFLOP/s).
// The groups run apart, and a wait tells only odd from even uses of a barrier.  A group that has done step i waits next for use (i + NG) / S of
// slot (i + NG) % S; that the use before it is over follows from step i - S being over (which step i waited for) only if NG <= S.  The
// same for a raw stage, whose copies may land in any order: R >= NG + S.
// Dynamic shared memory: [slot][activations: two halves of 64 k, mb * 128 B each][raw stage][8 KB of packed nibbles].
template <int NG, Sums SUMS>
__global__ void __launch_bounds__((3 + 4 * NG) * 32, NG == 2 ? 2 : 1) gemm_int4_kernel(const __grid_constant__ CUtensorMap map_x, const GemmParams p) {
  // warp 0: raw tiles, warp 1: MMA, then 4 NG transform + epilogue, last: activations
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ SharedCtl ctl;
  unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int n0 = blockIdx.x * BM, m0 = blockIdx.z * p.mb, ks = blockIdx.y;
  const int st0 = ks * p.kb_per_split, n_it = min(p.n_kb, st0 + p.kb_per_split) - st0;   // (in steps)
  const int S = p.stages, R = p.raw_stages;
  const uint32_t half_bytes = (uint32_t)p.mb * BKB, slot_bytes = 2 * half_bytes;          // (half: a multiple of 2 KB)
  unsigned char *raw_ring = smem + (size_t)S * slot_bytes;
  const uint32_t smem_s = sa(smem);
  const bool sent = SUMS == SENT && p.ksplit > 1, fetched = SUMS == FETCHED && p.ksplit > 1;
  const uint32_t a_col = (uint32_t)(p.mb + 31) & ~31u, tmem_cols = p.tmem_columns;

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(sa(&ctl.full[s]), 5);    // the activations of the slot have landed; one arrival per warp of a group: its fp16 weights are in tensor memory
      mbar_init(sa(&ctl.empty[s]), 1);   // the MMAs that read the slot have completed
    }
    for (int r = 0; r < R; ++r) {
      mbar_init(sa(&ctl.raw_full[r]), 1);
      mbar_init(sa(&ctl.raw_empty[r]), 4);
    }
    mbar_init(sa(&ctl.accum), 1);
    if (sent) expect_sums(p, ctl, ks, m0, p.M);
    ctl.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (sent) cluster_arrive();
  if (warp == 1) tmem_alloc(sa(&ctl.tmem_base), tmem_cols);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = ctl.tmem_base;
  const Fp16Out &o = p.o[0];
  int issued = 0;                   // stages that this thread has asked for
  if (p.pdl) launch_dependents();   // not before the tensor memory is ours: a block of the next GEMM would keep it while it waits for this kernel

  if (warp == 0) {
    // ---- raw nibble tiles: one contiguous bulk copy per step (weights: nobody before has written them)
    if (elect_one()) {
      const unsigned char *wt = p.w + ((size_t)blockIdx.x * p.n_kb + st0) * RAW_STEP;
      const uint32_t raw0 = sa(raw_ring), full0 = sa(&ctl.raw_full[0]), empty0 = sa(&ctl.raw_empty[0]);
      int r = 0;
      uint32_t par = 1;
      for (int it = 0; it < n_it; ++it) {
        if (it >= R && !wait_fast<0>(empty0 + r * 8, par, &ctl.abort)) { give_up(ctl, p.error_flag, 21); break; }
        issued = it + 1;
        const uint32_t fb = full0 + r * 8;
        mbar_expect_tx(fb, RAW_STEP);
        bulk_g2s(raw0 + r * RAW_STEP, wt, RAW_STEP, fb);
        wt += RAW_STEP;
        if (++r == R) { r = 0; par ^= 1u; }
      }
    }
  } else if (warp == 2 + 4 * NG) {
    // ---- activation tiles (two boxes of 64 fp16 of k per row)
    if (elect_one()) {
      if (p.pdl) wait_for_prerequisites();
      const uint32_t full0 = sa(&ctl.full[0]), empty0 = sa(&ctl.empty[0]);
      int s = 0, kx = st0 * 128;
      uint32_t par = 1;
      for (int it = 0; it < n_it; ++it) {
        if (it >= S && !wait_fast<0>(empty0 + s * 8, par, &ctl.abort)) { give_up(ctl, p.error_flag, 25); break; }
        issued = it + 1;
        const uint32_t fb = full0 + s * 8, dst = smem_s + s * slot_bytes;
        mbar_expect_tx(fb, slot_bytes);
        tma_load_2d(dst, &map_x, kx, m0, fb);
        tma_load_2d(dst + half_bytes, &map_x, kx + 64, m0, fb);
        kx += 128;
        if (++s == S) { s = 0; par ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = instr_desc(false, p.mb);
      const uint64_t bdesc0 = smem_desc_sw128(smem_s);
      const uint32_t full0 = sa(&ctl.full[0]), empty0 = sa(&ctl.empty[0]), slot16 = slot_bytes >> 4, half16 = half_bytes >> 4;
      int s = 0;
      uint32_t par = 0, acc = 0;
      for (int it = 0; it < n_it; ++it) {
        if (!wait_fast<0>(full0 + s * 8, par, &ctl.abort)) { give_up(ctl, p.error_flag, 22); break; }
        fence_after();
        const uint64_t b0 = bdesc0 + (uint64_t)(s * slot16), b1 = b0 + half16;
        const uint32_t at = tmem + a_col + s * 64;
        umma_ta(tmem, at, b0, idesc, acc);   // eight MMAs of 16 k each: 32 bytes of an activation row, eight columns of weights
        umma_ta(tmem, at + 8, b0 + 2, idesc, 1u);
        umma_ta(tmem, at + 16, b0 + 4, idesc, 1u);
        umma_ta(tmem, at + 24, b0 + 6, idesc, 1u);
        umma_ta(tmem, at + 32, b1, idesc, 1u);
        umma_ta(tmem, at + 40, b1 + 2, idesc, 1u);
        umma_ta(tmem, at + 48, b1 + 4, idesc, 1u);
        umma_ta(tmem, at + 56, b1 + 6, idesc, 1u);
        umma_commit(empty0 + s * 8);
        acc = 1u;
        if (++s == S) { s = 0; par ^= 1u; }
      }
      umma_commit(sa(&ctl.accum));
    }
  } else {
    // ---- transform + epilogue.  A warp reaches tensor-memory lanes [32 (warp % 4), +32): thread (warp, lane) owns row 32 (warp % 4) + lane.
    const int q = warp & 3, group = (warp - 2) >> 2;
    const int row = q * 32 + lane;
    const int ngroups = p.K / p.group;
    const __half *srow = p.scales + (size_t)min(n0 + row, p.N - 1) * ngroups;
    const __half2 offA = __float2half2_rn(1032.0f), offB = __float2half2_rn(72.0f);
    const uint32_t raw_full0 = sa(&ctl.raw_full[0]), raw_empty0 = sa(&ctl.raw_empty[0]), empty0 = sa(&ctl.empty[0]), full0 = sa(&ctl.full[0]);
    const unsigned char *raw_mine = raw_ring + row * 32;
    const uint32_t a_lane = tmem + ((uint32_t)(q * 32) << 16) + a_col;
    // scale index of a step: it moves on every (group / 128) steps
    const int steps_per_group = p.group / 128;
    int gidx = (st0 + group) / steps_per_group, gpos = (st0 + group) % steps_per_group;
    int r = group % R, s = group % S;
    uint32_t rpar = (group / R) & 1, spar = ((group / S) & 1) ^ 1;
    __half sc_next = group < n_it ? __ldg(srow + gidx) : __half(0);
    for (int it = group; it < n_it; it += NG) {
      const __half2 s2 = __half2half2(sc_next);
      gpos += NG;
      while (gpos >= steps_per_group) { gpos -= steps_per_group; ++gidx; }
      if (it + NG < n_it) sc_next = __ldg(srow + gidx);   // the next step's scale: its latency hides behind this step
      if (!warp_wait<0>(raw_full0 + r * 8, rpar, &ctl.abort)) { give_up(ctl, p.error_flag, 23); break; }
      uint32_t words[16];
#pragma unroll
      for (int h = 0; h < 4; ++h)
        *reinterpret_cast<uint4 *>(&words[4 * h]) = *reinterpret_cast<const uint4 *>(raw_mine + (size_t)r * RAW_STEP + (h >> 1) * RAW_TILE + (h & 1) * 16);
      if (it >= S && !warp_wait<0>(empty0 + s * 8, spar, &ctl.abort)) { give_up(ctl, p.error_flag, 26); break; }
      fence_after();
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t v[32];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          // a word holds eight consecutive k as offset-binary nibbles u = q + 8: bits [0,4) k0, [16,20) k1, [4,8) k2, [20,24) k3, and the
          // same again one byte up for k4..k7.  (1024 + u) and (64 + u) are exact in fp16; subtracting the offsets is exact; the
          // product with the scale is the one fp16 rounding of the reference's Int4ToHalf.
          const uint32_t w = words[8 * half + c], w8 = w >> 8;
          __half2 h[4];
          *reinterpret_cast<uint32_t *>(&h[0]) = (w & 0x000F000Fu) | 0x64006400u;
          *reinterpret_cast<uint32_t *>(&h[1]) = (w & 0x00F000F0u) | 0x54005400u;
          *reinterpret_cast<uint32_t *>(&h[2]) = (w8 & 0x000F000Fu) | 0x64006400u;
          *reinterpret_cast<uint32_t *>(&h[3]) = (w8 & 0x00F000F0u) | 0x54005400u;
          h[0] = __hmul2(__hsub2(h[0], offA), s2);
          h[1] = __hmul2(__hsub2(h[1], offB), s2);
          h[2] = __hmul2(__hsub2(h[2], offA), s2);
          h[3] = __hmul2(__hsub2(h[3], offB), s2);
#pragma unroll
          for (int j = 0; j < 4; ++j) v[4 * c + j] = *reinterpret_cast<const uint32_t *>(&h[j]);
        }
        tmem_st32(a_lane + s * 64 + half * 32, v);
      }
      tmem_wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(full0 + s * 8);
        mbar_arrive(raw_empty0 + r * 8);   // the nibbles have been used (not merely asked for): the raw stage may be refilled
      }
      r += NG;
      while (r >= R) { r -= R; rpar ^= 1u; }
      s += NG;
      while (s >= S) { s -= S; spar ^= 1u; }
    }
    if (sent) {
      if (p.pdl) wait_for_prerequisites();
      cluster_wait();             // everybody's barrier is there
    }
    if (p.pdl) wait_for_prerequisites();                // the residual and the output are others' until here
    const bool done = warp_wait(sa(&ctl.accum), 0, &ctl.abort);
    if (!done) give_up(ctl, p.error_flag, 24);
    fence_after();
    if (done && fetched) leave_sums(p, tmem, q, lane, group, NG, reinterpret_cast<float *>(smem));
    if (done && !sent && !fetched) epilogue_fp16<false>(p, o, tmem, q, lane, group, NG, n0, m0);
  }
  if (sent) {
    const bool idle = warp < 2 || warp == 2 + 4 * NG;
    if (idle) cluster_wait();
    SumAhead ahead{};
    ahead.pairs = fp16_pairs(o, n0 + (warp & 3) * 32);
    if (p.pdl) wait_for_prerequisites();
    sum_cluster<false, false>(p, o, ctl, tmem, smem, ks, n0, m0, p.M, idle ? -1 : (warp - 2) >> 2, NG, warp & 3, lane, ahead);
  } else if (fetched) {
    if (p.pdl) wait_for_prerequisites();
    fetch_sums<false, false>(p, o, ctl, smem_s, ks, n0, m0, p.M, (3 + 4 * NG) * 32);
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (ctl.abort) end_after_failure(ctl, warp == 0 ? sa(&ctl.raw_full[0]) : sa(&ctl.full[0]), issued, warp == 0 ? R : S, warp, sent || fetched ? p.ksplit : 1);
  if (warp == 1) tmem_dealloc(tmem, tmem_cols);
}

// ------------------------------------------------------------------------------------------ load-time tiling
// FP8 bytes W[n, k] (k contiguous; BF16: k counts bytes) -> tiles [n tile][k block of 128 bytes]: 16 KB each, the image of a 128 x 128-byte tile under the
// 128-byte swizzle (row r at (r / 8) * 1024 + (r % 8) * 128, its 16-byte chunk c at position c ^ (r % 8)); rows beyond n are zero.
__global__ void fp8_tile_kernel(const uint4 *__restrict__ src, uint4 *__restrict__ dst, int n, int k, int n_kb, size_t n_units) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n_units; i += (size_t)gridDim.x * blockDim.x) {
    const int u = (int)(i % 1024);            // 16-byte unit inside the tile
    const size_t tile = i / 1024;
    const int kb = (int)(tile % n_kb), nt = (int)(tile / n_kb);
    const int grp = u >> 6, r8 = (u >> 3) & 7, pc = u & 7;   // destination: 8-row group, row in it, physical chunk
    const int row = nt * BM + grp * 8 + r8, c = pc ^ r8;
    dst[i] = row < n ? src[((size_t)row * k + (size_t)kb * 128) / 16 + c] : make_uint4(0, 0, 0, 0);
  }
}
// Reference int4 rows (int8 [n, k/2]: byte j = k 2j in the high nibble, k 2j+1 in the low, two's complement) -> tiles
// [n tile][k block of 64]: 4 KB each, [128 rows][32 bytes]; a word holds eight consecutive k as offset-binary nibbles in the order
// the transform warps split with two masks: bits [0,4) k0, [16,20) k1, [4,8) k2, [20,24) k3, [8,12) k4, [24,28) k5, [12,16) k6,
// [28,32) k7.  Rows beyond n hold q = 0.
__global__ void int4_tile_kernel(const uint32_t *__restrict__ src, uint32_t *__restrict__ dst, int n, int k, int n_kb, size_t n_words) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n_words; i += (size_t)gridDim.x * blockDim.x) {
    const int wi = (int)(i % 1024);           // word inside the tile: row * 8 + word of the row
    const size_t tile = i / 1024;
    const int kb = (int)(tile % n_kb), nt = (int)(tile / n_kb);
    const int row = nt * BM + (wi >> 3), w = wi & 7;
    uint32_t o = 0x88888888u;
    if (row < n) {
      const uint32_t b = src[((size_t)row * (k / 2) + (size_t)kb * 32) / 4 + w];   // four bytes = k 0..7 of this word
      o = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t byte = (b >> (8 * j)) & 0xFFu;
        const uint32_t even = ((byte >> 4) ^ 8u) & 0xFu, odd = (byte ^ 8u) & 0xFu;   // k = 2j, 2j + 1
        o |= even << (4 * j);
        o |= odd << (16 + 4 * j);
      }
    }
    dst[i] = o;
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)ptr;
  }
  return fn;
}

// 2-D row-major byte/fp16 matrix [rows][row_bytes]: box = box_bytes x box_rows.
static int make_map(CUtensorMap *map, const void *base, CUtensorMapDataType dt, int elem_bytes, uint64_t row_elems, uint64_t rows, uint32_t box_elems,
                    uint32_t box_rows, CUtensorMapSwizzle sw) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return pt::set_error(PT_ERR_CUDA, "pt_gemm: cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[2] = {row_elems, rows};
  const cuuint64_t strides[1] = {row_elems * (uint64_t)elem_bytes};
  const cuuint32_t box[2] = {box_elems, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, dt, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return pt::set_error(PT_ERR_CUDA, "pt_gemm: cuTensorMapEncodeTiled failed (%d)", (int)r);
  return PT_OK;
}

}  // namespace tc
}  // namespace pt

using namespace pt;

extern "C" size_t pt_gemm_packed_bytes(int wfmt, int n_out, int k_in) {
  const size_t rows = (size_t)ceil_div(n_out, tc::BM) * tc::BM;
  return wfmt == PT_W_INT4 ? rows * (size_t)(k_in / 2) : rows * (size_t)k_in * (wfmt == PT_W_FP8 ? 1 : 2);
}

extern "C" int pt_gemm_repack(int wfmt, const void *w, int n_out, int k_in, void *packed, void *stream) {
  PT_REQUIRE(wfmt == PT_W_INT4 || wfmt == PT_W_FP8 || wfmt == PT_W_BF16 || wfmt == PT_W_FP16, "pt_gemm_repack: unknown weight format %d", wfmt);
  PT_REQUIRE(w && packed && w != packed, "pt_gemm_repack: needs distinct source and destination buffers");
  PT_REQUIRE(((uintptr_t)w & 15) == 0 && ((uintptr_t)packed & 15) == 0, "pt_gemm_repack: buffers must be 16-byte aligned");
  const int k_step = wfmt == PT_W_BF16 || wfmt == PT_W_FP16 ? 64 : 128;
  PT_REQUIRE(n_out > 0 && k_in > 0 && k_in % k_step == 0, "pt_gemm_repack: k_in=%d must be a positive multiple of %d", k_in, k_step);
  const int n_tiles = ceil_div(n_out, tc::BM);
  if (wfmt == PT_W_INT4) {
    const int n_kb = k_in / 64;
    const size_t n_words = (size_t)n_tiles * n_kb * 1024;
    tc::int4_tile_kernel<<<sm_count() * 8, 256, 0, as_stream(stream)>>>((const uint32_t *)w, (uint32_t *)packed, n_out, k_in, n_kb, n_words);
  } else {
    const int k_bytes = wfmt == PT_W_FP8 ? k_in : 2 * k_in, n_kb = k_bytes / 128;
    const size_t n_units = (size_t)n_tiles * n_kb * 1024;
    tc::fp8_tile_kernel<<<sm_count() * 8, 256, 0, as_stream(stream)>>>((const uint4 *)w, (uint4 *)packed, n_out, k_bytes, n_kb, n_units);
  }
  PT_LAUNCH_CHECK("pt_gemm_repack");
  return PT_OK;
}

// What a caller has to hand over for k-slices that it asks for, from when they were summed in global memory.  (Nothing touches it now: the slices
// of a tile meet in the shared memory of a cluster.  What was refused without it still is.)
constexpr size_t kGemmCounterBytes = 65536;
constexpr size_t kGemmMaxCounters = kGemmCounterBytes / sizeof(int);

constexpr int kGemmSmem = 220 * 1024;   // dynamic shared memory that a launch may ask for

extern "C" size_t pt_gemm_workspace_bytes(int m, int n_out, int max_ksplit) {
  return kGemmCounterBytes + (size_t)max_ksplit * m * n_out * sizeof(float);
}

extern "C" int pt_gemm(const pt_gemm_args *a, void *stream) {
  PT_REQUIRE(a, "pt_gemm: null args");
  PT_REQUIRE(a->wfmt == PT_W_INT4 || a->wfmt == PT_W_FP8 || a->wfmt == PT_W_BF16 || a->wfmt == PT_W_FP16, "pt_gemm: unknown weight format %d", a->wfmt);
  const bool int4 = a->wfmt == PT_W_INT4, bf16 = a->wfmt == PT_W_BF16, fp16 = a->wfmt == PT_W_FP16;
  const int k_step = bf16 || fp16 ? 64 : 128;
  PT_REQUIRE(a->m >= 1 && a->n_out >= 1 && a->k_in >= k_step && a->k_in % k_step == 0, "pt_gemm: bad shape m=%d n_out=%d k_in=%d (k_in a multiple of %d)",
             a->m, a->n_out, a->k_in, k_step);
  PT_REQUIRE(a->x && a->w && (a->out || a->n_parts), "pt_gemm: null x / w / out");
  PT_REQUIRE(((uintptr_t)a->x & 15) == 0 && ((uintptr_t)a->w & 15) == 0, "pt_gemm: x and w must be 16-byte aligned");
  if (bf16) {
    PT_REQUIRE(dense_epilogue_known(a->epilogue), "pt_gemm: BF16 epilogue %d (store, relu2, glu, gelu-mul, softcap or xielu)", a->epilogue);
    const char *bad = dense_ext_error(a->epilogue, a->n_out, a->ext);
    PT_REQUIRE(!bad, "pt_gemm: %s", bad);
    PT_REQUIRE(a->out_dtype == PT_DT_BF16 || a->out_dtype == PT_DT_F32, "pt_gemm: BF16 weights write bf16 or fp32, got type %d", a->out_dtype);
  } else {
    PT_REQUIRE(a->epilogue == PT_EPI_STORE || a->epilogue == PT_EPI_RESIDUAL || a->epilogue == PT_EPI_BIAS || ((int4 || fp16) && a->epilogue == PT_EPI_SWIGLU) ||
                   (fp16 && (a->epilogue == PT_EPI_BIAS_GELU || a->epilogue == PT_EPI_BIAS_RESIDUAL || a->epilogue == PT_EPI_RELU2 || a->epilogue == PT_EPI_GATED_RESIDUAL)),
               "pt_gemm: epilogue %d (store, residual or bias; INT4 and FP16: swiglu; FP16: relu2, gated residual, bias with gelu or residual)", a->epilogue);
    PT_REQUIRE(a->epilogue != PT_EPI_SWIGLU || a->n_out % 16 == 0, "pt_gemm: SwiGLU epilogue needs n_out %% 16 == 0, got %d", a->n_out);
  }
  const bool wants_bias = a->epilogue == PT_EPI_BIAS || a->epilogue == PT_EPI_BIAS_GELU || a->epilogue == PT_EPI_BIAS_RESIDUAL;
  const bool gated = !bf16 && a->epilogue == PT_EPI_GATED_RESIDUAL;
  const bool wants_residual = a->epilogue == PT_EPI_RESIDUAL || a->epilogue == PT_EPI_BIAS_RESIDUAL || gated;
  PT_REQUIRE(!wants_residual || a->residual, "pt_gemm: residual epilogue needs residual");
  PT_REQUIRE(!wants_bias || a->bias, "pt_gemm: bias epilogue needs bias");
  PT_REQUIRE(!gated || a->gate, "pt_gemm: gated residual epilogue needs gate");
  if (a->n_parts) {
    PT_REQUIRE(fp16 && a->parts && a->n_parts >= 1 && a->n_parts <= tc::MAX_PARTS && a->epilogue == PT_EPI_STORE, "pt_gemm: 1 to %d parts are for FP16, with epilogues of their own",
               tc::MAX_PARTS);
    long long n = 0;
    for (int i = 0; i < a->n_parts; ++i) {
      const pt_gemm_part &part = a->parts[i];
      PT_REQUIRE(part.out && part.n_out >= 1 && (i + 1 == a->n_parts || part.n_out % tc::BM == 0) && (part.epilogue == PT_EPI_STORE || part.epilogue == PT_EPI_RELU2),
                 "pt_gemm: part %d: n_out=%d (a multiple of %d but in the last), epilogue %d (store or relu2)", i, part.n_out, tc::BM, part.epilogue);
      n += part.n_out;
    }
    PT_REQUIRE(n == a->n_out, "pt_gemm: the parts have %lld rows, n_out=%d", n, a->n_out);
  }
  PT_REQUIRE(a->wfmt == PT_W_FP8 || a->w_tiled, "pt_gemm: INT4, BF16 and FP16 weights must be tiled with pt_gemm_repack");
  if (int4)
    PT_REQUIRE(a->scales && a->group >= 128 && a->group % 128 == 0 && a->k_in % a->group == 0,
               "pt_gemm: INT4 needs scales and a group (%d) that is a multiple of 128 dividing k_in=%d", a->group, a->k_in);

  const int out_ld = a->out_ld > 0 ? a->out_ld : (a->epilogue == PT_EPI_SWIGLU ? a->n_out / 2 : a->n_out);
  if (few::takes(*a)) {
    const cudaError_t e = few::run(*a, out_ld, as_stream(stream));
    if (e != cudaSuccess) return pt::set_error(PT_ERR_CUDA, "pt_gemm: %s", cudaGetErrorString(e));
    PT_LAUNCH_CHECK("pt_gemm");
    return PT_OK;
  }
  tc::GemmParams p{};
  p.M = a->m; p.N = a->n_out; p.K = a->k_in;
  p.group = int4 ? a->group : 0;
  p.w_tiled = a->w_tiled ? 1 : 0;
  p.w = (const unsigned char *)a->w;
  const bool grouped = bf16 && a->ext && a->ext->n_groups > 0;
  if (grouped) {
    const int rows = a->ext->group_rows;
    PT_REQUIRE(rows % 16 == 0 && rows >= 16 && rows <= 256 && a->m % rows == 0 && a->m / rows <= 65535, "pt_gemm: groups of %d rows (16 .. 256 in steps of 16) in %d rows",
               rows, a->m);
    p.group_of = a->ext->group_of;
    p.group_used = a->ext->group_used;
    p.group_stride = pt_gemm_packed_bytes(a->wfmt, a->n_out, a->k_in);
  }
  const tc::GemmPlan plan = tc::plan_gemm({int4, bf16, fp16, a->m, a->n_out, a->k_in, a->ksplit, grouped ? a->ext->group_rows : 0, sm_count()});
  PT_REQUIRE(plan.fits, "pt_gemm: tile does not fit shared memory");
  p.mb = plan.mb; p.n_kb = plan.n_kb; p.ksplit = plan.ksplit; p.kb_per_split = plan.kb_per_split;
  p.stages = plan.stages; p.raw_stages = plan.raw_stages; p.tmem_columns = plan.tmem_columns;
  p.n_tiles = plan.n_tiles;
  p.x = (const unsigned char *)a->x;
  p.x_pitch = (size_t)a->k_in * (bf16 || fp16 || int4 ? 2 : 1);
  p.x_warps = plan.x_warps;
  p.sum_offset = plan.sum_offset;
  p.scales = (const __half *)a->scales;
  p.o[0] = {(__half *)a->out, wants_residual ? (const __half *)a->residual : nullptr, wants_bias ? (const __half *)a->bias : nullptr, gated ? (const __half *)a->gate : nullptr, out_ld,
            a->n_out, a->epilogue, a->halve, int4 ? 1.0f : (a->x_scale > 0.f ? a->x_scale : 1.0f) * (a->w_scale > 0.f ? a->w_scale : 1.0f)};
  p.n_parts = std::max(1, a->n_parts);
  for (int i = 0, tile = 0; i < a->n_parts; ++i) {
    const pt_gemm_part &part = a->parts[i];
    p.part_tile[i] = tile;
    p.o[i] = {(__half *)part.out, nullptr, nullptr, nullptr, part.n_out, part.n_out, part.epilogue, 0, p.o[0].scale};
    tile += ceil_div(part.n_out, tc::BM);
  }
  if (bf16) p.dense = make_dense_out(a->out, out_ld, a->out_dtype, a->epilogue, a->alpha, a->ext);
  p.error_flag = a->error_flag;
  if (a->ksplit > 1 && p.ksplit > 1) {   // slices that the caller asked for
    const size_t need = pt_gemm_workspace_bytes(a->m, a->n_out, p.ksplit);
    PT_REQUIRE(a->workspace && a->workspace_bytes >= need, "pt_gemm: %d k-slices need %zu workspace bytes, got %zu", p.ksplit, need, a->workspace_bytes);
    PT_REQUIRE((size_t)plan.n_tiles * plan.m_tiles <= kGemmMaxCounters, "pt_gemm: %d x %d tiles exceed the %zu arrival counters of a k-slice workspace", plan.n_tiles,
               plan.m_tiles, kGemmMaxCounters);
  }
  // Row-major weights are an operand of a plain product, which the kernel before may have written: nothing of them is read early.
  p.pdl = a->pdl && p.w_tiled ? 1 : 0;

  CUtensorMap map_w, map_x;
  memset(&map_w, 0, sizeof(map_w));
  if (int4 || fp16) {
    if (int rc = tc::make_map(&map_x, a->x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (uint64_t)a->k_in, (uint64_t)a->m * p.n_parts, 64, (uint32_t)p.mb, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
  } else if (bf16) {
    if (int rc = tc::make_map(&map_x, a->x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)a->k_in, (uint64_t)a->m, 64, (uint32_t)p.mb, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
  } else {
    if (!p.w_tiled)
      if (int rc = tc::make_map(&map_w, a->w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)a->k_in, (uint64_t)a->n_out, 128, tc::BM, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    if (int rc = tc::make_map(&map_x, a->x, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)a->k_in, (uint64_t)a->m, 128, (uint32_t)p.mb, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
  }
  dim3 grid(ceil_div(plan.n_tiles, plan.na), p.ksplit, plan.m_tiles);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(plan.threads);
  cfg.dynamicSmemBytes = plan.smem;
  cfg.stream = as_stream(stream);
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  if (p.ksplit > 1) {   // the k-slices of a tile: one cluster
    attr[n_attr].id = cudaLaunchAttributeClusterDimension;
    attr[n_attr].val.clusterDim.x = 1;
    attr[n_attr].val.clusterDim.y = p.ksplit;
    attr[n_attr++].val.clusterDim.z = 1;
  }
  if (p.pdl) {
    attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n_attr++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n_attr;
  cudaError_t e;
  if (int4) {
    static std::atomic<uint64_t> allowed[4];
    const auto kernel = plan.int4_groups == 2 ? (plan.few ? tc::gemm_int4_kernel<2, tc::SENT> : tc::gemm_int4_kernel<2, tc::FETCHED>)
                                              : (plan.few ? tc::gemm_int4_kernel<4, tc::SENT> : tc::gemm_int4_kernel<4, tc::FETCHED>);
    PT_CUDA(allow_smem(kernel, kGemmSmem, allowed[2 * (plan.int4_groups == 2) + plan.few]));
    e = cudaLaunchKernelEx(&cfg, kernel, map_x, p);
  } else {
    const bool ext = bf16 && dense_needs_ext(a->epilogue, a->ext);
    static std::atomic<uint64_t> allowed[10];
    const auto kernel = plan.na == 2 ? (ext ? tc::gemm_dense_kernel<PT_W_BF16, 2, true, tc::FETCHED> : tc::gemm_dense_kernel<PT_W_BF16, 2, false, tc::FETCHED>)
                        : fp16       ? (plan.few ? tc::gemm_dense_kernel<PT_W_FP16, 1, false, tc::SENT> : tc::gemm_dense_kernel<PT_W_FP16, 1, false, tc::FETCHED>)
                        : !bf16      ? (plan.few ? tc::gemm_dense_kernel<PT_W_FP8, 1, false, tc::SENT> : tc::gemm_dense_kernel<PT_W_FP8, 1, false, tc::FETCHED>)
                        : ext        ? (plan.few ? tc::gemm_dense_kernel<PT_W_BF16, 1, true, tc::SENT> : tc::gemm_dense_kernel<PT_W_BF16, 1, true, tc::FETCHED>)
                                     : (plan.few ? tc::gemm_dense_kernel<PT_W_BF16, 1, false, tc::SENT> : tc::gemm_dense_kernel<PT_W_BF16, 1, false, tc::FETCHED>);
    PT_CUDA(allow_smem(kernel, kGemmSmem, allowed[plan.na == 2 ? 8 + ext : 2 * (fp16 ? 0 : !bf16 ? 1 : 2 + ext) + plan.few]));
    e = cudaLaunchKernelEx(&cfg, kernel, map_w, map_x, p);
  }
  if (e != cudaSuccess) return pt::set_error(PT_ERR_CUDA, "pt_gemm: %s", cudaGetErrorString(e));
  PT_LAUNCH_CHECK("pt_gemm");
  return PT_OK;
}
