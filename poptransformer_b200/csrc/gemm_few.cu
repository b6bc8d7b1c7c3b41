// Small products of up to eight activation rows (decode steps): Y[m, n] = sum_k X[m, k] * W[n, k] of the fp16 or bf16 weights that pt_gemm_repack tiled.  pt_gemm
// comes here; the results are those of its tensor-memory kernel up to the order of the sums.
//
// What bounds such a product is the latency of a launch: what lies between the end of the kernel in front and the last store.  A warp multiplies 16
// weight rows (mma.sync m16n8k16, fp32 sums in registers) with the activations of a k block, straight from the shared memory where bulk copies have put
// the weights before the kernel in front had ended.  tcgen05 is the wrong tool here: an MMA of 128 weight rows and 16 k takes 75 cycles however few
// activation rows it has (the weights' way out of shared memory), so four k blocks that were there in time took 1200 cycles, and commit, tensor
// memory and its loads another 700.  Measured on B200, us a launch in a row of launches, that kernel / this one at 1 row: 768 x 768 3.1 / 2.3, 2304 x 768
// 3.4 / 2.6, 768 x 3072 4.2 / 3.4, 2048 x 512 3.8 / 2.3, 2048 x 2048 4.1 / 3.7, 50257 x 768 16.7 / 14.0; at 8 rows 768 x 768 3.2 / 2.5, 2048 x 2048 4.2 / 3.9.
// At 16 rows, and of larger matrices, the two are level or that one is faster (1 row, 4096 x 4096: 8.1 / 8.1).
//
// A block has `units` runs of 16 weight rows times `warps_k` warps that take k blocks in turn, and `slices` blocks of a cluster share k.  All parts of a
// sum meet in one step: every warp sends its 16 x 8 sums to the block that writes them, by stores that arrive at a barrier there, or with one
// slice through its own shared memory.  They are added in a fixed order.  Warp 0 fetches weights, warp 1 activations (16-byte asynchronous
// copies into the swizzled image that ldmatrix reads without conflicts).  What was asked of the epilogue (residual) is requested before the products.
// Every wait is bounded, as in gemm_tc.cu, and the meetings of a cluster wait for threads that come in bounded time or have ended.  After a failure the sums
// go out all the same, so that nobody's wait runs out for another's failure, and a block that gave up stays until nobody can send to it.
#include "dense_out.cuh"
#include "fp16_out.cuh"
#include "gemm_few.h"
#include "mbarrier.cuh"
#include "tile_math.cuh"

namespace pt {
namespace few {

struct Params {
  const unsigned char *w, *x;
  int B, n_rt, nchunks, chunks_per_split, xs_stride, pdl;   // activation rows, units, k blocks (in all / of a slice), bytes of an activation row
  int N, epilogue, out_ld;
  float scale;             // fp16 outputs: factor of a sum
  const __half *residual, *bias;
  __half *out;
  int *error_flag;
  DenseOut dense;          // BF16
};
struct Tile { int units, warps_k, stages; uint32_t stage_bytes, sum_offset; };

struct Ctl {
  uint64_t full[MAX_STAGES], empty[MAX_STAGES], sums;
  volatile int abort;
};
__device__ __forceinline__ void give_up(Ctl &ctl, int *error_flag, int code) {
  if (!ctl.abort && error_flag) atomicCAS(error_flag, 0, code);
  ctl.abort = 1;
}
// A wait that looks again and again for some microseconds before it lets itself be suspended, from which it would wake 250 cycles late (measured on B200).
__device__ __noinline__ bool wait_on(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  for (int i = 0; i < 500; ++i)
    if (mbar_test(bar, parity)) return true;
  return mbar_wait(bar, parity, abort_flag);
}
__device__ __forceinline__ bool wait_fast(uint32_t bar, uint32_t parity, volatile int *abort_flag) { return mbar_test(bar, parity) || wait_on(bar, parity, abort_flag); }
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) { return __all_sync(0xffffffffu, wait_fast(bar, parity, abort_flag)); }
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// A warp's way out of the kernel: if its block has given up, not before the others of the cluster.
__device__ __forceinline__ void leave(const Ctl &ctl, int slices) {
  if (slices > 1 && __any_sync(0xffffffffu, ctl.abort)) stay_for_cluster();
}
__device__ __forceinline__ uint32_t in_block(uint32_t local, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  return a;
}
__device__ __forceinline__ void send(uint32_t at, float v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(at), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}

template <bool BF16, bool EXT>
__global__ void __launch_bounds__(64 + 32 * MAX_WARPS, 2) linear_kernel(const Params p, const Tile t) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ Ctl ctl;
  unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int R = t.units, KW = t.warps_k, CW = R * KW, S = t.stages, slices = gridDim.y, rank = blockIdx.y;
  const int u0 = blockIdx.x * R, units = min(R, p.n_rt - u0);
  const int kb0 = rank * p.chunks_per_split, n_kb = min(p.nchunks, kb0 + p.chunks_per_split) - kb0, n_st = (n_kb + KW - 1) / KW;
  const int own = rank < units ? (units - rank + slices - 1) / slices : 0, parts = slices * KW;     // units that this block writes, parts of their sums
  const uint32_t ring = smem_addr(smem), full0 = smem_addr(&ctl.full[0]), empty0 = smem_addr(&ctl.empty[0]), w_bytes = KW * R * UNIT_BYTES;
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full0 + s * 8, 1 + 32);    // the weights, and every lane's copies of activations
      mbar_init(empty0 + s * 8, CW);
    }
    mbar_init(smem_addr(&ctl.sums), 1);
    if (slices > 1 && own) mbar_expect_tx(smem_addr(&ctl.sums), own * parts * (UNIT * 8 * 4));
    ctl.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (slices > 1) { __syncwarp(); asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
  __syncthreads();
  if (p.pdl) launch_dependents();

  if (warp == 1) {
    if (p.pdl) wait_for_prerequisites();
    const int c = lane & 7, inv_rows = 65536 / p.B + 1;
    for (int st = 0, s = 0, par = 1; st < n_st; ++st) {
      if (st >= S && !warp_wait(empty0 + s * 8, par, &ctl.abort)) { give_up(ctl, p.error_flag, 25); break; }
      const int rows = min(KW, n_kb - st * KW) * p.B;       // (k block, activation row) pairs, eight 16-byte units each
      const uint32_t dst = ring + s * t.stage_bytes + w_bytes;
      const unsigned char *src = p.x + (size_t)(kb0 + st * KW) * ROW_BYTES + c * 16;
#pragma unroll 4
      for (int i = lane >> 3; i < rows; i += 4) {
        const int j = (i * inv_rows) >> 16, row = i - j * p.B;       // (i < 128)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + j * (8 * ROW_BYTES) + row * ROW_BYTES + ((c ^ (row & 7)) << 4)), "l"(src + j * ROW_BYTES + (size_t)row * p.xs_stride) : "memory");
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full0 + s * 8) : "memory");
      if (++s == S) { s = 0; par ^= 1; }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp == 0) {
    if (lane == 0) {
      int st = 0;
      for (int s = 0, par = 1; st < n_st; ++st) {
        if (st >= S && !wait_fast(empty0 + s * 8, par, &ctl.abort)) { give_up(ctl, p.error_flag, 21); break; }
        const int kbs = min(KW, n_kb - st * KW);
        mbar_expect_tx(full0 + s * 8, kbs * units * UNIT_BYTES);
        for (int j = 0; j < kbs; ++j) {           // runs of units that lie in one tile of 128 weight rows are contiguous
          const size_t kb = kb0 + st * KW + j;
          for (int u = 0; u < units;) {
            const int in = (u0 + u) & 7, run = min(units - u, 8 - in);
            bulk_g2s(ring + s * t.stage_bytes + (j * R + u) * UNIT_BYTES, p.w + ((size_t)((u0 + u) >> 3) * p.nchunks + kb) * (8 * UNIT_BYTES) + in * UNIT_BYTES, run * UNIT_BYTES,
                     full0 + s * 8);
            u += run;
          }
        }
        if (++s == S) { s = 0; par ^= 1; }
      }
      mbar_wait_ring(full0, st, S);     // (long over when the others end, but for failures)
    }
    __syncwarp();
  }
  if (warp < 2) {
    if (slices > 1) { __syncwarp(); asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
    leave(ctl, slices);
    return;
  }

  // ---- a warp has unit u of the block and k block kw of every stage
  const int cw = warp - 2, u = cw % R, kw = cw / R, g = lane >> 2, tig = lane & 3;
  if (p.pdl) wait_for_prerequisites();
  // What the epilogue needs of memory is asked for now: the residual of the unit that this warp writes first.
  const int e_m = lane >> 2, e_n = (u0 + rank + cw * slices) * UNIT + (lane & 3) * 4;
  const bool residual = !BF16 && (p.epilogue == PT_EPI_RESIDUAL || p.epilogue == PT_EPI_BIAS_RESIDUAL);
  const bool res_whole = residual && p.N % 4 == 0 && ((uintptr_t)p.residual & 7) == 0;
  Half4 res{};
  if (residual && cw < own && e_m < p.B && e_n < p.N) res = load4(p.residual + (size_t)e_m * p.N + e_n, e_n, p.N, res_whole);

  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  const bool active = u < units;
  const uint32_t a_off = (kw * R + u) * UNIT_BYTES + ((lane >> 3) & 1) * 1024 + (lane & 7) * 128, b_off = w_bytes + kw * (8 * ROW_BYTES) + (lane & 7) * 128;
  for (int st = 0, s = 0, par = 0; st < n_st; ++st) {
    const uint32_t stage = ring + s * t.stage_bytes;
    if (!warp_wait(full0 + s * 8, par, &ctl.abort)) { give_up(ctl, p.error_flag, 22); break; }
    if (active && st * KW + kw < n_kb) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t b[4];
        ldmatrix_x4(stage + b_off + (((4 * h + (lane >> 3)) ^ (lane & 7)) << 4), b);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          uint32_t a[4];
          ldmatrix_x4(stage + a_off + (((4 * h + 2 * k + (lane >> 4)) ^ (lane & 7)) << 4), a);
          if constexpr (BF16) mma16816_bf16(acc, a[0], a[1], a[2], a[3], b[2 * k], b[2 * k + 1]);
          else mma16816(acc, a[0], a[1], a[2], a[3], b[2 * k], b[2 * k + 1]);
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty0 + s * 8);
    if (++s == S) { s = 0; par ^= 1; }
  }

  // ---- the parts of every sum meet: [unit of this block][slice, warp][8 activation rows][16 weight rows]
  const uint32_t sums = ring + t.sum_offset, mine = ((2 * tig) * 20 + g) * 4;
  if (slices > 1) {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");     // everybody's barrier is there
    if (active) {
      const int nth = u / slices, to = u - nth * slices;
      const uint32_t at = in_block(sums + (nth * parts + rank * KW + kw) * ITEM + mine, to), bar = in_block(smem_addr(&ctl.sums), to);
      send(at, acc[0], bar);
      send(at + 80, acc[1], bar);
      send(at + 32, acc[2], bar);
      send(at + 112, acc[3], bar);
    }
    if (cw >= own) { leave(ctl, slices); return; }
    if (!warp_wait(smem_addr(&ctl.sums), 0, &ctl.abort)) give_up(ctl, p.error_flag, 27);
  } else {
    if (active) {
      float *at = reinterpret_cast<float *>(smem + t.sum_offset + (u * parts + kw) * ITEM + mine);
      at[0] = acc[0];
      at[20] = acc[1];
      at[8] = acc[2];
      at[28] = acc[3];
    }
    if (KW > 1) asm volatile("bar.sync 1, %0;" ::"r"(CW * 32) : "memory");
    else __syncwarp();
  }
  if (__any_sync(0xffffffffu, ctl.abort)) { leave(ctl, slices); return; }
  for (int i = cw; i < own; i += CW) {
    const int m = lane >> 2, n = (u0 + rank + i * slices) * UNIT + (lane & 3) * 4;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    const unsigned char *from = smem + t.sum_offset + (size_t)i * parts * ITEM + (lane >> 2) * 80 + (lane & 3) * 16;
    for (int k0 = 0; k0 < parts; k0 += 8) {     // eight loads in flight
      float4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = k0 + k < parts ? *reinterpret_cast<const float4 *>(from + (k0 + k) * ITEM) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int k = 0; k < 8; ++k) { sum.x += v[k].x; sum.y += v[k].y; sum.z += v[k].z; sum.w += v[k].w; }
    }
    if constexpr (!BF16) { sum.x *= p.scale; sum.y *= p.scale; sum.z *= p.scale; sum.w *= p.scale; }
    const bool glu = BF16 ? p.dense.epilogue == PT_EPI_GLU && n < p.dense.split_n : p.epilogue == PT_EPI_SWIGLU;      // (the same in the whole warp)
    float4 up;
    if (glu) {   // weight rows 0 .. 7 of the unit are gates, 8 .. 15 their ups
      up.x = __shfl_xor_sync(0xffffffffu, sum.x, 2); up.y = __shfl_xor_sync(0xffffffffu, sum.y, 2);
      up.z = __shfl_xor_sync(0xffffffffu, sum.z, 2); up.w = __shfl_xor_sync(0xffffffffu, sum.w, 2);
    }
    if (m >= p.B || n >= p.N) continue;
    if constexpr (BF16) {
      if (glu) {
        if (!(lane & 2)) dense_store_glu4<EXT>(p.dense, m, n, sum, up);
      } else if (n + 4 <= p.N) {
        dense_store4<EXT>(p.dense, m, n, sum);
      } else {
        dense_store<EXT>(p.dense, m, n, sum.x);
        if (n + 1 < p.N) dense_store<EXT>(p.dense, m, n + 1, sum.y);
        if (n + 2 < p.N) dense_store<EXT>(p.dense, m, n + 2, sum.z);
      }
    } else {
      Half4 y;
      if (glu) {
        if (lane & 2) continue;
        const float a[4] = {sum.x, sum.y, sum.z, sum.w}, b[4] = {up.x, up.y, up.z, up.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) y.v[j] = h_mul(__float2half_rn(b[j]), swish_h(__float2half_rn(a[j])));
        const int f = n / 16 * 8 + n % 8;
        store4(p.out + (size_t)m * p.out_ld + f, y, f, p.N / 2);
        continue;
      }
      Half4 bias{};
      if (p.bias) bias = load4(p.bias + n, n, p.N, n + 4 <= p.N && ((uintptr_t)p.bias & 7) == 0);
      if (i != cw && residual) res = load4(p.residual + (size_t)m * p.N + n, n, p.N, res_whole);
      y = finish4<false>(p.epilogue, sum, res, bias);
      store4(p.out + (size_t)m * p.out_ld + n, y, n, p.N);
    }
  }
}

template <bool BF16, bool EXT> static cudaError_t launch(const Params &p, const Plan &plan, cudaStream_t st) {
  static std::atomic<uint64_t> allowed{0};
  if (const cudaError_t e = allow_smem(linear_kernel<BF16, EXT>, BUDGET, allowed)) return e;
  const Tile t{plan.units, plan.warps_k, plan.stages, plan.stage_bytes, plan.sum_offset};
  return launch_early(linear_kernel<BF16, EXT>, Grid(dim3(plan.blocks / plan.slices, plan.slices), plan.slices, p.pdl), dim3(64 + 32 * plan.units * plan.warps_k), plan.smem, st, p, t);
}

// Whether a product of checked arguments (pt_gemm) is one of these kernels'.
bool takes(const pt_gemm_args &a) {
  return (a.wfmt == PT_W_FP16 || a.wfmt == PT_W_BF16) && a.ksplit <= 0 && !a.n_parts && a.epilogue != PT_EPI_GATED_RESIDUAL && !(a.ext && a.ext->n_groups > 0) && small(a.m, a.n_out, a.k_in) && pays(a.n_out, a.k_in, sm_count());
}
cudaError_t run(const pt_gemm_args &a, int out_ld, cudaStream_t st) {
  const bool bf16 = a.wfmt == PT_W_BF16;
  const Plan &plan = kept_plan(a.m, a.n_out, a.k_in, sm_count());
  Params p{};
  p.w = (const unsigned char *)a.w;
  p.x = (const unsigned char *)a.x;
  p.B = a.m; p.N = a.n_out;
  p.n_rt = ceil_to(a.n_out, UNIT);
  p.nchunks = a.k_in / 64;
  p.chunks_per_split = plan.kb_per_slice;
  p.xs_stride = a.k_in * 2;
  p.pdl = a.pdl ? 1 : 0;
  p.epilogue = a.epilogue;
  p.out_ld = out_ld;
  p.scale = (a.x_scale > 0.f ? a.x_scale : 1.0f) * (a.w_scale > 0.f ? a.w_scale : 1.0f);
  p.residual = (const __half *)a.residual;
  p.bias = a.epilogue == PT_EPI_BIAS || a.epilogue == PT_EPI_BIAS_GELU || a.epilogue == PT_EPI_BIAS_RESIDUAL ? (const __half *)a.bias : nullptr;
  p.out = (__half *)a.out;
  p.error_flag = a.error_flag;
  if (!bf16) return launch<false, false>(p, plan, st);
  p.dense = make_dense_out(a.out, out_ld, a.out_dtype, a.epilogue, a.alpha, a.ext);
  return dense_needs_ext(a.epilogue, a.ext) ? launch<true, true>(p, plan, st) : launch<true, false>(p, plan, st);
}

}  // namespace few
}  // namespace pt
