// Paged KV cache: append of the new token fused with split flash-decode attention.
//
// A warp takes chunks of 16 keys (32 of head width 64) of one (sequence, kv head) on its own: K and V rows come into shared memory of its own by
// asynchronous copies, both products run on the tensor cores, and the softmax keeps a running maximum and sum, so that nothing but the end of the work
// makes warps meet.  The warps of a block and, where there are few (sequence, kv head) pairs and long tables, the blocks of a cluster share the chunks;
// what they leave is summed through shared memory in a fixed order, which keeps the result deterministic.
// The warp that has the position `step` writes the new k/v into the pool and takes them from shared memory itself, so the append costs no
// extra pass over the cache.
//
// HBM-bound: algorithmic bytes = 2 * (step + 1) * head_dim * 2 per (sequence, kv-head), read once.
#include <algorithm>

#include "common.cuh"
#include "mbarrier.cuh"

namespace pt {

struct AttnParams {
  int runs;        // blocks of a cluster, which share the keys of a (sequence, kv head, part)
  int B, n_head, n_kv, qpk, qsplit, H, page, max_pages, max_len, rope_mode, softmax_mode, rot_half, out_ld, pdl;
  __half scale_h;
  int use_scale;
  const int *step;
  const __half *qkv, *sin_t, *cos_t;
  __half *pool;
  const int *page_table;
  __half *out;
  uint8_t *out8;   // optional: the same output cast to E4M3 with inv_out_scale (the input of an FP8 linear), [B, n_head * H]
  float inv_out_scale;
  float2 *ws_ml;   // [B, n_head, max_pages]: maximum and sum of the first warps that have keys
  int *error_flag;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// RoPE on one head vector (fp16), with the reference's fp16 roundings, sixteen channels (unit u) at a time: two runs of eight.
// Llama (rotate_half): y_j = fp16(fp16(x_j c_j) + fp16(-x_{j+H/2} s_j)), y_{j+H/2} = fp16(fp16(x_{j+H/2} c_j) + fp16(x_j s_j)).
// ChatGLM2: only the first H/2 channels rotate, as interleaved pairs (2i, 2i+1) with angle i:
//   y_{2i} = fp16(fp16(x_{2i} c_i) - fp16(x_{2i+1} s_i)), y_{2i+1} = fp16(fp16(x_{2i+1} c_i) + fp16(x_{2i} s_i)).
struct Half8 { __half v[8]; };
__device__ __forceinline__ Half8 load8(const __half *x) { return *reinterpret_cast<const Half8 *>(__builtin_assume_aligned(x, 16)); }
__device__ __forceinline__ void store8(__half *x, const Half8 &h) { *reinterpret_cast<uint4 *>(x) = *reinterpret_cast<const uint4 *>(&h); }
template <int H> __device__ __forceinline__ void rope_runs(int rope_mode, int u, int &first, int &second) {   // channels where the two runs of unit u begin
  first = rope_mode == PT_ROPE_LLAMA ? 8 * u : 16 * u;
  second = rope_mode == PT_ROPE_LLAMA ? H / 2 + 8 * u : 16 * u + 8;
}
template <int H> __device__ __forceinline__ void rope16(const AttnParams &p, int u, const __half *sin_r, const __half *cos_r, Half8 &a, Half8 &b) {
  if (p.rope_mode == PT_ROPE_NONE || (p.rope_mode == PT_ROPE_CHATGLM2 && u >= H / 32)) return;
  Half8 s, c;
  if ((((uintptr_t)sin_r | (uintptr_t)cos_r) & 15) == 0) {
    s = load8(sin_r + 8 * u);
    c = load8(cos_r + 8 * u);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) { s.v[i] = sin_r[8 * u + i]; c.v[i] = cos_r[8 * u + i]; }
  }
  if (p.rope_mode == PT_ROPE_LLAMA) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const __half x = a.v[i], y = b.v[i];
      a.v[i] = h_add(h_mul(x, c.v[i]), h_mul(__hneg(y), s.v[i]));
      b.v[i] = h_add(h_mul(y, c.v[i]), h_mul(x, s.v[i]));
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      Half8 &r = i < 4 ? a : b;
      const __half x = r.v[2 * (i & 3)], y = r.v[2 * (i & 3) + 1];
      r.v[2 * (i & 3)] = h_sub(h_mul(x, c.v[i]), h_mul(y, s.v[i]));
      r.v[2 * (i & 3) + 1] = h_add(h_mul(y, c.v[i]), h_mul(x, s.v[i]));
    }
  }
}

constexpr int NQ_MAX = 8;      // q heads of one kv head per block: the n side of an m16n8 tensor-core tile (larger groups take several blocks)
// Weight of a warp's largest score, max-subtracted mode (sums carry it too, and the quotient drops it).  Behind a high score the others of a long history are
// small: as fp16 fractions of 1 they lose bits below 2^-14 and are gone below 2^-25 while the sum still has them, as fractions of 2^15 not before
// 2^-29 (twenty below the largest score), where 100,000 keys together weigh less than a rounding of the output.
constexpr float WEIGHT_ONE = 32768.f;
constexpr int MAX_RUNS = 16;   // blocks of a cluster

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
  uint32_t t;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(t) : "r"(v));
  return t;
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_f2h2(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&h);
}
// Stores a value at an address of this block's shared memory in block `rank` of its cluster; it arrives there at the barrier `bar`.
__device__ __forceinline__ void send(const void *local, int rank, float v, uint32_t bar) {
  uint32_t a, there;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(local)), "r"(rank));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(bar), "r"(rank));
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(a), "r"(__float_as_uint(v)), "r"(there) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { __syncwarp(); asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Shared memory of a block of NW warps: every warp's K and V rows (afterwards its share of the output), the q heads, the new token's key and value
// row, statistics, and, if the launch has clusters, the outputs that their blocks send to the one that writes them.
template <int H, int NW> struct AttnSmem {
  static constexpr int KEYS = 2048 / H;        // keys that a warp takes at a time: 4 KB of K and of V
  static constexpr int LD = H + 8;             // rows padded by 16 bytes: eight rows of an ldmatrix lie in eight different bank groups
  static constexpr int OLD = H + 4;            // a head's outputs, in floats
  __half kv[NW][2][KEYS * LD];
  __half q[NQ_MAX * LD];
  __half fresh[2][H];                          // the new token's (rotated) key and its value
  float2 ml[NW][NQ_MAX];                       // maximum and sum of every warp
  float2 sent_ml[MAX_RUNS][NQ_MAX];            // maximum and sum of every block of the cluster
  uint64_t arrived;                            // what the cluster's blocks send has come
  volatile int abort;
  float sent[1];                               // [run][share]: the outputs this block writes
  static_assert(sizeof(__half) * 2 * KEYS * LD >= sizeof(float) * NQ_MAX * OLD, "a warp's outputs take the place of its keys and values");
};
// Outputs of a unit that one of R blocks writes: whole warps of one head's channels.
__host__ __device__ inline int attn_share(int outputs, int R) { return ((outputs + R - 1) / R + 31) & ~31; }

// One block, or the blocks of a cluster, handle one (sequence, kv head, part of the group's q heads); a warp takes every W-th chunk of its keys, W warps in all.
// Up to a few MB of cache the time is latency: step and page table, then K and V, then the sums.  Above that the HBM rate bounds it.  Hence no barrier of
// the block between the first key and the last, and 8.5 KB in flight per warp, sixteen warps to an SM.  A warp has one buffer for K and
// one for V: while it forms the weights and multiplies them the next K rows are on their way, and the V rows during the next scores.  A chunk costs a
// warp by itself about a microsecond, most of it the way to memory.  Of a short launch's 3.2 us (context 10) half went into branches on rows
// behind the newest token and into a chain step -> table -> rotation; hence copies that fill with zeros, and everything asked for at once.
//   scores [keys x heads] = K [16 keys x H] . q^T, K through ldmatrix, q (B operand) from shared memory into registers once.
//   out^T [H x heads] += V^T [H x 16 keys] . P^T [keys x heads]: V through ldmatrix.trans, the weights of a lane turned by movmatrix.
template <int H, int NW>
__global__ void __launch_bounds__(NW * 32, 16 / NW) kv_append_attn_kernel(const AttnParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  using Smem = AttnSmem<H, NW>;
  Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
  constexpr int KEYS = Smem::KEYS, T = KEYS / 16, LD = Smem::LD, THREADS = NW * 32;
  constexpr int U = H / 8, KS = H / 16;       // 16-byte units of a row; k-steps of the scores = m-tiles of the output
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tig = lane & 3;
  const int PAGE = p.page, R = p.runs, rank = blockIdx.x, W = R * NW;
  const int kvh = blockIdx.y / p.qsplit, qpart = blockIdx.y - kvh * p.qsplit, b = blockIdx.z;
  const int nq = p.qpk / p.qsplit, q_lo = qpart * nq;   // this block's heads of the group: q_lo .. q_lo + nq - 1
  const int share = attn_share(nq * H, R);              // outputs that this block writes if it is one of several
  if (R > 1) {
    if (tid == 0) {
      sm.abort = 0;
      mbar_init(smem_u32(&sm.arrived), 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      const int mine = max(0, min(nq * H - rank * share, share));
      mbar_expect_tx(smem_u32(&sm.arrived), R * (mine * sizeof(float) + nq * sizeof(float2)));
    }
    cluster_arrive();     // once all have come by here, a block may send
  }
  early_start();   // (the next kernel may fetch its weights meanwhile; everything this one reads was produced upstream)
  const int step = *p.step;
  // The q heads, the new token's key and its value, sixteen channels a thread, asked for together with the step.
  constexpr int UNITS = H / 16, MOST = ((NQ_MAX + 2) * UNITS + THREADS - 1) / THREADS;
  const __half *qrow = p.qkv + (size_t)b * (p.n_head + 2 * p.n_kv) * H;
  Half8 raw[MOST][2];
#pragma unroll
  for (int m = 0; m < MOST; ++m) {
    const int i = m * THREADS + tid, h = i / UNITS, u = i % UNITS;
    if (h >= nq + 2) continue;
    const int head = h < nq ? kvh * p.qpk + q_lo + h : p.n_head + (h - nq) * p.n_kv + kvh;
    int c0, c1;
    rope_runs<H>(h > nq ? PT_ROPE_NONE : p.rope_mode, u, c0, c1);
    raw[m][0] = load8(qrow + (size_t)head * H + c0);
    raw[m][1] = load8(qrow + (size_t)head * H + c1);
  }
  // Where this lane's eight rows of chunk c begin (lane mod KEYS / 8; they lie in one page, whose size is a multiple of eight), in the pool's K.
  const int *table = p.page_table + (size_t)b * p.max_pages;
  auto rows_of = [&](int c) {
    const int key = c * KEYS + 8 * (lane & (KEYS / 8 - 1)), pg = min(key / PAGE, p.max_pages - 1);
    return (((long long)table[pg] * 2 * p.n_kv + kvh) * PAGE + (key - pg * PAGE)) * H;
  };
  const int c_first = warp * R + rank;
  long long rows = rows_of(c_first);                    // (asked for together with the step)
  if (step < 0 || step >= p.max_len) {  // no page / no RoPE row for this position: report it
    if (tid == 0 && p.error_flag) atomicExch(p.error_flag, 12);
    if (R > 1) cluster_wait();
    return;
  }
  const int n_chunks = step / KEYS + 1, c_last = n_chunks - 1;

  __half *sK = sm.kv[warp][0], *sV = sm.kv[warp][1];
  // The rows of chunk c of K (which = 0) or V.  The newest token's and what lies behind it are zeros; the newest one's is written later.
  const long long v_rows = (long long)p.n_kv * PAGE * H;
  const int lane_row = lane / U, lane_unit = lane % U;       // (a step of the warp takes 32 / U rows)
  auto load = [&](int which, int c) {
    const uint32_t dst = smem_u32(which ? sV : sK) + (lane_row * LD + lane_unit * 8) * 2;
    const __half *src = p.pool + (which ? v_rows : 0) + lane_row * H + lane_unit * 8;
    const int left = step - c * KEYS - lane_row;
#pragma unroll
    for (int e = 0; e < KEYS / 8; ++e) {
      const __half *from = src + __shfl_sync(0xffffffffu, rows, e);
#pragma unroll
      for (int i = 0; i < U / 4; ++i) {
        const int r = i * (32 / U);      // (a row that is not read is filled with zeros; its address is not used)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (8 * e + r) * LD * 2), "l"(8 * e + r < left ? from + r * H : p.pool), "r"(8 * e + r < left ? 16 : 0) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (c_first < n_chunks) {   // the first rows go out before anything else
    load(0, c_first);
    load(1, c_first);
  }

  // ---- RoPE on the block's q heads and on the new key
  const __half *sin_r = p.sin_t + (size_t)step * p.rot_half, *cos_r = p.cos_t + (size_t)step * p.rot_half;
  for (int i = tid; i < (NQ_MAX - nq) * U; i += THREADS)   // unused head rows of the B operand: zeros
    *reinterpret_cast<uint4 *>(sm.q + (nq + i / U) * LD + i % U * 8) = make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int m = 0; m < MOST; ++m) {
    const int i = m * THREADS + tid, h = i / UNITS, u = i % UNITS;
    if (h >= nq + 2) continue;
    int c0, c1;
    rope_runs<H>(h > nq ? PT_ROPE_NONE : p.rope_mode, u, c0, c1);
    if (h <= nq) rope16<H>(p, u, sin_r, cos_r, raw[m][0], raw[m][1]);
    __half *to = h < nq ? sm.q + h * LD : sm.fresh[h - nq];
    store8(to + c0, raw[m][0]);
    store8(to + c1, raw[m][1]);
  }
  __syncthreads();
  uint32_t qf[KS][2];          // q as B operand: lane (g, tig) holds channels 2 tig, + 1, + 8, + 9 of every 16 of head g
#pragma unroll
  for (int k = 0; k < KS; ++k) {
    qf[k][0] = *reinterpret_cast<const uint32_t *>(sm.q + g * LD + k * 16 + 2 * tig);
    qf[k][1] = *reinterpret_cast<const uint32_t *>(sm.q + g * LD + k * 16 + 8 + 2 * tig);
  }

  float O[KS][4], M[2] = {-INFINITY, -INFINITY}, L[2] = {0.f, 0.f};   // lane (g, tig): channels 16 j + g and + 8 of heads 2 tig and 2 tig + 1
#pragma unroll
  for (int j = 0; j < KS; ++j) O[j][0] = O[j][1] = O[j][2] = O[j][3] = 0.f;
  const bool f32 = p.softmax_mode == PT_SOFTMAX_F32;
  if (!f32) M[0] = M[1] = 0.f;         // the reference exponentiates fp16 scores without subtracting the maximum
  const uint32_t k_lane = smem_u32(sK + (lane & 15) * LD + (lane >> 4) * 8);                            // matrices: keys 0-7 / 8-15, then channels + 8
  const uint32_t v_lane = smem_u32(sV + ((lane >> 4) * 8 + (lane & 7)) * LD + ((lane >> 3) & 1) * 8);   // ... channels 0-7 / 8-15, then keys + 8
  for (int c = c_first; c < n_chunks; c += W) {
    const bool more = c + W < n_chunks;
    const bool newest = c == c_last;               // this chunk ends with the new token
    const int slot = step - c * KEYS;
    if (newest && qpart == 0) {                    // one block of the group appends to the pool
      __half *at = p.pool + __shfl_sync(0xffffffffu, rows, slot >> 3) + (slot & 7) * H;
      for (int j = lane; j < 2 * U; j += 32) store8(at + (j < U ? 0 : v_rows) + j % U * 8, load8(sm.fresh[j / U] + j % U * 8));
    }
    if (more) rows = rows_of(c + W);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    if (newest && lane_row == slot % (32 / U)) store8(sK + slot * LD + lane_unit * 8, load8(sm.fresh[0] + lane_unit * 8));     // (the lanes that copied zeros there: they have waited for them)
    __syncwarp();              // K is there
    float sc[T][2][4] = {};    // (two chains each)
#pragma unroll
    for (int k = 0; k < KS; ++k)
#pragma unroll
      for (int t = 0; t < T; ++t) {
        uint32_t a[4];
        ldmatrix_x4(k_lane + (t * 16 * LD + k * 16) * 2, a);
        mma_f16(sc[t][k & 1], a, qf[k][0], qf[k][1]);
      }
    __syncwarp();              // K has been used
    if (more) load(0, c + W);
    else asm volatile("cp.async.commit_group;" ::: "memory");      // (the groups are counted)
    // lane (g, tig): keys 16 t + g (e = 0, 1) and + 8 (2, 3) against heads 2 tig and 2 tig + 1
    float w[T][4];
    bool in[T][2];
#pragma unroll
    for (int t = 0; t < T; ++t) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        __half s16 = __float2half_rn(sc[t][0][e] + sc[t][1][e]);   // fp16 matmul output
        if (p.use_scale) s16 = h_mul(s16, p.scale_h);              // ops.mul by fp16(1/sqrt(H))
        w[t][e] = __half2float(s16);
      }
      in[t][0] = c * KEYS + 16 * t + g <= step;
      in[t][1] = c * KEYS + 16 * t + 8 + g <= step;
    }
    if (f32) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float m = -INFINITY;
#pragma unroll
        for (int t = 0; t < T; ++t) m = fmaxf(m, fmaxf(in[t][0] ? w[t][h] : -INFINITY, in[t][1] ? w[t][h + 2] : -INFINITY));
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        const float top = fmaxf(M[h], m), was = M[h] == top ? 1.f : expf(M[h] - top), ref = top == -INFINITY ? 0.f : top;
        M[h] = top;
        L[h] *= was;
        if (__any_sync(0xffffffffu, was != 1.f)) {
#pragma unroll
          for (int j = 0; j < KS; ++j) { O[j][h] *= was; O[j][h + 2] *= was; }
        }
#pragma unroll
        for (int t = 0; t < T; ++t) {
          w[t][h] = in[t][0] ? WEIGHT_ONE * expf(w[t][h] - ref) : 0.f;
          w[t][h + 2] = in[t][1] ? WEIGHT_ONE * expf(w[t][h + 2] - ref) : 0.f;
        }
      }
    } else {
#pragma unroll
      for (int t = 0; t < T; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) w[t][e] = in[t][e >> 1] ? __half2float(__float2half_rn(expf(w[t][e]))) : 0.f;
    }
    uint32_t pf[T][2];
#pragma unroll
    for (int t = 0; t < T; ++t) {
      L[0] += w[t][0] + w[t][2];
      L[1] += w[t][1] + w[t][3];
      // The weights are rounded to fp16 for the tensor core; they are at most 2^15 (max-subtracted mode, see WEIGHT_ONE) or fp16 values already
      // (the reference's fp16 softmax mode), so this costs at most 2^-11 relative per weight.
      pf[t][0] = transpose8x8(pack_f2h2(w[t][0], w[t][1]));
      pf[t][1] = transpose8x8(pack_f2h2(w[t][2], w[t][3]));
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    if (newest && lane_row == slot % (32 / U)) store8(sV + slot * LD + lane_unit * 8, load8(sm.fresh[1] + lane_unit * 8));
    __syncwarp();              // V is there
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
      for (int j = 0; j < KS; ++j) {
        uint32_t a[4];
        ldmatrix_x4_trans(v_lane + (t * 16 * LD + j * 16) * 2, a);
        mma_f16(O[j], a, pf[t][0], pf[t][1]);
      }
    __syncwarp();              // V has been used
    if (more) load(1, c + W);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }

  // ---- the warps of the block that have keys
  const int n_warps = min(NW, (n_chunks - rank + R - 1) / R);      // (none: a block of a cluster that has no keys)
  float *own = reinterpret_cast<float *>(sm.kv[warp]);             // [head][channel]
  float2 *left = p.ws_ml + ((size_t)b * p.n_head + (size_t)kvh * p.qpk + q_lo) * p.max_pages + c_first;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) L[h] += __shfl_xor_sync(0xffffffffu, L[h], o);
    const int qh = 2 * tig + h;
    if (g == 0) sm.ml[warp][qh] = make_float2(M[h], L[h]);
    if (qh >= nq || warp >= n_warps) continue;
    if (g == 0 && c_first < p.max_pages) left[(size_t)qh * p.max_pages] = make_float2(M[h], L[h]);     // (how the keys were shared out can be read there)
#pragma unroll
    for (int j = 0; j < KS; ++j) {
      own[qh * Smem::OLD + 16 * j + g] = O[j][h];
      own[qh * Smem::OLD + 16 * j + g + 8] = O[j][h + 2];
    }
  }
  __syncthreads();
  // n parts of a head, lane i holding the maximum and sum of part i: the parts' weights and the sum.
  auto weigh = [&](float2 ml, float &m, float &l) {
    m = warp_max(ml.x);
    const float f = ml.x == m ? 1.f : expf(ml.x - m);
    l = warp_sum(ml.y * f);
    return f;
  };
  auto write = [&](int qh, int ch, float o) {
    const __half y = __float2half_rn(o);
    const size_t col = ((size_t)kvh * p.qpk + q_lo + qh) * H + ch;
    p.out[(size_t)b * p.out_ld + col] = y;
    if (p.out8) p.out8[(size_t)b * p.n_head * H + col] = (uint8_t)__nv_cvt_float_to_fp8(__half2float(y) * p.inv_out_scale, __NV_SATFINITE, __NV_E4M3);
  };
  const uint32_t arrived = smem_u32(&sm.arrived);
  if (R > 1) cluster_wait();
  for (int e0 = warp * 32; e0 < nq * H; e0 += THREADS) {           // 32 channels of one head
    const int qh = e0 / H, ch = e0 % H + lane;
    float m, l, o = 0.f;
    const float f = weigh(lane < n_warps ? sm.ml[lane][qh] : make_float2(-INFINITY, 0.f), m, l);
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      const float v = i < n_warps ? reinterpret_cast<const float *>(sm.kv[i])[qh * Smem::OLD + ch] : 0.f;
      o += v * __shfl_sync(0xffffffffu, f, i);
    }
    if (R == 1) {
      write(qh, ch, o / l);
    } else {   // the blocks of the cluster: block r gets outputs [r share, (r + 1) share) of the nq heads from all, and everybody's statistics
      const int to = e0 / share;
      send(&sm.sent[rank * share + e0 + lane - to * share], to, o, arrived);
      if (e0 % H == 0 && lane < R) {
        send(&sm.sent_ml[rank][qh].x, lane, m, arrived);
        send(&sm.sent_ml[rank][qh].y, lane, l, arrived);
      }
    }
  }
  if (R == 1) return;
  if (!__all_sync(0xffffffffu, mbar_wait(arrived, 0, &sm.abort))) {
    if (p.error_flag) atomicCAS(p.error_flag, 0, 13);
    sm.abort = 1;
    stay_for_cluster();     // what was late may still come
    return;
  }
  for (int e0 = warp * 32; e0 < share && rank * share + e0 < nq * H; e0 += THREADS) {
    const int e = rank * share + e0 + lane, qh = e / H;
    float m, l, o = 0.f;
    const float f = weigh(lane < R ? sm.sent_ml[lane][qh] : make_float2(-INFINITY, 0.f), m, l);
    for (int i = 0; i < R; ++i) o += sm.sent[i * share + e0 + lane] * __shfl_sync(0xffffffffu, f, i);
    write(qh, e % H, o / l);
  }
}

// dense[kv][b][h][l][:] = l <= step ? token (step - l) of the paged cache : 0
__global__ void kv_export_kernel(const __half *pool, const int *page_table, const int *step_dev, int B, int n_kv, int H, int page,
                                 int max_pages, int max_len, __half *dense) {
  const int step = *step_dev;
  const size_t total = (size_t)2 * B * n_kv * max_len * (H / 8);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    size_t r = i;
    const int u = r % (H / 8); r /= (H / 8);
    const int l = r % max_len; r /= max_len;
    const int h = r % n_kv; r /= n_kv;
    const int b = r % B; r /= B;
    const int kv = (int)r;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (l <= step) {
      const int t = step - l;
      const int phys = page_table[(size_t)b * max_pages + t / page];
      v = *reinterpret_cast<const uint4 *>(pool + ((((size_t)phys * 2 + kv) * n_kv + h) * page + t % page) * H + u * 8);
    }
    reinterpret_cast<uint4 *>(dense)[i] = v;
  }
}

// Copies the page being filled (slots 0 .. step % page) of row parent[r] into row r's spare page.
__global__ void kv_reorder_pages_kernel(__half *pool, const int *page_table, const int *spare, const int *parent, const int *step_dev,
                                        int n_kv, int H, int page, int max_pages) {
  const int r = blockIdx.x, step = *step_dev;
  const int pg = step / page, n_slots = step % page + 1;
  const int src = page_table[(size_t)parent[r] * max_pages + pg], dst = spare[r];
  const size_t page_elems = (size_t)2 * n_kv * page * H;
  const uint4 *s4 = reinterpret_cast<const uint4 *>(pool + (size_t)src * page_elems);
  uint4 *d4 = reinterpret_cast<uint4 *>(pool + (size_t)dst * page_elems);
  const int row_u = H / 8;                       // 16-byte units per token
  const int total = 2 * n_kv * n_slots * row_u;  // only the filled slots of each (k|v, head) tile
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < total; i += gridDim.y * blockDim.x) {
    const int u = i % row_u, t = (i / row_u) % n_slots, hk = i / (row_u * n_slots);
    const size_t off = ((size_t)hk * page + t) * row_u + u;
    d4[off] = s4[off];
  }
}
// new_table[r][p < pg] = old[parent[r]][p]; new_table[r][pg] = spare[r]; spare[r] = old[r][pg]; later pages stay.
__global__ void kv_reorder_table_kernel(int *table, const int *old, int *spare, const int *parent, const int *step_dev, int rows,
                                        int page, int max_pages) {
  const int pg = *step_dev / page;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows * max_pages; i += gridDim.x * blockDim.x) {
    const int r = i / max_pages, p = i - r * max_pages;
    if (p < pg) table[i] = old[(size_t)parent[r] * max_pages + p];
    else if (p == pg) {
      table[i] = spare[r];
      spare[r] = old[i];
    }
  }
}

}  // namespace pt

using namespace pt;

static size_t align256(size_t v) { return (v + 255) / 256 * 256; }

extern "C" size_t pt_attn_workspace_bytes(int batch, int n_head, int head_dim, int max_pages) {
  const size_t heads = (size_t)batch * n_head;
  (void)head_dim;
  return align256(heads * sizeof(int)) + align256(heads * max_pages * sizeof(float2));
}

// Warps per block and blocks per cluster that share the keys of one of `units` (sequence, kv head, part).  Sixteen warps fit an SM whatever the block, so
// blocks get as many as keep all units on the SMs at once.  A cluster's meeting costs 0.5 to 1 us: it is worth it where a unit's table has 20
// chunks for each block (of 16 warps), and as long as every block has an SM (clusters of sixteen: of a GPC).  The table's room decides, since the step is not
// known here: at context 10 in room for 2048 a cluster takes 4.2 us where one block took 3.9 (12 heads of 64), at 100 and more it is ahead (4.3 and 6.5).  Leaving
// histories of one page to the first block mends the former and costs every other launch of a cluster 0.12 us: not done.  Measured on B200, us a launch in a row of
// launches, of (rows, q heads, kv heads, head width, context, room) the kernel before / as warps x blocks:
//   (1, 12, 12, 64, 159, 352)     6.4 / 8x1 3.6, 16x1 3.8, 4x1 4.6, 16x2 4.2         (16, 25, 25, 64, 255, 448)    11.8 / 4x1 8.1, 8x1 9.3, 4x2 11.2
//   (1, 32, 32, 128, 511, 704)    8.0 / 16x4 5.2, 16x2 6.1, 16x1 7.8, 8x4 5.8        (4, 32, 32, 128, 511, 704)    12.7 / 16x1 8.3, 8x2 9.2, 16x2 13.3
//   (9, 32, 32, 128, 511, 704)   20.2 / 8x1 15.3, 4x1 16.0, 16x1 17.4                (16, 32, 32, 128, 511, 704)   29.6 / 4x1 25.8 (bytes alone 20.5)
//   (8, 32, 2, 128, 1151, 1344)  16.6 / 16x4 8.4, 16x2 11.2, 16x8 18.9               (1, 32, 2, 128, 1151, 1344)   14.0 / 16x8 6.2, 16x4 8.1
//   (1, 32, 2, 128, 30000, 32768) 54 / 16x16 21, 16x8 34                             (1, 8, 8, 128, 30000, 32768)  34.6 / 16x8 33.4, 16x16 47
struct AttnSplit { int warps, runs; };
static AttnSplit split_keys(int units, int max_pages, int page, int head_dim) {
  const int chunks = (int)std::min<long long>((long long)max_pages * page * head_dim / 2048 + 1, 1 << 20);
  const int sms = sm_count(), warps = units > 2 * sms ? 4 : units > sms || chunks < 16 ? 8 : 16;
  int runs = 1;
  while (warps == 16 && runs < (units <= 4 ? 16 : 8) && 2 * units * runs <= sms && chunks >= 20 * runs) runs *= 2;
  return {warps, runs};
}
template <int H, int NW> static cudaError_t launch_attn(const AttnParams &p, cudaStream_t stream) {
  static std::atomic<uint64_t> allowed{0}, wide{0};
  const auto kernel = kv_append_attn_kernel<H, NW>;
  const int nq = p.qpk / p.qsplit;
  const size_t smem = sizeof(AttnSmem<H, NW>) + (p.runs > 1 ? (size_t)p.runs * attn_share(nq * H, p.runs) * sizeof(float) : 0);
  cudaError_t e = allow_smem(kernel, 200 * 1024, allowed);
  if (e == cudaSuccess) e = allow_wide_clusters(kernel, wide);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.runs, p.n_kv * p.qsplit, p.B);
  cfg.blockDim = dim3(NW * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  if (p.runs > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = p.runs;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  if (p.pdl) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  return cudaLaunchKernelEx(&cfg, kernel, p);
}
template <int H> static cudaError_t launch_attn(const AttnParams &p, int warps, cudaStream_t stream) {
  return warps == 16 ? launch_attn<H, 16>(p, stream) : warps == 8 ? launch_attn<H, 8>(p, stream) : launch_attn<H, 4>(p, stream);
}

extern "C" int pt_kv_append_attn(const pt_attn_args *a, void *stream) {
  PT_REQUIRE(a, "pt_kv_append_attn: null args");
  PT_REQUIRE(a->batch > 0 && a->n_head > 0 && a->n_kv > 0 && a->n_head % a->n_kv == 0,
             "pt_kv_append_attn: n_head=%d must be a positive multiple of n_kv=%d", a->n_head, a->n_kv);
  PT_REQUIRE(a->head_dim == 64 || a->head_dim == 128, "pt_kv_append_attn: head_dim=%d (supported: 64, 128)", a->head_dim);
  PT_REQUIRE(a->page_size >= 8 && a->page_size <= 128 && a->page_size % 8 == 0, "pt_kv_append_attn: page_size=%d must be a multiple of 8 in 8..128",
             a->page_size);
  PT_REQUIRE(a->max_pages > 0, "pt_kv_append_attn: max_pages=%d", a->max_pages);
  PT_REQUIRE(a->rope_mode >= PT_ROPE_NONE && a->rope_mode <= PT_ROPE_CHATGLM2, "pt_kv_append_attn: bad rope_mode %d", a->rope_mode);
  PT_REQUIRE(a->softmax_mode == PT_SOFTMAX_F32 || a->softmax_mode == PT_SOFTMAX_F16, "pt_kv_append_attn: bad softmax_mode %d", a->softmax_mode);
  PT_REQUIRE(a->step_dev && a->qkv && a->pool && a->page_table && a->out && a->workspace, "pt_kv_append_attn: null pointer argument");
  PT_REQUIRE(a->rope_mode == PT_ROPE_NONE || (a->rope_sin && a->rope_cos), "pt_kv_append_attn: RoPE needs sin/cos tables");
  const size_t need = pt_attn_workspace_bytes(a->batch, a->n_head, a->head_dim, a->max_pages);
  PT_REQUIRE(a->workspace_bytes >= need, "pt_kv_append_attn: workspace needs %zu bytes, got %zu", need, a->workspace_bytes);

  AttnParams p{};
  p.B = a->batch; p.n_head = a->n_head; p.n_kv = a->n_kv; p.qpk = a->n_head / a->n_kv; p.H = a->head_dim;
  {  // at most NQ_MAX q heads per block (the n side of the tensor-core tile): larger groups are shared out over several blocks
    int nq_blk = p.qpk;
    if (p.qpk > NQ_MAX)
      for (nq_blk = NQ_MAX; p.qpk % nq_blk; --nq_blk) {}
    p.qsplit = p.qpk / nq_blk;
  }
  p.page = a->page_size; p.max_pages = a->max_pages; p.rope_mode = a->rope_mode; p.softmax_mode = a->softmax_mode;
  p.rot_half = a->rope_mode == PT_ROPE_CHATGLM2 ? a->head_dim / 4 : a->head_dim / 2;
  p.out_ld = a->out_ld > 0 ? a->out_ld : a->n_head * a->head_dim;
  p.use_scale = a->score_scale != 1.0f;
  p.scale_h = __float2half_rn(a->score_scale);
  p.step = a->step_dev;
  p.qkv = (const __half *)a->qkv; p.sin_t = (const __half *)a->rope_sin; p.cos_t = (const __half *)a->rope_cos;
  p.pool = (__half *)a->pool; p.page_table = a->page_table; p.out = (__half *)a->out;
  p.out8 = (uint8_t *)a->out_fp8;
  PT_REQUIRE(!a->out_fp8 || a->out_fp8_scale > 0.f, "pt_kv_append_attn: out_fp8 needs out_fp8_scale > 0");
  p.inv_out_scale = a->out_fp8 ? 1.0f / a->out_fp8_scale : 0.f;
  const size_t heads = (size_t)a->batch * a->n_head;
  char *ws = (char *)a->workspace;
  p.ws_ml = (float2 *)(ws + align256(heads * sizeof(int)));
  p.error_flag = a->error_flag;
  p.pdl = a->pdl ? 1 : 0;
  PT_REQUIRE(a->max_len >= 0 && a->max_len <= a->page_size * a->max_pages, "pt_kv_append_attn: max_len=%d exceeds the %d positions of the page table",
             a->max_len, a->page_size * a->max_pages);
  p.max_len = a->max_len > 0 ? a->max_len : a->page_size * a->max_pages;

  const AttnSplit split = split_keys(a->batch * a->n_kv * p.qsplit, a->max_pages, a->page_size, a->head_dim);
  p.runs = split.runs;
  const cudaError_t le = p.H == 128 ? launch_attn<128>(p, split.warps, as_stream(stream)) : launch_attn<64>(p, split.warps, as_stream(stream));
  if (le != cudaSuccess) return pt::set_error(PT_ERR_CUDA, "pt_kv_append_attn: %s", cudaGetErrorString(le));
  PT_LAUNCH_CHECK("pt_kv_append_attn");
  return PT_OK;
}

extern "C" int pt_kv_export(const void *pool, const int32_t *page_table, const int32_t *step_dev, int batch, int n_kv, int head_dim,
                            int page_size, int max_pages, int max_len, void *dense_out, void *stream) {
  PT_REQUIRE(pool && page_table && step_dev && dense_out, "pt_kv_export: null pointer argument");
  PT_REQUIRE(head_dim % 8 == 0 && max_len <= page_size * max_pages, "pt_kv_export: max_len=%d exceeds page capacity %d", max_len,
             page_size * max_pages);
  kv_export_kernel<<<sm_count() * 4, 256, 0, as_stream(stream)>>>((const __half *)pool, page_table, step_dev, batch, n_kv, head_dim, page_size,
                                                          max_pages, max_len, (__half *)dense_out);
  PT_LAUNCH_CHECK("pt_kv_export");
  return PT_OK;
}

extern "C" int pt_kv_reorder_pages(void *pool, const int32_t *page_table, const int32_t *spare_pages, const int32_t *parent,
                                   const int32_t *step_dev, int rows, int n_kv, int head_dim, int page_size, int max_pages, void *stream) {
  PT_REQUIRE(pool && page_table && spare_pages && parent && step_dev, "pt_kv_reorder_pages: null pointer argument");
  PT_REQUIRE(rows > 0 && n_kv > 0 && head_dim % 8 == 0 && page_size > 0 && max_pages > 0, "pt_kv_reorder_pages: bad shape");
  dim3 grid(rows, 8);
  kv_reorder_pages_kernel<<<grid, 256, 0, as_stream(stream)>>>((__half *)pool, page_table, spare_pages, parent, step_dev, n_kv, head_dim,
                                                              page_size, max_pages);
  PT_LAUNCH_CHECK("pt_kv_reorder_pages");
  return PT_OK;
}

extern "C" int pt_kv_reorder_table(int32_t *page_table, int32_t *table_tmp, int32_t *spare_pages, const int32_t *parent,
                                   const int32_t *step_dev, int rows, int page_size, int max_pages, void *stream) {
  PT_REQUIRE(page_table && table_tmp && spare_pages && parent && step_dev, "pt_kv_reorder_table: null pointer argument");
  PT_REQUIRE(rows > 0 && page_size > 0 && max_pages > 0, "pt_kv_reorder_table: bad shape");
  cudaStream_t st = as_stream(stream);
  PT_CUDA(cudaMemcpyAsync(table_tmp, page_table, (size_t)rows * max_pages * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
  kv_reorder_table_kernel<<<ceil_div(rows * max_pages, 256), 256, 0, st>>>(page_table, table_tmp, spare_pages, parent, step_dev, rows,
                                                                          page_size, max_pages);
  PT_LAUNCH_CHECK("pt_kv_reorder_table");
  return PT_OK;
}
