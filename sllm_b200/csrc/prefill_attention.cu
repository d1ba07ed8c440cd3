// Causal prompt attention on the 5th-generation tensor cores (tcgen05 + TMEM + TMA), heads of 64, 128 or 256 channels.
//
// Fresh sequences: their tokens are contiguous rows of the packed qkv activation [T, (hq + 2 hkv) * hd] (bf16, q and k already
// rotated) and start at position 0, so K and V are read from that tensor with TMA instead of from the paged cache.  Optional sliding
// window (key tiles outside it are not visited) and attention sinks.
//
// What bounds it: exponentials (16 a clock and SM) take 1024 cycles for 128 queries x 128 keys, products 512 (S) and 1024 (P V, twice)
// with 128 channels, so neither may wait for the other.  A CTA carries two items, 128-row query tiles that share their keys and values: two
// heads of a group (or, with one query head per kv head, two neighbouring tiles of one head).  While one item's softmax runs, the
// tensor cores work on the other.  Heads of 256 channels fill the tensor memory with one item; its next scores are computed ahead.
//
//   warp 0      TMA producer: Q once, then K and V tiles through rings of two stages
//   warp 1      TMEM owner; issues S = Q K^T and O += P V of all items
//   warps 4 ..  softmax, four warps per item, thread = query row: the row's scores are read once into registers, P goes back to
//               tensor memory in place of S as the A operand of the second product, O stays in tensor memory
// P enters its product as two bf16 values, hi = bf16(p) and lo = bf16(p - hi), 16 significant bits that are multiplied one after the other;
// the row's sum takes p itself.  Results are as far from 64 bits as their rounding to bf16 takes them (2-norm 0.00166), as with the fp32
// probabilities of attention.cu; one bf16 value gives 0.0021 (4000 tokens, heads of 128: 0.00204 with the maximum of every tile).
// With E4M3 results (kStrict) a row keeps O in registers, o <- o alpha + P V of the tile with the maximum of every tile, and reads its
// scores twice: the next product quantises, where a last bit's difference becomes a sixteenth of a value, and this order is the one
// that FP8 models have been run and compared with.
// Otherwise O is rescaled only when a row's maximum has grown by more than 2^8 since the last time: exponents relative to an older maximum are
// as exact, and sums hold 2^8 times larger values with ease.
//
// Measured (B200, us; before: one item per CTA whose scores, softmax and products followed one another, or the pages' rows one by one):
//   8192 tokens, 32 + 2 x 8 heads x 128              2324 ->  671 (0.82 PFLOP/s), E4M3 results 1260
//   2048 + 1098 + 1623 + 674 tokens, the same heads   431 ->  147,                E4M3 results  241
//   2048 + 782 tokens, 16 + 2 x 4 heads x 256        3285 ->   90
//   1000 + 536 + 823 tokens, 64 + 2 x 8 heads x 64    880 ->   87, with a window of 128 69
// (P as one bf16 value: 532, 127, 79, 78 and 66 in the same run)
// Replaces the reference's scalar prefill kernels (causal_attention_kernel.hip.cpp:388-495).
#include "pair_mma.cuh"
#include "api.h"
#include "tmap.h"

namespace sllm {

constexpr int kPfTile = 128;            // query rows of an item

template <int HD>
struct PfShape {
  static constexpr int kItems = HD == 256 ? 1 : 2;
  static constexpr int kKeys = HD == 256 ? 64 : 128;       // keys of a tile
  static constexpr int kChunks = HD / 64;
  static constexpr int kQBytes = kChunks * kPfTile * 128;  // of an item; chunks of [rows x 64 channels], 128-byte swizzle
  static constexpr int kKvBytes = kChunks * kKeys * 128;   // of a K or V tile
  static constexpr int kThreads = 128 + 128 * kItems;
  // tensor memory: two score tiles (of the items, or of the even and odd tiles of one item), then O of the items.  P takes the place of
  // its scores: of 32 keys the upper halves of the values in 16 columns and the lower ones in the next 16.  The next product into
  // these columns is issued after the one that reads P.
  static constexpr uint32_t kTmemO = 2 * kKeys;
  static constexpr size_t kSmem = kItems * kQBytes + 4 * kKvBytes + 256 + 1024;
};

struct PrefillParams {
  const int* tiles;        // [num_tiles][4]: first token row of the sequence, sequence length, q0, unused
  int hq, hkv, window;
  int pair_heads;          // 1: the items are two heads on one tile; 0: two tiles of one head
  float scale_log2;        // softmax scale * log2(e)
  const float* sinks;      // optional [hq]: scores that join the denominator only
  __nv_bfloat16* out_bf16; // [T, hq * HD] or null
  uint8_t* out_fp8;        // E4M3 [T, hq * 128] or null
  float* out_scale;        // [hq, ld_scale]
  int ld_scale;
  int* status;
};

struct __align__(8) PrefillBarriers {
  uint64_t q_full;
  uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2];
  uint64_t s_full[2], p_ready[2], o_full[2];
  uint32_t tmem_base;
  int abort_flag;
};

// MN-major operand (rows = K index, 128-byte rows of 64 contiguous MN elements, MN blocks of 64 elements `mn_block_stride` bytes
// apart), 128-byte swizzle: LBO = MN-block stride, SBO = 1024.
__device__ __forceinline__ uint64_t make_smem_desc_sw128_mn(uint32_t smem_addr, uint32_t mn_block_stride) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>((mn_block_stride >> 4) & 0x3FFF) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}
// D[tmem] (+)= A[tmem] * B[smem]: A holds two 16-bit elements of a row per column.
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,"
      "%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 2^x; kNormal: a subnormal result becomes zero.
template <bool kNormal>
__device__ __forceinline__ float pf_ex2(float x) {
  float y;
  if constexpr (kNormal) asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  else asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// P of 32 keys from their scores: 2^(s scale - m), as a sum of two 16-bit values (16 significant bits), and the sums of P.
template <bool kNormal>
__device__ __forceinline__ void pf_probabilities(const uint32_t (&s)[32], float scale, float m, uint32_t (&hi)[16], uint32_t (&lo)[16],
                                                 float (&sum)[4]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float p0 = pf_ex2<kNormal>(fmaf(__uint_as_float(s[2 * i]), scale, -m));
    const float p1 = pf_ex2<kNormal>(fmaf(__uint_as_float(s[2 * i + 1]), scale, -m));
    __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
    hi[i] = *reinterpret_cast<const uint32_t*>(&h);
    h = __floats2bfloat162_rn(p0 - __uint_as_float(hi[i] << 16), p1 - __uint_as_float(hi[i] & 0xffff0000u));
    lo[i] = *reinterpret_cast<const uint32_t*>(&h);
    sum[2 * (i & 1)] += p0;
    sum[2 * (i & 1) + 1] += p1;
  }
}

// The rows of kStrict: heads of 128 channels without window and sinks, O in registers.  Scores are read for the maximum and again for the exponentials; P(32 keys)
// overwrites score columns that have been read.
__device__ __forceinline__ void strict_rows(const PrefillParams& p, PrefillBarriers* bars, uint32_t lane_addr, uint32_t o_addr, int item, int head,
                                            int qt, int qpos, int nt, int tok0, int seq_len, volatile int* abort_flag) {
  constexpr int HD = 128, kKeys = 128;
  const uint32_t s_addr = lane_addr + item * kKeys;
  float o[HD];
#pragma unroll
  for (int i = 0; i < HD; ++i) o[i] = 0.f;
  float m = -INFINITY, l = 0.f;
  bool ok = true;
  for (int j = 0; j < nt; ++j) {
    ok = __all_sync(0xffffffffu, mbar_wait(&bars->s_full[item], j & 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_TMEM_FULL));
    if (!ok) break;
    tc_fence_after();
    const int k0 = j * kKeys, hi = k0 + kKeys - 1 > qt ? qpos - k0 : kKeys;     // keys up to hi are visible
    float tmax = -INFINITY;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t v[32];
      tmem_ld32(s_addr + c * 32, v);
      tmem_wait_regs(v);
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float x = __uint_as_float(v[i]);
        tmax = fmaxf(tmax, c * 32 + i > hi ? -INFINITY : x);
      }
    }
    const float m_new = fmaxf(m, tmax * p.scale_log2);
    const float alpha = (m == -INFINITY) ? 0.f : exp2f(m - m_new);
    const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
    float psum = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t v[32], w[16];
      tmem_ld32(s_addr + c * 32, v);
      tmem_wait_regs(v);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int k = c * 32 + 2 * i;
        float p0 = exp2f(__uint_as_float(v[2 * i]) * p.scale_log2 - m_use), p1 = exp2f(__uint_as_float(v[2 * i + 1]) * p.scale_log2 - m_use);
        if (k > hi) p0 = 0.f;
        if (k + 1 > hi) p1 = 0.f;
        const __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
        psum += __bfloat162float(h.x) + __bfloat162float(h.y);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
      }
      tmem_st16(s_addr + c * 16, w);
    }
    l = l * alpha + psum;
    m = m_new;
    tmem_wait_st();
    tc_fence_before();
    mbar_arrive(&bars->p_ready[item]);
    ok = __all_sync(0xffffffffu, mbar_wait(&bars->o_full[item], j & 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_TMEM_FULL));
    if (!ok) break;
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t v[32];
      tmem_ld32(o_addr + c * 32, v);
      tmem_wait_regs(v);
#pragma unroll
      for (int i = 0; i < 32; ++i) o[c * 32 + i] = fmaf(o[c * 32 + i], alpha, __uint_as_float(v[i]));
    }
    tc_fence_before();
  }
  if (ok && qpos < seq_len) {
    const float inv = l > 0.f ? 1.f / l : 0.f;
    const size_t row = static_cast<size_t>(tok0 + qpos), base = (row * p.hq + head) * HD;
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < HD; ++i) {
      o[i] = __bfloat162float(__float2bfloat16_rn(o[i] * inv));
      const float a = fabsf(o[i]);
      if (a == a && a <= 3.0e38f) amax = fmaxf(amax, a);
    }
    const float scale = amax > 0.f ? amax / 448.f : 1.f;
#pragma unroll
    for (int i = 0; i < HD; i += 16) {
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        w[k] = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) w[k] |= static_cast<uint32_t>(f32_to_e4m3(__fdiv_rn(o[i + 4 * k + b], scale))) << (8 * b);
      }
      *reinterpret_cast<uint4*>(p.out_fp8 + base + i) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    p.out_scale[static_cast<size_t>(head) * p.ld_scale + row] = scale;
  }
}

template <int HD, bool kStrict>
__global__ void __launch_bounds__(PfShape<HD>::kThreads, 1)
prefill_attention_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_kv, const PrefillParams p) {
  using S = PfShape<HD>;
  constexpr int kKeys = S::kKeys, kItems = S::kItems;
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_s = smem;                                     // [kItems]
  uint8_t* k_s = q_s + kItems * S::kQBytes;                // [2]
  uint8_t* v_s = k_s + 2 * S::kKvBytes;                    // [2]
  PrefillBarriers* bars = reinterpret_cast<PrefillBarriers*>(v_s + 2 * S::kKvBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int* tile = p.tiles + 4 * blockIdx.y;
  const int tok0 = tile[0], seq_len = tile[1], q0 = tile[2];
  const int head0 = p.pair_heads ? blockIdx.x * kItems : blockIdx.x;
  const int kvh = head0 / (p.hq / p.hkv);
  const int item_rows = p.pair_heads ? 0 : kPfTile;        // rows between the items
  const int rows_end = min(seq_len, q0 + (kItems - 1) * item_rows + kPfTile);
  const int first = p.window > 0 ? max(0, q0 - p.window + 1) / kKeys * kKeys : 0;
  const int nt = (rows_end - first + kKeys - 1) / kKeys;   // causal: key tiles up to the last row's
  volatile int* abort_flag = &bars->abort_flag;

  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->k_full[s], 1);
      mbar_init(&bars->k_empty[s], 1);
      mbar_init(&bars->v_full[s], 1);
      mbar_init(&bars->v_empty[s], 1);
      mbar_init(&bars->s_full[s], 1);
      mbar_init(&bars->p_ready[s], 128);
      mbar_init(&bars->o_full[s], 1);
    }
    bars->abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_kv);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  // No early trigger of dependent launches here: with one, the dependent GEMM's CTAs become resident
  // beside this kernel's for its whole run, and runs of a few hundred decode steps then showed an
  // occasional bounded wait of that GEMM running out (status 101, a 2 s stall); without it 1200 steps
  // ran clean.  Dependents therefore start when this grid completes.

  if (warp < 4) {
    // 128 x 72 + 256 x 216 of 384 x 168 registers; 128 x 72 + 128 x 216 of 256 x 168 and more
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == 0) {
      if (elect_one()) {
        const int xk = (p.hq + kvh) * HD, xv = (p.hq + p.hkv + kvh) * HD;
        mbar_expect_tx(&bars->q_full, kItems * S::kQBytes);
        for (int i = 0; i < kItems; ++i)
          for (int c = 0; c < S::kChunks; ++c)
            tma_load_2d(q_s + i * S::kQBytes + c * kPfTile * 128, &tm_q, &bars->q_full,
                        (head0 + (p.pair_heads ? i : 0)) * HD + c * 64, tok0 + q0 + i * item_rows);
        int ks = 0, vs = 0;
        for (int j = 0; j < nt; ++j) {
          const int st = j & 1, y = tok0 + first + j * kKeys;
          if (!mbar_wait(&bars->k_empty[st], ((j >> 1) & 1) ^ 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_SMEM_EMPTY)) break;
          mbar_expect_tx(&bars->k_full[st], S::kKvBytes);
          for (int c = 0; c < S::kChunks; ++c)
            tma_load_2d(k_s + st * S::kKvBytes + c * kKeys * 128, &tm_kv, &bars->k_full[st], xk + c * 64, y);
          ks = j + 1;
          if (!mbar_wait(&bars->v_empty[st], ((j >> 1) & 1) ^ 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_SMEM_EMPTY)) break;
          mbar_expect_tx(&bars->v_full[st], S::kKvBytes);
          for (int c = 0; c < S::kChunks; ++c)
            tma_load_2d(v_s + st * S::kKvBytes + c * kKeys * 128, &tm_kv, &bars->v_full[st], xv + c * 64, y);
          vs = j + 1;
        }
        // every copy has landed before the CTA may leave
        int dummy = 0;
        mbar_wait(&bars->q_full, 0, &dummy, p.status, SLLM_DEV_TIMEOUT_DRAIN, 200000000LL);
        for (int j = max(0, ks - 2); j < ks; ++j)
          mbar_wait(&bars->k_full[j & 1], (j >> 1) & 1, &dummy, p.status, SLLM_DEV_TIMEOUT_DRAIN, 200000000LL);
        for (int j = max(0, vs - 2); j < vs; ++j)
          mbar_wait(&bars->v_full[j & 1], (j >> 1) & 1, &dummy, p.status, SLLM_DEV_TIMEOUT_DRAIN, 200000000LL);
      }
      __syncwarp();
    } else if (warp == 1) {
      // S: A = Q (K-major), B = K tile (K-major).  PV: A = P (tensor memory), B = V tile (MN-major).
      constexpr uint32_t idesc_s = make_idesc(kFmtBf16, 128, kKeys, 0, 0);
      constexpr uint32_t idesc_pv = make_idesc(kFmtBf16, 128, HD, 0, 1);
      const uint32_t q_addr = smem_u32(q_s), k_addr = smem_u32(k_s), v_addr = smem_u32(v_s);
      // scores of item i (with one item: of tile j into buffer j & 1); the buffer's P has been multiplied by products issued earlier
      auto issue_s = [&](int i, int j) {
        const int b = kItems == 2 ? i : j & 1;
        const uint32_t ka = k_addr + (j & 1) * S::kKvBytes, qa = q_addr + i * S::kQBytes;
        if (elect_one()) {
#pragma unroll
          for (int c = 0; c < S::kChunks; ++c)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16(tmem_base + b * kKeys, make_smem_desc_sw128(qa + c * kPfTile * 128) + 2 * k,
                       make_smem_desc_sw128(ka + c * kKeys * 128) + 2 * k, idesc_s, (c | k) != 0);
          tc_commit(&bars->s_full[b]);
          if (i == kItems - 1) tc_commit(&bars->k_empty[j & 1]);
        }
        __syncwarp();
      };
      auto issue_pv = [&](int i, int j) {
        const int b = kItems == 2 ? i : j & 1;
        const uint32_t va = v_addr + (j & 1) * S::kKvBytes;
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < kKeys / 16; ++k) {           // 16 keys, 8 columns of P
            const uint64_t vd = make_smem_desc_sw128_mn(va + k * 16 * 128, kKeys * 128);
            const uint32_t o = tmem_base + S::kTmemO + i * HD, pa = tmem_base + b * kKeys + (kStrict ? k * 8 : k / 2 * 32 + (k & 1) * 8);
            umma_f16_ts(o, pa, vd, idesc_pv, (!kStrict && j > 0) || k > 0);
            if (!kStrict) umma_f16_ts(o, pa + 16, vd, idesc_pv, 1);
          }
          tc_commit(&bars->o_full[i]);
          if (i == kItems - 1) tc_commit(&bars->v_empty[j & 1]);
        }
        __syncwarp();
      };
      auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
        const bool ok = __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, p.status, code));
        tc_fence_after();
        return ok;
      };
      bool ok = wait(&bars->q_full, 0, SLLM_DEV_TIMEOUT_TMA_FULL) && wait(&bars->k_full[0], 0, SLLM_DEV_TIMEOUT_TMA_FULL);
      if (ok)
        for (int i = 0; i < kItems; ++i) issue_s(i, 0);
      const int own = seq_len - first - (nt - 1) * kKeys;  // keys of the last tile that are the sequence's (or more)
      for (int j = 0; ok && j < nt; ++j) {
        const bool more = j + 1 < nt;
        if (kItems == 1 && more) {                         // the next scores run under this tile's softmax
          ok = wait(&bars->k_full[(j + 1) & 1], ((j + 1) >> 1) & 1, SLLM_DEV_TIMEOUT_TMA_FULL);
          if (!ok) break;
          issue_s(0, j + 1);
        }
        ok = wait(&bars->v_full[j & 1], (j >> 1) & 1, SLLM_DEV_TIMEOUT_TMA_FULL);
        // Rows behind the sequence are another request's: their P is zero, but zero times an infinity of theirs would not be.
        // (Only the last tile has any; its stage is not filled again.)
        if (!more && own < kKeys) {
          uint8_t* v = v_s + (j & 1) * S::kKvBytes;
          for (int c = 0; c < S::kChunks; ++c)
            for (int e = (c * kKeys + own) * 8 + lane; e < (c + 1) * kKeys * 8; e += 32)       // 16-byte units
              *reinterpret_cast<uint4*>(v + e * 16) = make_uint4(0, 0, 0, 0);
          fence_proxy_async_smem();
          __syncwarp();
        }
        for (int i = 0; ok && i < kItems; ++i) {
          ok = kItems == 2 ? wait(&bars->p_ready[i], j & 1, SLLM_DEV_TIMEOUT_TMEM_EMPTY)
                           : wait(&bars->p_ready[j & 1], (j >> 1) & 1, SLLM_DEV_TIMEOUT_TMEM_EMPTY);
          if (!ok) break;
          issue_pv(i, j);
          if (kItems == 2 && more) {
            if (i == 0) ok = wait(&bars->k_full[(j + 1) & 1], ((j + 1) >> 1) & 1, SLLM_DEV_TIMEOUT_TMA_FULL);
            if (ok) issue_s(i, j + 1);
          }
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    const int item = (warp - 4) >> 2, q = warp & 3, r = q * 32 + lane;
    const int head = head0 + (p.pair_heads ? item : 0), qt = q0 + item * item_rows, qpos = qt + r;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t o_addr = lane_addr + S::kTmemO + item * HD;
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    if constexpr (kStrict) {
      strict_rows(p, bars, lane_addr, o_addr, item, head, qt, qpos, nt, tok0, seq_len, abort_flag);
    } else {
    for (int j = 0; j < nt; ++j) {
      const int b = kItems == 2 ? item : j & 1;
      const uint32_t ph = (kItems == 2 ? j : j >> 1) & 1, s_addr = lane_addr + b * kKeys;
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->s_full[b], ph, abort_flag, p.status, SLLM_DEV_TIMEOUT_TMEM_FULL));
      if (!ok) break;
      tc_fence_after();
      uint32_t sr[kKeys / 32][32];
#pragma unroll
      for (int c = 0; c < kKeys / 32; ++c) tmem_ld32(s_addr + c * 32, sr[c]);
#pragma unroll
      for (int c = 0; c < kKeys / 32; ++c) tmem_wait_regs(sr[c]);
      const int k0 = first + j * kKeys;
      const bool edge = k0 + kKeys - 1 > qt || (p.window > 0 && k0 <= qt + kPfTile - 1 - p.window);
      const int hi = edge ? qpos - k0 : kKeys, lo = edge && p.window > 0 ? qpos - k0 - p.window + 1 : 0;   // keys [lo, hi] are visible
      float mn[4] = {INFINITY, INFINITY, INFINITY, INFINITY};                // of visible keys
      if (edge) {
#pragma unroll
        for (int i = 0; i < kKeys; ++i) {
          if (i > hi || i < lo) sr[i >> 5][i & 31] = 0xff800000u;
          else mn[i & 3] = fminf(mn[i & 3], __uint_as_float(sr[i >> 5][i & 31]));
        }
      } else {
#pragma unroll
        for (int i = 0; i < kKeys; ++i) mn[i & 3] = fminf(mn[i & 3], __uint_as_float(sr[i >> 5][i & 31]));
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < kKeys; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(sr[i >> 5][i & 31]));
      const float m_new = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2;
      float alpha = 1.f;
      if (m == -INFINITY) {
        m = m_new;                                         // nothing but zeros in O and l
      } else if (m_new > m + 8.f) {
        alpha = pf_ex2<false>(m - m_new);
        l *= alpha;
        m = m_new;
      }
      if (__any_sync(0xffffffffu, alpha != 1.f)) {         // (not in the first tile)
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->o_full[item], (j - 1) & 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_TMEM_FULL));
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t o[32];
          tmem_ld32(o_addr + c * 32, o);
          tmem_wait_regs(o);
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st32(o_addr + c * 32, o);
        }
      }
      const float m_use = m == -INFINITY ? 0.f : m;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
      if (__any_sync(0xffffffffu, fmaf(fminf(fminf(mn[0], mn[1]), fminf(mn[2], mn[3])), p.scale_log2, -m_use) < -126.f)) {
        // subnormal probabilities: the exact exponential takes three instructions more, so it has a way of its own that reads the
        // scores again (8192 tokens, 32 heads x 128: 715 us with it throughout)
#pragma unroll 1
        for (int c = 0; c < kKeys / 32; ++c) {
          uint32_t v[32], h[16], e[16];
          tmem_ld32(s_addr + c * 32, v);
          tmem_wait_regs(v);
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i > hi || c * 32 + i < lo) v[i] = 0xff800000u;
          pf_probabilities<false>(v, p.scale_log2, m_use, h, e, sum);
          tmem_st16(s_addr + c * 32, h);
          tmem_st16(s_addr + c * 32 + 16, e);
        }
      } else {
#pragma unroll
        for (int c = 0; c < kKeys / 32; ++c) {
          uint32_t h[16], e[16];
          pf_probabilities<true>(sr[c], p.scale_log2, m_use, h, e, sum);
          tmem_st16(s_addr + c * 32, h);
          tmem_st16(s_addr + c * 32 + 16, e);
        }
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      tmem_wait_st();
      // With one item S(j + 1) says nothing of O(j - 1): each phase of o_full is seen before the next can complete, so that a parity
      // stands for one phase.  (Two items: S(j) follows PV(j - 1).)
      if (kItems == 1 && j > 0) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->o_full[0], (j - 1) & 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_TMEM_FULL));
        if (!ok) break;
      }
      tc_fence_before();
      mbar_arrive(&bars->p_ready[b]);
    }
    if (ok) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->o_full[item], (nt - 1) & 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_TMEM_FULL));
      tc_fence_after();
    }
    if (ok) {
      if (p.sinks && l > 0.f) l += pf_ex2<false>(fmaf(p.sinks[head], 1.4426950408889634f, -m));
      const float inv = l > 0.f ? 1.f / l : 0.f;
      const bool live = qpos < seq_len;
      const size_t row = static_cast<size_t>(tok0 + qpos), base = (row * p.hq + head) * HD;
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t o[32];
        tmem_ld32(o_addr + c * 32, o);
        tmem_wait_regs(o);
        if (live) {
          uint4* dst = reinterpret_cast<uint4*>(p.out_bf16 + base + c * 32);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 w;
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&w);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              h[k] = __floats2bfloat162_rn(__uint_as_float(o[i * 8 + 2 * k]) * inv, __uint_as_float(o[i * 8 + 2 * k + 1]) * inv);
            dst[i] = w;
          }
        }
      }
    }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int HD, bool kStrict>
static int prefill_go(const void* qkv, int total_tokens, int qkv_ld, int num_tiles, PrefillParams& p, cudaStream_t st) {
  using S = PfShape<HD>;
  CUtensorMap tq, tkv;
  int rc = cached_kmajor_tmap(&tq, qkv, 2, total_tokens, qkv_ld, static_cast<long long>(qkv_ld) * 2, kPfTile);
  if (rc == SLLM_OK) rc = cached_kmajor_tmap(&tkv, qkv, 2, total_tokens, qkv_ld, static_cast<long long>(qkv_ld) * 2, S::kKeys);
  if (rc != SLLM_OK) return rc;
  static bool cfg = false;
  if (!cfg) {
    if (cudaFuncSetAttribute(prefill_attention_kernel<HD, kStrict>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(S::kSmem)) !=
        cudaSuccess)
      return SLLM_ERR_CUDA;
    cfg = true;
  }
  const int heads = p.pair_heads ? p.hq / S::kItems : p.hq;
  return launch_kernel(prefill_attention_kernel<HD, kStrict>, dim3(heads, num_tiles), dim3(S::kThreads), S::kSmem, st, 1u, tq, tkv, p) == cudaSuccess
             ? SLLM_OK
             : SLLM_ERR_CUDA;
}

}  // namespace sllm

using namespace sllm;

// Query rows that a tile of sllm_prefill_attention covers: 256 where an item's neighbour is the next tile of its head.
SLLM_EXPORT int sllm_prefill_tile_rows(int hq, int hkv, int hd) {
  return hd == 256 || (hkv > 0 && (hq / hkv) % 2 == 0) ? kPfTile : 2 * kPfTile;
}

// tiles: device int32 [num_tiles][4] = {first token row of the sequence, sequence length, q0, 0}, q0 in steps of
// sllm_prefill_tile_rows, ordered by the caller (most keys first).  qkv row stride is qkv_ld elements.  window: 0 or the number of
// positions that a row sees; sm_scale > 0; sinks: optional [hq].  E4M3 results (out_fp8, out_scale): heads of 128 without window and sinks.
SLLM_EXPORT int sllm_prefill_attention(const void* qkv, int total_tokens, int qkv_ld, const int* tiles, int num_tiles,
                                       int hq, int hkv, int hd, int window, float sm_scale, const float* sinks, void* out_bf16,
                                       void* out_fp8, float* out_scale, int ld_scale, int* status, void* stream) {
  if (!qkv || !tiles || num_tiles <= 0 || hq <= 0 || hkv <= 0 || hq % hkv || window < 0 || !(sm_scale > 0.f)) return SLLM_ERR_INVALID_ARGUMENT;
  if ((hd != 64 && hd != 128 && hd != 256) || (out_fp8 && (hd != 128 || window || sinks)))
    return SLLM_ERR_UNSUPPORTED_SHAPE;
  if (!out_bf16 && !(out_fp8 && out_scale)) return SLLM_ERR_INVALID_ARGUMENT;
  if (num_tiles > 65535) return SLLM_ERR_LIMIT;
  if ((reinterpret_cast<uintptr_t>(out_bf16) | reinterpret_cast<uintptr_t>(out_fp8)) & 15) return SLLM_ERR_ALIGNMENT;
  PrefillParams p = {};
  p.tiles = tiles; p.hq = hq; p.hkv = hkv; p.window = window; p.scale_log2 = sm_scale * 1.4426950408889634f; p.sinks = sinks;
  p.pair_heads = sllm_prefill_tile_rows(hq, hkv, hd) == kPfTile;
  p.out_bf16 = static_cast<__nv_bfloat16*>(out_bf16); p.out_fp8 = static_cast<uint8_t*>(out_fp8);
  p.out_scale = out_scale; p.ld_scale = ld_scale; p.status = status;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (out_fp8) return prefill_go<128, true>(qkv, total_tokens, qkv_ld, num_tiles, p, st);
  return hd == 64 ? prefill_go<64, false>(qkv, total_tokens, qkv_ld, num_tiles, p, st)
                  : hd == 128 ? prefill_go<128, false>(qkv, total_tokens, qkv_ld, num_tiles, p, st)
                              : prefill_go<256, false>(qkv, total_tokens, qkv_ld, num_tiles, p, st);
}
