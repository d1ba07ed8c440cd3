// Product of many rows:  Y[m, n] = act(sum_k X[m, k] W[n, k]) (+ residual), bf16 out, for prompts (gemm_tcgen05.cu serves decoding).
// Operands are bf16, or E4M3 with one fp32 scale per row and 128 columns on both sides (the scaled form).
//
// What bounds it: the way of the operands to the tensor cores.  A 128 x 128 tile of one CTA needs 32 KB of operands per 4.2 MFLOP;
// two CTAs that share a 256 x BN tile (cta_group::2) hold half of W's tile each and need half of that for BN = 256.  Persistent
// pairs (one per two SMs) keep two accumulators in tensor memory, so that the output of a tile runs under the products of the next.
//
//   warp 0      producer: each CTA copies its 128 rows of X and BN / 2 rows of W per 128-byte K block; the bytes of both CTAs
//               count on the first CTA's barrier
//   warp 1      owns the tensor memory; in the first CTA it issues the products for both
//   warps 2, 3  scaled form: the scales of the K blocks, every other chunk of four each
//   warps 4 ..  epilogue, thread = output row: a group of four warps per 128 columns (64 for BN = 64)
// Scaled: every K block has an accumulator of its own (two or four in turn), which the epilogue warps fold into fp32 registers with
// scale_x[kb, m] scale_w[kb, n] while the next block is multiplied; fp32 pairs go through one instruction each.
// bf16: the K blocks i, i + parts, i + 2 parts, .. form partial sum i, in an accumulator of its own, and the epilogue warps add the
// partial sums in fp32 registers while the next one is multiplied.  Tensor memory rounds every addition towards zero, so that a
// chain of K / 64 blocks in one accumulator is off by twice as much as two chains of half the length (2048 x 4096 x 14336 of one
// sign: 7.0e-5 of the result against 3.0e-5, beyond the rounding to bf16).  The partial sums are those of the kernels that serve fewer
// rows (two of gemm_tcgen05.cu's issuers, four of gemm_w4.cu's), so that results have the same bits on both sides of the line.
// Tiles are visited in groups of eight columns of tiles, all rows within a group, so that what runs at one time shares its
// operands in L2.  Tiles leave through shared memory: a warp stores its own 32 x 64 pieces and waits for no other.
//
// Measured (B200, one launch, m x n x k, us; before: the 128 x 128 tiles of gemm_tcgen05.cu):
//                          bf16 before -> now             E4M3 before -> now
//   130 x 4096 x 4096          38 ->   31                     32 ->   25
//   527 x 6144 x 4096          71 ->   39                     58 ->   47
//   1500 x 2048 x 9216        129 ->   61                    106 ->   84
//   5400 x 4096 x 14336       909 ->  426                    736 ->  565
//   8192 x 28672 x 4096      3060 -> 1227 (1.57 PFLOP/s)    2500 -> 1634 (1.18 PFLOP/s)
// (bf16 in one chain per tile, which is less exact: 30, 35, 57, 414, 1220 us; with L2 warm the second takes 29.4 and 30.7.  The largest
// E4M3 product takes up to 2250 us right behind others of its size, when the power limit holds the clock.)
// bf16 with 256 columns keeps the tensor pipe 96 % active (4096 x 14336 x 4096); narrower tiles are held by operands out of L2.  E4M3
// spends about 2000 cycles a K block in the promotion (pipe 26 % active); reading 128 x 256 sums out of tensor memory alone takes 560.
#include "pair_mma.cuh"
#include "api.h"
#include "tmap.h"

namespace sllm {

constexpr int kGpRows = 128;                // rows of X per CTA, of W per CTA: BN / 2
constexpr int kGpMaxStages = 8;
constexpr int kGpScaleChunk = 4;            // K blocks whose scales are staged at a time
constexpr int kGpScaleRing = 4;             // such chunks in flight
constexpr int kGpGroupN = 8;                // columns of tiles per raster group

template <int BN, bool kScaled>
struct GpShape {
  static constexpr int kABytes = kGpRows * 128;
  static constexpr int kBBytes = BN / 2 * 128;
  static constexpr int kStage = kABytes + kBBytes;
  static constexpr int kStages = BN == 256 ? (kScaled ? 5 : 6) : BN == 128 ? 7 : 8;
  static constexpr int kGroups = BN >= 128 ? 2 : 1;        // epilogue groups of four warps
  static constexpr int kCols = BN / kGroups;               // columns per epilogue thread
  static constexpr int kThreads = 128 + 128 * kGroups;
  // 128 fp32 sums a thread need more than the 168 registers of 384 threads: the first four warps hand theirs over
  static constexpr bool kMoveRegs = kThreads == 384;
  static constexpr int kOutBytes = 4 * kGroups * 4096;     // 32 rows x 64 columns per epilogue warp
  static constexpr int kScaleBytes = kScaled ? kGpScaleRing * kGpScaleChunk * (kGpRows + BN) * 4 : 0;
  static constexpr int kAcc = BN < 256 ? 4 : 2;            // accumulators: of partial sums in turn; scaled: of K blocks
  static constexpr uint32_t kTmem = kAcc * BN;
};

struct __align__(16) GpShared {
  uint64_t full[kGpMaxStages];              // first CTA's: the bytes of both
  uint64_t empty[kGpMaxStages];
  uint64_t acc_full[4];
  uint64_t acc_empty[4];                    // first CTA's: the epilogue warps of both
  uint64_t scale_full[kGpScaleRing];
  uint64_t scale_empty[kGpScaleRing];
  uint32_t tmem_base;
  int abort_flag;
};

struct GpParams {
  int m, n, num_kb, tiles_m, tiles_n;
  int parts;                                // partial sums of a tile (scaled: one chain, promoted block by block)
  int ldy, ld_sx, ld_sw;
  int epilogue;                             // 0 store, 1 add residual, 2 square of relu, 3 soft cap
  float act_arg;
  const float* alpha;                       // optional factor of the sums (bf16 operands)
  int w_const;                              // no kernel writes w: its first tiles are requested ahead of the previous kernel's end
  const float *scale_x, *scale_w;           // [num_kb, ld]
  const __nv_bfloat16* residual;            // [m, ldy]
  int* status;
};

__device__ __forceinline__ void gp_cp_async4(void* dst, const void* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(in ? 4 : 0) : "memory");
}

// Tile number -> row and column of tiles.
__device__ __forceinline__ void gp_tile(const GpParams& p, int t, int& tm, int& tn) {
  const int per = kGpGroupN * p.tiles_m, g = t / per, r = t - g * per, wide = min(kGpGroupN, p.tiles_n - g * kGpGroupN);
  tm = r / wide;
  tn = g * kGpGroupN + r - tm * wide;
}

// The K blocks of a tile in the order that they are multiplied: those of partial sum 0, of partial sum 1, ..  (Two at a time, so that
// neighbours along K follow one another, took as long.)
struct GpBlocks {
  int kb = 0, part = 0;
  __device__ __forceinline__ bool first() const { return kb == part; }
  __device__ __forceinline__ bool last(const GpParams& p) const { return kb + p.parts >= p.num_kb; }
  __device__ __forceinline__ void next(const GpParams& p) {
    kb += p.parts;
    if (kb >= p.num_kb) kb = ++part;
  }
};

template <int BN, bool kScaled>
__global__ void __launch_bounds__(GpShape<BN, kScaled>::kThreads, 1)
gemm_prompt_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                   const __grid_constant__ CUtensorMap tm_y, const GpParams p) {
  using S = GpShape<BN, kScaled>;
  constexpr int kElems = kScaled ? 128 : 64;               // operand elements of a K block
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* out_s = smem + S::kStages * S::kStage;
  float* scale_s = reinterpret_cast<float*>(out_s + S::kOutBytes);     // [kGpScaleRing][kGpScaleChunk][kGpRows | BN]
  GpShared* sh = reinterpret_cast<GpShared*>(out_s + S::kOutBytes + S::kScaleBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_rank()), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int tiles = p.tiles_m * p.tiles_n;
  volatile int* abort_flag = &sh->abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::kStages; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    for (int b = 0; b < S::kAcc; ++b) {
      mbar_init(&sh->acc_full[b], 1);
      mbar_init(&sh->acc_empty[b], 2 * 4 * S::kGroups);
    }
    for (int b = 0; b < kGpScaleRing; ++b) {
      mbar_init(&sh->scale_full[b], 32);
      mbar_init(&sh->scale_empty[b], 4 * S::kGroups);
    }
    sh->abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_x);
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_y);
  }
  if (warp == 1) pair_tmem_alloc(&sh->tmem_base, S::kTmem);
  tc_fence_before();
  __syncthreads();
  cluster_sync_pair();                                     // both CTAs' barriers exist and both hold their tensor memory
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;

  if (warp < 4) {
    // with kMoveRegs 128 x 72 + 256 x 216 of the 384 x 168 registers of the launch
    if constexpr (S::kMoveRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == 0) {
      if (elect_one()) {
        auto load_w = [&](int s, int kb, int tn) {
          pair_tma_load_2d(smem + s * S::kStage + S::kABytes, &tm_w, leader_addr(&sh->full[s]), kb * kElems, tn * BN + rank * (BN / 2));
        };
        auto load_x = [&](int s, int kb, int tm) {
          pair_tma_load_2d(smem + s * S::kStage, &tm_x, leader_addr(&sh->full[s]), kb * kElems, (tm * 2 + rank) * kGpRows);
        };
        // the first stages' weights, which mostly do not depend on the previous kernel
        int tm, tn;
        gp_tile(p, pair, tm, tn);
        const int pre = min(p.num_kb, S::kStages);
        if (!p.w_const) pdl_wait();
        GpBlocks first;
        for (int i = 0; i < pre; ++i, first.next(p)) {
          if (rank == 0) mbar_expect_tx(&sh->full[i], 2 * S::kStage);
          load_w(i, first.kb, tn);
        }
        pdl_wait();
        int it = 0;                                        // K blocks over all tiles
        bool ok = true;
        for (int t = pair; ok && t < tiles; t += pairs) {
          gp_tile(p, t, tm, tn);
          GpBlocks b;
          for (int i = 0; i < p.num_kb; ++i, ++it, b.next(p)) {
            const int s = it % S::kStages;
            if (it >= pre) {
              if (!mbar_wait(&sh->empty[s], ((it / S::kStages) & 1) ^ 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_SMEM_EMPTY)) {
                ok = false;
                break;
              }
              if (rank == 0) mbar_expect_tx(&sh->full[s], 2 * S::kStage);
              load_w(s, b.kb, tn);
            }
            load_x(s, b.kb, tm);
          }
        }
        pdl_trigger();
        // every copy has landed before the pair may leave (at once unless something gave up): a stage's last fill
        if (rank == 0) {
          int dummy = 0;
          for (int j = max(0, it - S::kStages); j < it; ++j)
            mbar_wait(&sh->full[j % S::kStages], (j / S::kStages) & 1, &dummy, p.status, SLLM_DEV_TIMEOUT_DRAIN, 200000000LL);
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      if (rank == 0) {
        constexpr uint32_t idesc = make_idesc(kScaled ? kFmtE4M3 : kFmtBf16, 256, BN);
        int it = 0, acc = 0;                               // acc: accumulators handed over so far
        bool ok = true;
        for (int t = pair; ok && t < tiles; t += pairs) {
          GpBlocks b;
          for (int i = 0; i < p.num_kb; ++i, ++it, b.next(p)) {
            const int s = it % S::kStages, buf = acc % S::kAcc;
            ok = mbar_wait(&sh->full[s], (it / S::kStages) & 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_TMA_FULL);
            if (ok && (kScaled || b.first()))
              ok = mbar_wait(&sh->acc_empty[buf], ((acc / S::kAcc) & 1) ^ 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_TMEM_EMPTY);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t a_addr = smem_u32(smem + s * S::kStage);
            const uint64_t ad = make_smem_desc_sw128(a_addr), bd = make_smem_desc_sw128(a_addr + S::kABytes);
            const bool last = kScaled || b.last(p);
            if (elect_one()) {
#pragma unroll
              for (int k = 0; k < 4; ++k)                  // 4 x 32 bytes of K
                pair_umma<kScaled>(tmem_base + buf * BN, ad + 2 * k, bd + 2 * k, idesc, k > 0 || (!kScaled && !b.first()));
              pair_commit(&sh->empty[s]);
              if (last) pair_commit(&sh->acc_full[buf]);
            }
            __syncwarp();
            acc += last;
          }
        }
      }
    } else if (kScaled) {
      pdl_wait();
      const int chunks = (p.num_kb + kGpScaleChunk - 1) / kGpScaleChunk;
      int ci = 0;                                          // chunks over all tiles
      bool ok = true;
      for (int t = pair; ok && t < tiles; t += pairs) {
        int tm, tn;
        gp_tile(p, t, tm, tn);
        const int m0 = (tm * 2 + rank) * kGpRows, n0 = tn * BN;
        for (int c = 0; c < chunks; ++c, ++ci) {
          if ((ci & 1) != (warp & 1)) continue;
          const int slot = ci % kGpScaleRing, kb0 = c * kGpScaleChunk, cnt = min(kGpScaleChunk, p.num_kb - kb0);
          ok = mbar_wait(&sh->scale_empty[slot], ((ci / kGpScaleRing) & 1) ^ 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_SMEM_EMPTY);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          float* dst = scale_s + slot * kGpScaleChunk * (kGpRows + BN);
          for (int j = 0; j < cnt; ++j, dst += kGpRows + BN) {
            const float* sx = p.scale_x + static_cast<size_t>(kb0 + j) * p.ld_sx + m0;
            const float* sw = p.scale_w + static_cast<size_t>(kb0 + j) * p.ld_sw + n0;
#pragma unroll
            for (int i = lane; i < kGpRows; i += 32) gp_cp_async4(dst + i, m0 + i < p.m ? sx + i : p.scale_x, m0 + i < p.m);
#pragma unroll
            for (int i = lane; i < BN; i += 32) gp_cp_async4(dst + kGpRows + i, n0 + i < p.n ? sw + i : p.scale_w, n0 + i < p.n);
          }
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&sh->scale_full[slot])) : "memory");
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  } else {
    if constexpr (S::kMoveRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    pdl_wait();
    const int q = warp & 3, grp = (warp - 4) >> 2, row = q * 32 + lane;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + grp * S::kCols;
    uint8_t* stage = out_s + (warp - 4) * 4096;
    uint8_t* stage_row = stage + lane * 128;
    const uint32_t empty_addr = leader_addr(&sh->acc_empty[0]);
    int acc = 0;
    bool ok = true;
    // 64 output columns: activation, residual, bf16, out
    auto emit = [&](const float (&v)[64], int y_row, int y_col) {
      if (lane == 0) bulk_wait_read();                     // the warp's last piece has left its buffer
      __syncwarp();
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          x[j] = v[u * 8 + j];
          if (p.epilogue == 2) x[j] = x[j] > 0.f ? x[j] * x[j] : 0.f;
          else if (p.epilogue == 3) x[j] = p.act_arg * tanhf(x[j] / p.act_arg);
        }
        if (p.epilogue == 1 && y_row + lane < p.m && y_col + u * 8 < p.n) {
          const uint4 rr = *reinterpret_cast<const uint4*>(p.residual + static_cast<size_t>(y_row + lane) * p.ldy + y_col + u * 8);
          const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>(&rr);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            x[2 * j] += __bfloat162float(r2[j].x);
            x[2 * j + 1] += __bfloat162float(r2[j].y);
          }
        }
        uint4 w;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&w);
#pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(x[2 * j], x[2 * j + 1]);
        *reinterpret_cast<uint4*>(stage_row + ((u ^ (lane & 7)) << 4)) = w;
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && y_row < p.m && y_col < p.n) {
        tma_store_2d(&tm_y, stage, y_col, y_row);
        bulk_commit();
      }
    };
    if constexpr (kScaled) {
      int ci = 0;                                          // chunks of scales over all tiles
      for (int t = pair; t < tiles; t += pairs) {
        int tm, tn;
        gp_tile(p, t, tm, tn);
        uint64_t sum[S::kCols / 2];
#pragma unroll
        for (int c = 0; c < S::kCols / 2; ++c) sum[c] = 0ull;
        for (int kb0 = 0; kb0 < p.num_kb; kb0 += kGpScaleChunk, ++ci) {
          const int slot = ci % kGpScaleRing, cnt = min(kGpScaleChunk, p.num_kb - kb0);
          if (ok) ok = mbar_wait(&sh->scale_full[slot], (ci / kGpScaleRing) & 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_TMA_FULL);
          for (int j = 0; j < cnt; ++j, ++acc) {
            const float* sc = scale_s + (slot * kGpScaleChunk + j) * (kGpRows + BN);
            const uint64_t sx = pack_f32x2(sc[row], sc[row]);
            const ulonglong2* sw = reinterpret_cast<const ulonglong2*>(sc + kGpRows + grp * S::kCols);
            if (ok) ok = mbar_wait(&sh->acc_full[acc % S::kAcc], (acc / S::kAcc) & 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_TMEM_FULL);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) {
              tc_fence_after();
              const uint32_t src = lane_addr + (acc % S::kAcc) * BN;
              // 32 columns at a time: their scales are read and multiplied while the sums are on their way
#pragma unroll
              for (int c = 0; c < S::kCols / 32; ++c) {
                uint32_t r[32];
                tmem_ld32(src + c * 32, r);
                uint64_t s2[16];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  const ulonglong2 w2 = sw[c * 8 + i];
                  s2[2 * i] = mul_f32x2(sx, w2.x);
                  s2[2 * i + 1] = mul_f32x2(sx, w2.y);
                }
                tmem_wait_regs(r);
                if (c == S::kCols / 32 - 1) {              // the accumulator is free for another block
                  tc_fence_before();
                  __syncwarp();
                  if (lane == 0) mbar_arrive_remote(empty_addr + 8 * (acc % S::kAcc));
                }
#pragma unroll
                for (int i = 0; i < 16; ++i)
                  sum[c * 16 + i] = fma_f32x2(pack_b32x2(r[2 * i], r[2 * i + 1]), s2[i], sum[c * 16 + i]);
              }
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh->scale_empty[slot]);
        }
        if (ok) {
#pragma unroll
          for (int c = 0; c < S::kCols / 64; ++c) {
            float v[64];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const float2 x = unpack_f32x2(sum[c * 32 + i]);
              v[2 * i] = x.x;
              v[2 * i + 1] = x.y;
            }
            emit(v, (tm * 2 + rank) * kGpRows + q * 32, tn * BN + grp * S::kCols + c * 64);
          }
        }
      }
    } else {
      const float alpha = p.alpha ? *p.alpha : 1.f;
      for (int t = pair; ok && t < tiles; t += pairs) {
        int tm, tn;
        gp_tile(p, t, tm, tn);
        float sum[S::kCols];
#pragma unroll
        for (int c = 0; c < S::kCols; ++c) sum[c] = 0.f;
        for (int part = 0; part < p.parts; ++part, ++acc) {
          ok = mbar_wait(&sh->acc_full[acc % S::kAcc], (acc / S::kAcc) & 1, abort_flag, p.status, SLLM_DEV_TIMEOUT_TMEM_FULL);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < S::kCols / 32; ++c) {
            uint32_t r[32];
            tmem_ld32(lane_addr + (acc % S::kAcc) * BN + c * 32, r);
            tmem_wait_regs(r);
#pragma unroll
            for (int j = 0; j < 32; ++j) sum[c * 32 + j] += __uint_as_float(r[j]);
          }
          tc_fence_before();                               // all of it is in registers
          __syncwarp();
          if (lane == 0) mbar_arrive_remote(empty_addr + 8 * (acc % S::kAcc));
        }
        if (!ok) break;
#pragma unroll
        for (int c = 0; c < S::kCols / 64; ++c) {
          float v[64];
#pragma unroll
          for (int i = 0; i < 64; ++i) v[i] = sum[c * 64 + i] * alpha;
          emit(v, (tm * 2 + rank) * kGpRows + q * 32, tn * BN + grp * S::kCols + c * 64);
        }
      }
    }
    if (lane == 0) bulk_wait_all();
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_pair();                                     // nothing of the other CTA reaches this one any more
  if (warp == 1) {
    tc_fence_after();
    pair_tmem_dealloc(tmem_base, S::kTmem);
  }
}

template <int BN, bool kScaled>
static int gemm_prompt_go(const void* x, const void* w, void* y, long long ldx, int k, GpParams& p, cudaStream_t st) {
  using S = GpShape<BN, kScaled>;
  const int eb = kScaled ? 1 : 2;
  CUtensorMap tx, tw, ty;
  int rc = cached_kmajor_tmap(&tx, x, eb, p.m, k, ldx * eb, kGpRows);
  if (rc == SLLM_OK) rc = cached_kmajor_tmap(&tw, w, eb, p.n, k, static_cast<long long>(k) * eb, BN / 2);
  if (rc == SLLM_OK) rc = cached_kmajor_tmap(&ty, y, 2, p.m, p.n, static_cast<long long>(p.ldy) * 2, 32);
  if (rc != SLLM_OK) return rc;
  p.tiles_m = (p.m + 255) / 256;
  p.tiles_n = (p.n + BN - 1) / BN;
  const size_t smem = S::kStages * S::kStage + S::kOutBytes + S::kScaleBytes + sizeof(GpShared) + 1024;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_prompt_kernel<BN, kScaled>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) !=
        cudaSuccess)
      return SLLM_ERR_CUDA;
    configured = true;
  }
  const long long tiles = static_cast<long long>(p.tiles_m) * p.tiles_n;
  const int pairs = tiles < 74 ? static_cast<int>(tiles) : 74;
  return launch_kernel_cluster(gemm_prompt_kernel<BN, kScaled>, dim3(2 * pairs), dim3(S::kThreads), smem, st, 2u, 1u, tx, tw, ty, p) ==
                 cudaSuccess
             ? SLLM_OK
             : SLLM_ERR_CUDA;
}

}  // namespace sllm

using namespace sllm;

// x [m, k] (row stride ldx elements), w [n, k] contiguous, y [m, n] bf16 (row stride ldy): bf16 operands, or with scale_x / scale_w
// E4M3 and scales [ceil(k / 128), ld].  epilogue: 0 store, 1 add residual [m, ldy], 2 square of relu, 3 act_arg tanh(. / act_arg).
// alpha: optional device scalar that multiplies the sums of bf16 operands.  parts: partial sums of bf16 operands, 1 to 4 (K blocks of 64
// taken in turn).  w_const: no kernel of the stream writes w.  bn: columns of a pair's tile, 128, 256 or (scaled) 64.  n and ldy
// are multiples of 8, rows of x and w of 16 bytes.
SLLM_EXPORT int sllm_gemm_prompt(const void* x, const void* w, void* y, const float* scale_x, const float* scale_w, const void* residual,
                                 int m, int n, int k, long long ldx, int ldy, int ld_sx, int ld_sw, int epilogue, float act_arg,
                                 const float* alpha, int parts, int w_const, int bn, int* status, void* stream) {
  if (!x || !w || !y || m <= 0 || n <= 0 || k <= 0 || ldx < k || ldy < n || epilogue < 0 || epilogue > 3 || (epilogue == 1) != (residual != nullptr))
    return SLLM_ERR_INVALID_ARGUMENT;
  if (epilogue == 3 && !(act_arg > 0.f)) return SLLM_ERR_INVALID_ARGUMENT;
  if (parts < 1 || parts > 4) return SLLM_ERR_INVALID_ARGUMENT;
  if (scale_x && (alpha || parts != 1)) return SLLM_ERR_UNSUPPORTED_SHAPE;
  if (!scale_x != !scale_w || (scale_x && (ld_sx < m || ld_sw < n))) return SLLM_ERR_INVALID_ARGUMENT;
  if ((n & 7) || (ldy & 7) || (reinterpret_cast<uintptr_t>(residual) & 15)) return SLLM_ERR_ALIGNMENT;
  const bool scaled = scale_x != nullptr;
  GpParams p = {};
  p.m = m; p.n = n; p.num_kb = scaled ? (k + 127) / 128 : (k + 63) / 64;
  p.parts = parts < p.num_kb ? parts : p.num_kb;
  p.ldy = ldy; p.ld_sx = ld_sx; p.ld_sw = ld_sw; p.epilogue = epilogue; p.act_arg = act_arg; p.alpha = alpha; p.w_const = w_const;
  p.scale_x = scale_x; p.scale_w = scale_w; p.residual = static_cast<const __nv_bfloat16*>(residual); p.status = status;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (bn) {
    case 64: return scaled ? gemm_prompt_go<64, true>(x, w, y, ldx, k, p, st) : SLLM_ERR_UNSUPPORTED_SHAPE;
    case 128: return scaled ? gemm_prompt_go<128, true>(x, w, y, ldx, k, p, st) : gemm_prompt_go<128, false>(x, w, y, ldx, k, p, st);
    case 256: return scaled ? gemm_prompt_go<256, true>(x, w, y, ldx, k, p, st) : gemm_prompt_go<256, false>(x, w, y, ldx, k, p, st);
    default: return SLLM_ERR_INVALID_ARGUMENT;
  }
}
