// Attention in ONE kernel on the 5th-generation tensor cores (sm_100a):
//   S = scale * q^T k  ->  softmax over keys  ->  out = P v            (per image / head)
// (qdiff/quant_block.py:344-360 and 191-203, ldm/modules/diffusionmodules/openaimodel.py:384-406:
// the reference keeps both matmuls and the softmax in floating point).  fp32 accuracy comes from
// split-bf16 operands as in gemm_bf16_tc.cu (hi*hi + hi*lo + lo*hi, fp32 accumulation in tensor
// memory).  Scores and probabilities never touch global memory.
//
// A CTA owns 128 queries of one image at a time and walks the keys in blocks of 128:
//   phase 1  tcgen05.mma (M=128, N=128) accumulates a block's scores in one of two score buffers
//            (tensor-memory columns [0, 128) and [128, 256)) from TMA-fed q / k plane tiles; the
//            scores of block b + 1 are multiplied while the softmax works on block b;
//   phase 2  the epilogue warps hold the block's scores in registers, fold its row maximum into the
//            running maximum (online softmax: the output accumulator is rescaled in tensor memory
//            in the warps where a maximum grew), and write the UNNORMALISED probabilities
//            exp(s - max) as two bf16 planes straight into shared memory in the 128-byte-swizzled
//            K-major layout an MMA A operand needs;
//   phase 3  tcgen05.mma (N=channels<=256) accumulates P v in columns [256, 512), A operand
//            = those shared-memory planes, B operand = TMA-fed v plane tiles;
//   phase 4  after the last key block the epilogue divides by the row sum and writes
//            out[image][channel][query].
// A stage of the operand ring holds both planes of both operands of a 64-element K chunk (phase 1:
// q and k, phase 3: v), i.e. all three products of it, so nothing is copied twice; heads of up to 64
// channels keep the two q tiles in shared memory for all key blocks, and four smaller stages.
// Bound: the softmax's instruction issue and the tensor pipe about equally.  Measured with the plane
// splits in front, key blocks of 256 with one score buffer -> this: 16 heads x 40 channels x 4096
// tokens 530 -> 360 us, 40 x 24 x 1024 119 -> 90 us, 16 x 80 x 1024 60 -> 47 us, 128 x 40 x 4096 queries
// x 77 keys 220 -> 205 us, 256 x 256 x 256 162 -> 161 us; error against 64 bits unchanged (6e-6 - 1.6e-5).
// Every mbarrier wait is bounded, and a softmax warp that gave up joins the rest of the named barriers, so
// that no other warp is left at one.
#include "common.cuh"
#include "tc_common.cuh"

namespace modiff {
namespace {

constexpr int kChunkBytes = 128;                 // 64 bf16 of K per tile row
constexpr int kATile = 128 * kChunkBytes;        // 16 KB: 128 queries
constexpr int kMaxStages = 4;
constexpr int kRingBytes = 8 * kATile;           // 128 KB: 2 stages of 64 KB or 4 of 32 KB
constexpr int kQBytes = 2 * kATile;              // resident q planes of heads of up to 64 channels
constexpr int kPBytes = 2 * 2 * kATile;          // two planes x two 64-key chunks (128 keys) x 16 KB
constexpr int kEpiWarps = 8;
constexpr int kThreads = 64 + 32 * kEpiWarps;

struct AttnParams {
  int batch, c, t, tk;          // images*heads, channels per head, queries, keys
  int tkp;                      // keys padded to a multiple of 64
  int crow;                     // channel rows of the v planes (multiple of 64, <= 256)
  int cch;                      // 64-element K chunks of phase 1: ceil(cp / 64)
  int n_s;                      // score columns per key block: min(128, tkp)
  int nsb;                      // key blocks: ceil(tkp / 128)
  int q_resident;               // one K chunk: q stays in shared memory for all key blocks
  int stages, stage_bytes;
  int q_tiles;                  // ceil(t / 128)
  int total_tiles;
  float scale;
  float* out;                   // [batch][c][t]
};

// two floats -> packed bf16 pair (round to nearest even), first argument in the low half
__device__ inline uint32_t bf16_pair(float lo_half, float hi_half) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi_half), "f"(lo_half));
  return r;
}
// 2^x for x <= 0 through the hardware exp2 (relative error ~2^-22, far below the 2^-16 the
// split probabilities keep)
__device__ inline float exp2_neg(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The twelve MMAs of one K chunk: hi*hi, hi*lo, lo*hi of two planes each, one elected lane.
__device__ inline void issue_chunk(uint32_t d_tmem, uint32_t a_hi, uint32_t a_lo, uint32_t b_hi,
                                   uint32_t b_lo, uint32_t idesc, bool fresh) {
  const uint64_t ah = make_smem_desc(a_hi), al = make_smem_desc(a_lo);
  const uint64_t bh = make_smem_desc(b_hi), bl = make_smem_desc(b_lo);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    tc_mma_bf16(d_tmem, ah + (uint64_t)(2 * k), bh + (uint64_t)(2 * k), idesc, (fresh && k == 0) ? 0u : 1u);
#pragma unroll
  for (int k = 0; k < 4; ++k) tc_mma_bf16(d_tmem, ah + (uint64_t)(2 * k), bl + (uint64_t)(2 * k), idesc, 1u);
#pragma unroll
  for (int k = 0; k < 4; ++k) tc_mma_bf16(d_tmem, al + (uint64_t)(2 * k), bh + (uint64_t)(2 * k), idesc, 1u);
}

__global__ void __launch_bounds__(kThreads, 1)
attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const AttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[kMaxStages], bar_empty[kMaxStages];
  __shared__ __align__(8) uint64_t bar_s_full[2], bar_q_full, bar_q_empty;
  __shared__ __align__(8) uint64_t bar_p_ready, bar_p_free, bar_o_full, bar_o_empty;
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh;
  __shared__ float red_max[2][128], red_sum[2][128];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  volatile int* abort_flag = &abort_sh;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t p_smem = raw;                       // probability planes
  const uint32_t ring = raw + kPBytes;               // operand stages
  const uint32_t q_smem = ring + kRingBytes;         // resident q planes

  if (threadIdx.x == 0) {
    abort_sh = 0;
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    mbar_init(smem_u32(&bar_s_full[0]), 1);
    mbar_init(smem_u32(&bar_s_full[1]), 1);
    mbar_init(smem_u32(&bar_q_full), 1);
    mbar_init(smem_u32(&bar_q_empty), 1);
    mbar_init(smem_u32(&bar_p_ready), kEpiWarps);
    mbar_init(smem_u32(&bar_p_free), 1);
    mbar_init(smem_u32(&bar_o_full), 1);
    mbar_init(smem_u32(&bar_o_empty), kEpiWarps);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base_sh)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_sh;
  const uint32_t k_tile_bytes = (uint32_t)p.n_s * kChunkBytes;
  const uint32_t v_tile_bytes = (uint32_t)p.crow * kChunkBytes;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    // Stages in the order the MMA warp consumes them: scores(0), then scores(b + 1), values(b) ...
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0, qphase = 0;
      bool ok = true;
      auto scores = [&](int img, int qt, int sb) {
        for (int ch = 0; ch < p.cch && ok; ++ch) {
          ok = mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1u, abort_flag);
          if (!ok) return;
          const uint32_t full = smem_u32(&bar_full[stage]);
          const uint32_t dst = ring + stage * p.stage_bytes;
          const uint32_t k_dst = dst + (p.q_resident ? 0 : 2 * kATile);
          mbar_arrive_expect_tx(full, 2 * k_tile_bytes + (p.q_resident ? 0u : 2u * kATile));
          for (int part = 0; part < 2; ++part) {
            if (!p.q_resident)
              tma_load_3d(dst + part * kATile, &map_q, full, ch * 64, qt * 128, img * 2 + part);
            // key rows beyond tkp are filled with zeros by the copy and masked in the softmax
            tma_load_3d(k_dst + part * kATile, &map_k, full, ch * 64, sb * 128, img * 2 + part);
          }
          if (++stage == p.stages) { stage = 0; phase ^= 1u; }
        }
      };
      for (int tile = blockIdx.x; tile < p.total_tiles && ok; tile += gridDim.x) {
        const int img = tile / p.q_tiles, qt = tile % p.q_tiles;
        if (p.q_resident) {
          ok = mbar_wait(smem_u32(&bar_q_empty), qphase ^ 1u, abort_flag);
          qphase ^= 1u;
          if (!ok) break;
          const uint32_t full = smem_u32(&bar_q_full);
          mbar_arrive_expect_tx(full, 2u * kATile);
          for (int part = 0; part < 2; ++part)
            tma_load_3d(q_smem + part * kATile, &map_q, full, 0, qt * 128, img * 2 + part);
        }
        scores(img, qt, 0);
        for (int sb = 0; sb < p.nsb && ok; ++sb) {
          if (sb + 1 < p.nsb) scores(img, qt, sb + 1);
          const int kch = min(2, (p.tkp - sb * 128) >> 6);
          for (int kc = 0; kc < kch && ok; ++kc) {
            ok = mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1u, abort_flag);
            if (!ok) break;
            const uint32_t full = smem_u32(&bar_full[stage]);
            mbar_arrive_expect_tx(full, 2 * v_tile_bytes);
            for (int part = 0; part < 2; ++part)
              tma_load_3d(ring + stage * p.stage_bytes + part * v_tile_bytes, &map_v, full,
                          sb * 128 + kc * 64, 0, img * 2 + part);
            if (++stage == p.stages) { stage = 0; phase ^= 1u; }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    // All lanes walk the loop (descriptors and addresses stay warp-uniform values); one
    // elected lane issues the MMAs and commits.
    {
      const uint32_t idesc_s = make_idesc_bf16(128, p.n_s);
      const uint32_t idesc_o = make_idesc_bf16(128, p.crow);
      int stage = 0;
      uint32_t phase = 0, tphase = 0, pphase = 0, qphase = 0;
      bool ok = true;
      // scores of key block sb into its buffer.  The softmax has finished reading that buffer's
      // previous scores: its p_ready for them preceded the values product issued before this one
      // (or, for the first two blocks of a tile, the previous tile's last ones).
      auto scores = [&](int sb) {
        for (int ch = 0; ch < p.cch; ++ch) {
          ok = mbar_wait(smem_u32(&bar_full[stage]), phase, abort_flag);
          if (!ok) return;
          tc_fence_after();
          const uint32_t src = ring + stage * p.stage_bytes;
          const uint32_t a_src = p.q_resident ? q_smem : src;
          const uint32_t b_src = p.q_resident ? src : src + 2 * kATile;
          if (elect_one()) {
            issue_chunk(tmem_base + (uint32_t)((sb & 1) * 128), a_src, a_src + kATile, b_src, b_src + kATile,
                        idesc_s, ch == 0);
            tc_commit(smem_u32(&bar_empty[stage]));
            if (ch == p.cch - 1) {
              tc_commit(smem_u32(&bar_s_full[sb & 1]));
              if (p.q_resident && sb == p.nsb - 1) tc_commit(smem_u32(&bar_q_empty));
            }
          }
          __syncwarp();
          if (++stage == p.stages) { stage = 0; phase ^= 1u; }
        }
      };
      for (int tile = blockIdx.x; tile < p.total_tiles; tile += gridDim.x) {
        bool fresh_pv = true;
        if (p.q_resident) {
          ok = mbar_wait(smem_u32(&bar_q_full), qphase, abort_flag);
          qphase ^= 1u;
          if (!ok) break;
        }
        scores(0);
        for (int sb = 0; sb < p.nsb && ok; ++sb) {
          if (sb + 1 < p.nsb) scores(sb + 1);
          if (!ok) break;
          // phase 3: the probability planes of this block sit in shared memory; the tile's first
          // product also needs the previous tile's output drained
          ok = mbar_wait(smem_u32(&bar_p_ready), pphase, abort_flag);
          pphase ^= 1u;
          if (ok && fresh_pv) ok = mbar_wait(smem_u32(&bar_o_empty), tphase ^ 1u, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const int kch = min(2, (p.tkp - sb * 128) >> 6);
          for (int kc = 0; kc < kch; ++kc) {
            ok = mbar_wait(smem_u32(&bar_full[stage]), phase, abort_flag);
            if (!ok) break;
            tc_fence_after();
            const uint32_t a_src = p_smem + (uint32_t)(kc * kATile);     // plane stride 2 tiles
            const uint32_t b_src = ring + stage * p.stage_bytes;
            if (elect_one()) {
              issue_chunk(tmem_base + 256u, a_src, a_src + 2 * kATile, b_src, b_src + v_tile_bytes, idesc_o,
                          fresh_pv);
              tc_commit(smem_u32(&bar_empty[stage]));
              if (kc == kch - 1) tc_commit(smem_u32(&bar_p_free));
            }
            __syncwarp();
            fresh_pv = false;
            if (++stage == p.stages) { stage = 0; phase ^= 1u; }
          }
        }
        if (!ok) break;
        if (elect_one()) tc_commit(smem_u32(&bar_o_full));
        __syncwarp();
        tphase ^= 1u;
      }
    }
  } else {
    // ------------------------------------------------------------ softmax + epilogue (warps 2..9)
    // Two warps share a tensor-memory lane quarter; a lane is one query row, each warp of the
    // pair takes half of the columns.
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int ccols = p.crow >> 1;           // channel columns of this warp (multiple of 32)
    uint8_t* p_ptr = smem_raw;
    uint32_t tphase = 0, sphases = 0, fphase = 0;     // bit i of sphases: score buffer i
    // scores in units of log2: exp(scale * s) = 2^(s * scale2)
    const float scale2 = p.scale * 1.4426950408889634f;
    bool ok = true;
    int tile = blockIdx.x, left = 0;                  // left: named barriers that a failed wait skipped
    for (; tile < p.total_tiles; tile += gridDim.x) {
      const int img = tile / p.q_tiles, qt = tile % p.q_tiles;
      const int q = qt * 128 + row;
      float m_run = -INFINITY;      // running row maximum (the same in both warps of a pair)
      float l_part = 0.0f;          // running sum of this warp's columns, in units of 2^(-m_run)
      for (int sb = 0; sb < p.nsb; ++sb) {
        const int nk = min(128, p.tkp - sb * 128) >> 1;       // this warp's keys: 32 or 64
        ok = mbar_wait(smem_u32(&bar_s_full[sb & 1]), (sphases >> (sb & 1)) & 1u, abort_flag);
        sphases ^= 1u << (sb & 1);
        if (!ok) { left = 2 * (p.nsb - sb) + 1; break; }
        tc_fence_after();
        // ---- this warp's scores -> registers; row maximum folded into the running maximum
        float s[64];
        float mx = -INFINITY;
#pragma unroll
        for (int c0 = 0; c0 < 64; c0 += 32) {
          if (c0 < nk) {
            const int col0 = half * nk + c0;
            int a[32];
            tc_ld32(t_lane + (uint32_t)((sb & 1) * 128 + col0), a);
            tc_wait_ld();
            const int left = p.tk - (sb * 128 + col0);        // real keys from this column on
            if (left >= 32) {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                s[c0 + j] = __int_as_float(a[j]) * scale2;
                mx = fmaxf(mx, s[c0 + j]);
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                s[c0 + j] = __int_as_float(a[j]) * scale2;
                if (j < left) mx = fmaxf(mx, s[c0 + j]);
              }
            }
          }
        }
        red_max[half][row] = mx;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        const float m_new = fmaxf(m_run, fmaxf(red_max[0][row], red_max[1][row]));
        // 2^(m_run - m_new): 0 for the first block (m_run = -inf), 1 while the maximum stands
        const float alpha = exp2_neg(m_run - m_new);
        l_part *= alpha;
        m_run = m_new;
        // ---- exp, row sum, probabilities -> shared memory (K-major rows of 128 bytes, the
        //      16-byte chunk index XORed with row % 8: the layout TMA writes with 128-byte swizzle)
        // the MMAs that read the previous contents of the planes (and accumulated into the
        // output columns) have completed
        ok = mbar_wait(smem_u32(&bar_p_free), fphase ^ 1u, abort_flag);
        fphase ^= 1u;
        if (!ok) { left = 2 * (p.nsb - sb); break; }
        if (sb > 0 && __any_sync(0xffffffffu, alpha != 1.0f)) {
          // online softmax: bring the accumulated output to the new maximum
          tc_fence_after();
          for (int c0 = 0; c0 < ccols; c0 += 32) {
            int a[32];
            tc_ld32(t_lane + 256u + (uint32_t)(half * ccols + c0), a);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) a[j] = __float_as_int(__int_as_float(a[j]) * alpha);
            tc_st32(t_lane + 256u + (uint32_t)(half * ccols + c0), a);
          }
          tc_wait_st();
        }
#pragma unroll
        for (int c0 = 0; c0 < 64; c0 += 32) {
          if (c0 < nk) {
            const int col0 = half * nk + c0;                  // multiple of 32
            const int left = p.tk - (sb * 128 + col0);
            const int kc = col0 >> 6;                         // 64-key chunk of the block
            const int chunk0 = (col0 & 63) >> 3;              // first 16-byte chunk of the row: 0 or 4
            uint8_t* hi_row = p_ptr + (size_t)(0 * 2 + kc) * kATile + (size_t)row * 128;
            uint8_t* lo_row = p_ptr + (size_t)(1 * 2 + kc) * kATile + (size_t)row * 128;
#pragma unroll
            for (int g8 = 0; g8 < 4; ++g8) {
              uint32_t hw[4], lw[4];
#pragma unroll
              for (int e = 0; e < 8; e += 2) {
                float pv[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                  const int j = g8 * 8 + e + u;
                  pv[u] = exp2_neg(s[c0 + j] - m_run);
                  if (left < 32) pv[u] = j < left ? pv[u] : 0.0f;
                  l_part += pv[u];
                }
                const uint32_t h = bf16_pair(pv[0], pv[1]);
                hw[e >> 1] = h;
                lw[e >> 1] = bf16_pair(pv[0] - __uint_as_float(h << 16),
                                       pv[1] - __uint_as_float(h & 0xffff0000u));
              }
              const int chunk = (chunk0 + g8) ^ (row & 7);
              *reinterpret_cast<uint4*>(hi_row + chunk * 16) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
              *reinterpret_cast<uint4*>(lo_row + chunk * 16) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
            }
          }
        }
        // a block of 64 keys fills one chunk; its MMAs then read one chunk only
        tc_fence_before();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (lane == 0) mbar_arrive(smem_u32(&bar_p_ready));
      }
      if (!ok) break;
      red_sum[half][row] = l_part;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      const float inv = 1.0f / (red_sum[0][row] + red_sum[1][row]);
      // ---- output
      ok = mbar_wait(smem_u32(&bar_o_full), tphase, abort_flag);
      if (!ok) break;
      tc_fence_after();
      for (int c0 = 0; c0 < ccols; c0 += 32) {
        int a[32];
        tc_ld32(t_lane + 256u + (uint32_t)(half * ccols + c0), a);
        tc_wait_ld();
        if (q < p.t) {
          float* dst = p.out + ((size_t)img * p.c + half * ccols + c0) * p.t + q;
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (half * ccols + c0 + j < p.c) dst[(size_t)j * p.t] = __int_as_float(a[j]) * inv;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_o_empty));
      tphase ^= 1u;
    }
    // after a failed wait: the barriers of the remaining tiles and those skipped
    for (tile += gridDim.x; tile < p.total_tiles; tile += gridDim.x) left += 2 * p.nsb + 1;
    for (; left > 0; --left) {
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
  }

  // ---------------------------------------------------------------- teardown
  __syncwarp();
  if (abort_sh) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u)
                 : "memory");
  }
}

}  // namespace

int read_device_status_attention(int* status, int reset) {
  return read_status_this_unit(status, reset);
}

}  // namespace modiff

using namespace modiff;

extern "C" int modiff_attention_tc(const uint16_t* q_planes, const uint16_t* k_planes,
                                   const uint16_t* v_planes, float* out, int batch, int c, int t,
                                   int tk, int cp, int tkp, int crow, float scale, void* stream) {
  MODIFF_CHECK_ARG(q_planes && k_planes && v_planes && out, "NULL pointer argument");
  MODIFF_CHECK_ARG(batch > 0 && c > 0 && t > 0 && tk > 0, "bad shape");
  if (tkp < tk || tkp % 64 || crow < c || crow > 256 || crow % 64 || cp < c || cp % 8 || cp < 64 ||
      cp > 256)
    return set_error(MODIFF_ERR_UNSUPPORTED,
                     "single-kernel attention needs keys padded to a multiple of 64, channel rows a "
                     "multiple of 64 <= 256 and 64 <= cp <= 256 (got tkp=%d crow=%d cp=%d)", tkp, crow,
                     cp);
  MODIFF_CHECK_ARG((((uintptr_t)q_planes | (uintptr_t)k_planes | (uintptr_t)v_planes) & 15) == 0,
                   "plane buffers must be 16-byte aligned");
  EncodeTiledFn encode = get_encode_fn();
  if (!encode) return set_error(MODIFF_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is not available");

  AttnParams p;
  p.batch = batch;
  p.c = c;
  p.t = t;
  p.tk = tk;
  p.tkp = tkp;
  p.crow = crow;
  p.cch = ceil_div(cp, 64);
  p.n_s = tkp < 128 ? tkp : 128;
  p.nsb = ceil_div(tkp, 128);
  p.q_resident = p.cch == 1 && crow == 64;
  p.stage_bytes = p.q_resident ? 2 * kATile : 4 * kATile;
  p.stages = kRingBytes / p.stage_bytes;
  p.q_tiles = ceil_div(t, 128);
  p.total_tiles = batch * p.q_tiles;
  p.scale = scale;
  p.out = out;

  CUtensorMap map_q, map_k, map_v;
  auto make = [&](CUtensorMap* m, const void* base, int inner, int rows, int box_rows) -> CUresult {
    cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)rows, (cuuint64_t)batch * 2};
    cuuint64_t strides[2] = {(cuuint64_t)inner * 2, (cuuint64_t)inner * rows * 2};
    cuuint32_t box[3] = {64u, (cuuint32_t)box_rows, 1u};
    cuuint32_t estr[3] = {1, 1, 1};
    return encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box,
                  estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = make(&map_q, q_planes, cp, t, 128);            // [image*2+part][query][cp]
  if (r == CUDA_SUCCESS) r = make(&map_k, k_planes, cp, tkp, p.n_s);   // [image*2+part][key][cp]
  if (r == CUDA_SUCCESS) r = make(&map_v, v_planes, tkp, crow, crow);  // [image*2+part][channel][key]
  if (r != CUDA_SUCCESS)
    return set_error(MODIFF_ERR_CUDA, "cuTensorMapEncodeTiled(attention operands) failed: %d", (int)r);

  static int sm_count = 0;
  if (!sm_count) {
    int dev = 0;
    MODIFF_CUDA(cudaGetDevice(&dev));
    MODIFF_CUDA(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev));
  }
  const size_t smem = (size_t)kPBytes + kRingBytes + (p.q_resident ? kQBytes : 0);
  static SmemLimit smem_limit;
  MODIFF_CUDA(raise_smem_limit(attention_tc_kernel, smem, smem_limit));
  const int grid = p.total_tiles < sm_count ? p.total_tiles : sm_count;
  attention_tc_kernel<<<grid, kThreads, smem, (cudaStream_t)stream>>>(map_q, map_k, map_v, p);
  MODIFF_LAUNCH_CHECK("attention_tc_kernel");
  return MODIFF_OK;
}
