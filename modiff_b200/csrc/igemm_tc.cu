// Int8 implicit-GEMM conv / linear on the 5th-generation tensor cores (sm_100a):
//   - activation-code tiles (128 output pixels x 128 input channels of one filter tap) and
//     weight-code tiles arrive by TMA (cp.async.bulk.tensor, 128-byte swizzle) into a
//     shared-memory ring;
//   - one elected thread issues tcgen05.mma.cta_group::1.kind::i8 (M=128, N=128|144, K=32)
//     with int32 accumulators in tensor memory, double buffered across output tiles;
//   - eight epilogue warps read the accumulators with tcgen05.ld and apply the modulation
//     epilogue  out = o_hat + acc * delta_x * delta_w[c] (+ bias), writing the new o_hat.
// Persistent kernel, one CTA per SM, warp specialised (TMA / MMA / epilogue).
// Every mbarrier wait is bounded: when a limit runs out the kernel records an error word,
// every role leaves its loop, tensor memory is released and the kernel returns.
//
// Reference arithmetic: qdiff/quant_layer.py:345-365 (see igemm_simt.cu).
#include <cstdlib>

#include "common.cuh"
#include "tc_common.cuh"

namespace modiff {

int launch_igemm_simt(const int8_t* codes, const int8_t* wcodes, int with_sum_rows,
                      const float* x_scale, const float* w_scale, const int32_t* w_corr,
                      float* o_hat, int accumulate, const float* bias, const modiff_conv_geom* g,
                      int per_sample, int32_t* acc_out, cudaStream_t s, const float* x_zp,
                      const int32_t* w_csum);

namespace {

constexpr int kTileM = 128;
constexpr int kChunkK = 128;          // bytes of K per pipeline stage (one swizzle atom row)
constexpr int kATileBytes = kTileM * kChunkK;
constexpr int kEpiWarps = 8;
constexpr int kOSlots = 3;                // ring of cached-output half tiles (64 channels each)
constexpr int kOHalfBytes = 64 * 128 * 4;
constexpr int kThreads = 64 + 32 * kEpiWarps + 32;   // TMA warp, MMA warp, epilogue warps, store warp
constexpr int kStoreWarp = 2 + kEpiWarps;
constexpr int kMaxStages = 6;


struct TcParams {
  modiff_conv_geom g;
  Derived d;
  int bw, bh, bn;                // box of output pixels forming one M tile
  int tiles_w, tiles_h, tiles_n; // tiles along each direction
  int n_tiles;                   // output-channel tiles
  int total_tiles;
  int umma_n;                    // 128, or 144 with the receptive-field-sum rows
  int stages;
  int nbuf;                      // accumulator buffers in tensor memory (1 or 2)
  int buf_cols;                  // columns per buffer
  int tmem_cols;                 // allocation (power of two)
  int a_bytes;                   // bytes one activation-tile copy delivers
  int o_bytes;                   // bytes one cached-output-tile copy delivers
  int row_epi;                   // linear layers: the cached output is token-major [rows][cout];
                                 // a ring slot holds two swizzled boxes of 128 rows x 32 channels
  int chunks[2];                 // 128-byte K chunks per tap of segment 0 / 1
  int cbeg[2];                   // first channel of segment 0 / 1
  int nseg;
  int with_sum;
  int accumulate;
  int per_sample;
  int ksplit;                    // CTAs of a cluster sharing one tile's K range (1 = off)
  int fused_round;               // K split: round as the bulk-copy epilogue does (one fma)
  const float* x_scale;
  const float* w_scale;
  const int32_t* w_corr;
  const float* x_zp;             // offset (8-bit asymmetric) activation codes, else NULL
  const int32_t* w_csum;         // [2][cout] sum of centred weight codes per segment
  const float* bias;
  float* o_hat;
  int32_t* acc_out;
};

struct TileCoord {
  int tn, th, tw, nt;
};
__device__ inline TileCoord decode_tile(int tile, const TcParams& p) {
  TileCoord t;
  t.nt = tile % p.n_tiles;
  int m = tile / p.n_tiles;
  t.tw = m % p.tiles_w;
  m /= p.tiles_w;
  t.th = m % p.tiles_h;
  t.tn = m / p.tiles_h;
  return t;
}

// TMA_EPI: the cached-output tile arrives by bulk tensor copies (global -> shared, during the products).
// NCHW layers store the new values straight from registers - a lane is a pixel - and release the ring
// slot as soon as it has been read; sending them back through the slot with a bulk store cost another
// 0.25 - 0.45 us a launch (256 -> 256, 1x1 at 8x8, one image 6.1 -> 5.8 us; 768 -> 768 at 2x2, five
// images, unsplit 25.2 -> 23.1 us).  Token-major layers, whose lanes are rows, keep the bulk store.  Used for
// full-size layers with per-tensor scales and no bias; the generic variant reads and writes o_hat
// directly and covers everything else.
//
// KSPLIT (layers with fewer tiles than SMs, e.g. 768 channels at 2x2 or 4x4): a cluster of
// `p.ksplit` CTAs shares ONE tile.  Each CTA accumulates a contiguous part of the K range
// (taps x channel chunks) in its own tensor memory, leaves the int32 partial sums in its shared
// memory, and after a cluster barrier each CTA adds up, across the cluster's shared memories,
// the 128 / ksplit output channels it owns and applies the epilogue to them.  Integer addition
// is associative, so the accumulators equal the unsplit kernel's bit for bit.
template <int NSEG, bool WITH_SUM, bool TMA_EPI, bool KSPLIT = false>
__global__ void __launch_bounds__(kThreads, 1)
igemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                const __grid_constant__ CUtensorMap map_o, const TcParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[kMaxStages];
  __shared__ __align__(8) uint64_t bar_empty[kMaxStages];
  __shared__ __align__(8) uint64_t bar_tmem_full[2];
  __shared__ __align__(8) uint64_t bar_tmem_empty[2];
  __shared__ __align__(8) uint64_t bar_o_full[kOSlots];
  __shared__ __align__(8) uint64_t bar_o_empty[kOSlots];
  __shared__ __align__(8) uint64_t bar_o_ready[kOSlots];
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh;
  __shared__ float ep_scale[2][128];
  __shared__ int ep_corr[2][128];
  __shared__ int ep_off[2][128];
  __shared__ float ep_bias[128];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  volatile int* abort_flag = &abort_sh;

  // 1024-byte aligned tile ring (the dynamic segment is declared with that alignment),
  // followed by the cached-output ring
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t ring = raw;
  const int b_rows = p.umma_n;
  const uint32_t b_tile_bytes = (uint32_t)b_rows * kChunkK;
  const uint32_t stage_bytes = kATileBytes + ((b_tile_bytes + 1023u) & ~1023u);
  const uint32_t obuf = ring + (uint32_t)p.stages * stage_bytes;   // kOSlots x 32 KB
  float* obuf_ptr = reinterpret_cast<float*>(smem_raw + (obuf - raw));

  if (threadIdx.x == 0) {
    abort_sh = 0;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&bar_tmem_full[b]), 1);
      mbar_init(smem_u32(&bar_tmem_empty[b]), kEpiWarps);
    }
    for (int b = 0; b < kOSlots; ++b) {
      mbar_init(smem_u32(&bar_o_full[b]), 1);
      mbar_init(smem_u32(&bar_o_empty[b]), p.row_epi ? 1 : kEpiWarps);
      mbar_init(smem_u32(&bar_o_ready[b]), kEpiWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base_sh)),
                 "r"((uint32_t)p.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_sh;

  // KSPLIT: one tile per cluster, this CTA's share of its K iterations; else a persistent walk
  const int krank = KSPLIT ? (int)cluster_ctarank() : 0;
  const int tile_first = KSPLIT ? (int)blockIdx.x / p.ksplit : (int)blockIdx.x;
  const int tile_step = KSPLIT ? p.total_tiles : (int)gridDim.x;
  const int it_all = p.d.taps * p.chunks[0];
  const int it_lo = KSPLIT ? (krank * it_all) / p.ksplit : 0;
  const int it_hi = KSPLIT ? ((krank + 1) * it_all) / p.ksplit : it_all;

  const int k_iters_seg0 = p.d.taps * p.chunks[0];
  const int k_iters_seg1 = (p.nseg == 2) ? p.d.taps * p.chunks[1] : 0;
  const int howo = p.d.ho * p.d.wo;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      uint32_t ophase = 0;
      int oslot = 0;
      bool ok = true;
      for (int tile = tile_first; tile < p.total_tiles && ok; tile += tile_step) {
        const TileCoord t = decode_tile(tile, p);
        for (int seg = 0; seg < p.nseg && ok; ++seg) {
          for (int tap = 0; tap < p.d.taps && ok; ++tap) {
            const int r = tap / p.g.kw, sx = tap % p.g.kw;
            const int plane = (r % p.g.stride) * p.g.stride + (sx % p.g.stride);
            const int dh = r / p.g.stride, dw = sx / p.g.stride;
            for (int ch = 0; ch < p.chunks[seg]; ++ch) {
              if (KSPLIT) {
                const int itn = tap * p.chunks[0] + ch;
                if (itn < it_lo || itn >= it_hi) continue;    // another CTA of the cluster's
              }
              ok = mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1u, abort_flag);
              if (!ok) break;
              const uint32_t full = smem_u32(&bar_full[stage]);
              const uint32_t a_dst = ring + stage * stage_bytes;
              const uint32_t b_dst = a_dst + kATileBytes;
              const int c0 = p.cbeg[seg] + ch * kChunkK;
              mbar_arrive_expect_tx(full, (uint32_t)p.a_bytes + b_tile_bytes);
              tma_load_5d(a_dst, &map_a, full, c0, t.tw * p.bw + dw, t.th * p.bh + dh, plane,
                          t.tn * p.bn);
              tma_load_2d(b_dst, &map_b, full, tap * p.d.kp + c0, t.nt * b_rows);
              if (++stage == p.stages) { stage = 0; phase ^= 1u; }
            }
          }
        }
        if (TMA_EPI && ok) {
          // After this tile's operand copies are queued: claim two slots of the cached-output
          // ring (as soon as earlier stores have drained them) and fetch both 64-channel halves.
          for (int half = 0; half < 2 && ok; ++half) {
            ok = mbar_wait(smem_u32(&bar_o_empty[oslot]), ophase ^ 1u, abort_flag);
            if (!ok) break;
            const uint32_t ofull = smem_u32(&bar_o_full[oslot]);
            if (p.accumulate && p.row_epi) {
              mbar_arrive_expect_tx(ofull, (uint32_t)kOHalfBytes);
              for (int b2 = 0; b2 < 2; ++b2)
                tma_load_2d(obuf + oslot * kOHalfBytes + b2 * (kOHalfBytes / 2), &map_o, ofull,
                            t.nt * 128 + half * 64 + b2 * 32, t.tn * p.bn);
            } else if (p.accumulate) {
              mbar_arrive_expect_tx(ofull, (uint32_t)p.o_bytes);
              tma_load_3d(obuf + oslot * kOHalfBytes, &map_o, ofull, t.th * p.bh * p.d.wo,
                          t.nt * 128 + half * 64, t.tn * p.bn);
            } else {
              mbar_arrive(ofull);
            }
            if (++oslot == kOSlots) { oslot = 0; ophase ^= 1u; }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    // All lanes walk the loop (descriptors and addresses stay warp-uniform values); one
    // elected lane issues the MMAs and commits.
    {
      const uint32_t idesc = make_idesc_i8(kTileM, p.umma_n);
      int stage = 0;
      uint32_t phase = 0;
      int buf = 0;
      uint32_t bphase = 0;
      bool ok = true;
      for (int tile = tile_first; tile < p.total_tiles; tile += tile_step) {
        ok = mbar_wait(smem_u32(&bar_tmem_empty[buf]), bphase ^ 1u, abort_flag);
        if (!ok) break;
        tc_fence_after();
        for (int seg = 0; seg < p.nseg; ++seg) {
          const uint32_t d_tmem = tmem_base + (uint32_t)(buf * p.buf_cols + seg * p.umma_n);
          const int iters = KSPLIT ? it_hi - it_lo : (seg == 0 ? k_iters_seg0 : k_iters_seg1);
          for (int it = 0; it < iters; ++it) {
            ok = mbar_wait(smem_u32(&bar_full[stage]), phase, abort_flag);
            if (!ok) break;
            tc_fence_after();
            const uint32_t a_src = ring + stage * stage_bytes;
            const uint64_t adesc = make_smem_desc(a_src);
            const uint64_t bdesc = make_smem_desc(a_src + kATileBytes);
            if (elect_one()) {
#pragma unroll
              for (int k = 0; k < kChunkK / 32; ++k) {
                // advancing K by 32 bytes inside the swizzle atom = +2 in the address field
                tc_mma_i8(d_tmem, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc,
                          (it > 0 || k > 0) ? 1u : 0u);
              }
              tc_commit(smem_u32(&bar_empty[stage]));
            }
            __syncwarp();
            if (++stage == p.stages) { stage = 0; phase ^= 1u; }
          }
          if (!ok) break;
        }
        if (!ok) break;
        if (elect_one()) tc_commit(smem_u32(&bar_tmem_full[buf]));
        __syncwarp();
        if (++buf == p.nbuf) { buf = 0; bphase ^= 1u; }
      }
    }
  } else if (warp == kStoreWarp) {
    // ------------------------------------------------------------ cached-output store warp
    // Token-major layers: writes each finished half tile back with bulk tensor stores and hands the
    // ring slot to the producer as soon as the stores have read shared memory.
    if (TMA_EPI && p.row_epi && lane == 0) {
      int oslot = 0;
      uint32_t ophase = 0;
      bool ok = true;
      for (int tile = tile_first; tile < p.total_tiles && ok; tile += tile_step) {
        const TileCoord t = decode_tile(tile, p);
        for (int hh = 0; hh < 2; ++hh) {
          ok = mbar_wait(smem_u32(&bar_o_ready[oslot]), ophase, abort_flag);
          if (!ok) break;
          for (int b2 = 0; b2 < 2; ++b2)
            tma_store_2d(&map_o, obuf + oslot * kOHalfBytes + b2 * (kOHalfBytes / 2),
                         t.nt * 128 + hh * 64 + b2 * 32, t.tn * p.bn);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          mbar_arrive(smem_u32(&bar_o_empty[oslot]));
          if (++oslot == kOSlots) { oslot = 0; ophase ^= 1u; }
        }
      }
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9)
    // Two warps share each tensor-memory lane quarter; each takes 64 of the 128 columns.
    const int quarter = warp & 3;           // lane quarter this warp may read
    const int half = (warp - 2) >> 2;       // which 64 columns this warp handles
    const int ep_tid = threadIdx.x - 64;    // 0..255
    const int row = quarter * 32 + lane;    // accumulator row = output pixel of the tile
    const size_t M = (size_t)p.g.batch * howo;
    const int tile_px = p.bh * p.bw;        // pixels per image in one tile
    const int ni = row / tile_px;
    const int pl = row % tile_px;           // pixel index inside the image's part of the tile
    const int hi = pl / p.bw;
    const int wi = pl % p.bw;
    const int col0 = half * 64;
    int buf = 0;
    uint32_t bphase = 0;
    uint32_t ophase = 0;
    int oslot = 0;
    int last_nt = -1;
    bool ok = true;
    for (int tile = tile_first; tile < p.total_tiles; tile += tile_step) {
      const TileCoord t = decode_tile(tile, p);
      // per-tile channel parameters (only when the channel tile changes)
      if (t.nt != last_nt) {
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (ep_tid < 128) {
          const int co = t.nt * 128 + ep_tid;
          const bool cv = co < p.g.cout;
          for (int seg = 0; seg < NSEG; ++seg) {
            float sc = cv ? p.w_scale[seg * p.g.cout + co] : 0.0f;
            if (TMA_EPI) sc = __fmul_rn(p.x_scale[seg], sc);
            ep_scale[seg][ep_tid] = sc;
            ep_corr[seg][ep_tid] = (cv && p.w_corr) ? p.w_corr[seg * p.g.cout + co] : 0;
            // codes stored as q - 128: (zp - 128) * sum of the channel's centred weights comes
            // back out of the integer accumulator
            ep_off[seg][ep_tid] = (cv && p.x_zp)
                ? -((int)p.x_zp[seg] - 128) * p.w_csum[seg * p.g.cout + co] : 0;
          }
          ep_bias[ep_tid] = (cv && p.bias) ? p.bias[co] : 0.0f;
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        last_nt = t.nt;
      }

      if (ok) ok = mbar_wait(smem_u32(&bar_tmem_full[buf]), bphase, abort_flag);
      if (!ok) continue;               // on to the next tile's barriers
      tc_fence_after();
      const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * p.buf_cols);
      int rsum[2] = {0, 0};
      const bool offset_codes = p.x_zp != nullptr;
      if (WITH_SUM) {
#pragma unroll
        for (int seg = 0; seg < NSEG; ++seg) tc_ld1(t_row + seg * p.umma_n + 128, rsum[seg]);
        tc_wait_ld();
      }

      if (TMA_EPI) {
        // Each half tile (64 channels) sits in one ring slot as [image][channel][pixel]; lanes
        // walk consecutive pixels.  The two warps of a lane quarter take 32 channels each.
        const int sub = (warp - 2) >> 2;          // 0 / 1: which 32 channels of the half
        for (int hh = 0; hh < 2; ++hh) {
          ok = mbar_wait(smem_u32(&bar_o_full[oslot]), ophase, abort_flag);
          if (!ok) break;
          float* orow = obuf_ptr + (size_t)oslot * (kOHalfBytes / 4) + (size_t)ni * 64 * tile_px +
                        (size_t)(sub * 32) * tile_px + pl;
          const int colbase = hh * 64 + sub * 32;
          // token-major layers: this warp's box is 128 rows x 32 channels, a row = 128 bytes whose
          // 16-byte chunks are XORed with row % 8 (the 128-byte swizzle of the tensor copy), so the
          // eight lanes of a quarter-warp touch eight different bank groups
          uint8_t* rbox = reinterpret_cast<uint8_t*>(obuf_ptr) + (size_t)oslot * kOHalfBytes +
                          (size_t)sub * (kOHalfBytes / 2) + (size_t)row * 128;
          float v[32];
          if (p.row_epi) {
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4) {
              float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
              if (p.accumulate) f = *reinterpret_cast<const float4*>(rbox + ((j4 ^ (row & 7)) << 4));
              v[4 * j4] = f.x; v[4 * j4 + 1] = f.y; v[4 * j4 + 2] = f.z; v[4 * j4 + 3] = f.w;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = p.accumulate ? orow[j * tile_px] : 0.0f;
            // the slot has been read: new values go to memory straight from registers (a lane is a
            // pixel, so a warp writes runs of consecutive pixels per channel)
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_o_empty[oslot]));
          }
#pragma unroll
          for (int seg = 0; seg < NSEG; ++seg) {
            int a[32];
            tc_ld32(t_row + seg * p.umma_n + colbase, a);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              int iv = a[j];
              if (WITH_SUM) iv += ep_corr[seg][colbase + j] * rsum[seg];
              if (offset_codes) iv += ep_off[seg][colbase + j];
              v[j] = fmaf((float)iv, ep_scale[seg][colbase + j], v[j]);
            }
          }
          if (p.row_epi) {
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4)
              *reinterpret_cast<float4*>(rbox + ((j4 ^ (row & 7)) << 4)) =
                  make_float4(v[4 * j4], v[4 * j4 + 1], v[4 * j4 + 2], v[4 * j4 + 3]);
            // make the tile visible to the bulk-copy engine, then tell the store warp
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          } else {
            const int n = t.tn * p.bn + ni;
            const int co0 = t.nt * 128 + colbase;
            if (n < p.g.batch) {
              float* obase = p.o_hat + ((size_t)n * p.g.cout + co0) * howo + t.th * p.bh * p.d.wo + pl;
              if (co0 + 32 <= p.g.cout) {
#pragma unroll
                for (int j = 0; j < 32; ++j) obase[(size_t)j * howo] = v[j];
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (co0 + j < p.g.cout) obase[(size_t)j * howo] = v[j];
              }
            }
          }
          if (hh == 1) tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if (p.row_epi) mbar_arrive(smem_u32(&bar_o_ready[oslot]));
            if (hh == 1) mbar_arrive(smem_u32(&bar_tmem_empty[buf]));   // accumulators consumed
          }
          if (++oslot == kOSlots) { oslot = 0; ophase ^= 1u; }
        }
        if (!ok) continue;
      } else if (KSPLIT) {
        // partial sums of this CTA's K range -> its own shared memory as [column][row] (the tile
        // ring is idle: every product that read it has completed); column 128 = the sum row
        int32_t* part = reinterpret_cast<int32_t*>(smem_raw);
#pragma unroll 1
        for (int c2 = 0; c2 < 2; ++c2) {
          int a[32];
          tc_ld32(t_row + col0 + c2 * 32, a);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) part[(col0 + c2 * 32 + j) * 128 + row] = a[j];
        }
        if (WITH_SUM && half == 0) part[128 * 128 + row] = rsum[0];
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_tmem_empty[buf]));
      } else {
        const int n = t.tn * p.bn + ni;
        const int hw = (t.th * p.bh + hi) * p.d.wo + (t.tw * p.bw + wi);
        const bool valid = n < p.g.batch;
        const size_t m = (size_t)n * howo + hw;
        float xs[2];
        xs[0] = p.per_sample ? (valid ? p.x_scale[n] : 0.0f) : p.x_scale[0];
        xs[1] = (NSEG == 2) ? p.x_scale[1] : 0.0f;
#pragma unroll 1
        for (int c2 = 0; c2 < 2; ++c2) {
          const int co0 = t.nt * 128 + col0 + c2 * 32;
          const int ncols = min(32, p.g.cout - co0);   // <= 0 on a ragged last tile
          float* obase = p.o_hat + ((size_t)n * p.g.cout + co0) * howo + hw;
          // linear layers (one pixel per row): a thread's 32 channels are 128 contiguous bytes
          const bool row_vec = (howo == 1) && (ncols == 32) && ((p.g.cout & 3) == 0) &&
                               ((reinterpret_cast<uintptr_t>(p.o_hat) & 15) == 0);
          float v[32];
          if (row_vec) {
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4) {
              float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
              if (p.accumulate && valid) f = *reinterpret_cast<const float4*>(obase + 4 * j4);
              v[4 * j4] = f.x; v[4 * j4 + 1] = f.y; v[4 * j4 + 2] = f.z; v[4 * j4 + 3] = f.w;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              v[j] = (p.accumulate && valid && j < ncols) ? obase[(size_t)j * howo] : 0.0f;
          }
#pragma unroll
          for (int seg = 0; seg < NSEG; ++seg) {
            int a[32];
            tc_ld32(t_row + seg * p.umma_n + col0 + c2 * 32, a);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const int cl = col0 + c2 * 32 + j;
              int iv = a[j];
              if (WITH_SUM) iv += ep_corr[seg][cl] * rsum[seg];
              if (offset_codes) iv += ep_off[seg][cl];
              v[j] += (float)iv * __fmul_rn(xs[seg], ep_scale[seg][cl]);
              if (p.acc_out && valid && j < ncols)
                p.acc_out[((size_t)seg * M + m) * p.g.cout + co0 + j] = iv;
            }
          }
          if (valid && row_vec) {
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4) {
              const int cb = col0 + c2 * 32 + 4 * j4;
              *reinterpret_cast<float4*>(obase + 4 * j4) =
                  make_float4(v[4 * j4] + ep_bias[cb], v[4 * j4 + 1] + ep_bias[cb + 1],
                              v[4 * j4 + 2] + ep_bias[cb + 2], v[4 * j4 + 3] + ep_bias[cb + 3]);
            }
          } else if (valid) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j < ncols) obase[(size_t)j * howo] = v[j] + ep_bias[col0 + c2 * 32 + j];
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_tmem_empty[buf]));
      }
      if (++buf == p.nbuf) { buf = 0; bphase ^= 1u; }
    }
  }

  if (KSPLIT) {
    __syncwarp();
    cluster_sync_all();          // every CTA's partial sums are in its shared memory
    if (warp >= 2 && warp < 2 + kEpiWarps && tile_first < p.total_tiles && !abort_sh) {
      const TileCoord t = decode_tile(tile_first, p);
      const int ep_tid = threadIdx.x - 64;
      const int row = ep_tid & 127;
      const int cols_cta = 128 / p.ksplit;             // output channels this CTA finishes
      const int cpt = cols_cta / 2;                    // ... and each of its threads
      const int cbase = krank * cols_cta + (ep_tid >> 7) * cpt;
      const int tile_px = p.bh * p.bw;
      const int ni = row / tile_px, pl = row % tile_px;
      const int n = t.tn * p.bn + ni;
      const int hw = (t.th * p.bh + pl / p.bw) * p.d.wo + (t.tw * p.bw + pl % p.bw);
      const bool valid = n < p.g.batch;
      const size_t m = (size_t)n * howo + hw;
      const float xs = p.per_sample ? (valid ? p.x_scale[n] : 0.0f) : p.x_scale[0];
      const bool offset_codes = p.x_zp != nullptr;
      uint32_t peer[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) peer[r] = map_to_cta(raw, (uint32_t)(r < p.ksplit ? r : 0));
      int rs = 0;
      if (WITH_SUM) {
#pragma unroll
        for (int r = 0; r < 8; ++r)
          if (r < p.ksplit) rs += ld_cluster_s32(peer[r] + (uint32_t)(128 * 128 + row) * 4u);
      }
      // eight channels at a time: all loads of a group (cached output, every CTA's partial
      // sums) are issued before the first use
      for (int j0 = 0; j0 < cpt; j0 += 8) {
        float old[8];
        int iv[8];
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
          const int co = t.nt * 128 + cbase + j0 + jj;
          old[jj] = (p.accumulate && valid && co < p.g.cout)
                        ? p.o_hat[((size_t)n * p.g.cout + co) * howo + hw] : 0.0f;
          iv[jj] = 0;
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          if (r < p.ksplit) {
#pragma unroll
            for (int jj = 0; jj < 8; ++jj)
              iv[jj] += ld_cluster_s32(peer[r] + (uint32_t)((cbase + j0 + jj) * 128 + row) * 4u);
          }
        }
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
          const int cl = cbase + j0 + jj;
          const int co = t.nt * 128 + cl;
          int a = iv[jj];
          if (WITH_SUM) a += ep_corr[0][cl] * rs;
          if (offset_codes) a += ep_off[0][cl];
          if (valid && co < p.g.cout) {
            const float sc = __fmul_rn(xs, ep_scale[0][cl]);
            // the rounding of the unsplit kernel's epilogue that this layer would have taken:
            // one fused multiply-add (bulk-copy epilogue) or product, sum, bias (generic)
            const float v = p.fused_round ? fmaf((float)a, sc, old[jj])
                                          : __fadd_rn(__fadd_rn(__fmul_rn((float)a, sc), old[jj]),
                                                      ep_bias[cl]);
            p.o_hat[((size_t)n * p.g.cout + co) * howo + hw] = v;
            if (p.acc_out) p.acc_out[m * p.g.cout + co] = a;
          }
        }
      }
    }
  }

  // ---------------------------------------------------------------- teardown
  __syncwarp();
  if (abort_sh) {
    // give copies that may still be in flight time to land before the CTA retires
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  tc_fence_before();
  __syncthreads();
  if (KSPLIT) cluster_sync_all();   // peers may still be reading this CTA's partial sums
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"((uint32_t)p.tmem_cols)
                 : "memory");
  }
}

// ---------------------------------------------------------------- host side
bool is_pow2(int v) { return v > 0 && (v & (v - 1)) == 0; }

}  // namespace

// Whether the tensor-core kernel covers this geometry; the message says why not.
bool tc_supported(const modiff_conv_geom* g, int per_sample, const char** why) {
  Derived d = derive(*g);
  static const char* msgs[] = {"cin < 128", "output width/height not a power of two <= 128",
                               "split not a multiple of 128", "cin not a multiple of 16",
                               "kernel larger than 7x7"};
  if (g->cin < 128) { *why = msgs[0]; return false; }
  if (g->cin % 16) { *why = msgs[3]; return false; }
  if (!is_pow2(d.wo) || !is_pow2(d.ho) || d.wo > 128) { *why = msgs[1]; return false; }
  if (g->split % 128) { *why = msgs[2]; return false; }
  if (g->kh > 7 || g->kw > 7) { *why = msgs[4]; return false; }
  (void)per_sample;
  return true;
}

int launch_igemm_tc(const int8_t* codes, const int8_t* wcodes, int with_sum_rows,
                    const float* x_scale, const float* w_scale, const int32_t* w_corr,
                    float* o_hat, int accumulate, const float* bias, const modiff_conv_geom* g,
                    int per_sample, int32_t* acc_out, cudaStream_t s, const float* x_zp,
                    const int32_t* w_csum) {
  EncodeTiledFn encode = get_encode_fn();
  if (!encode) return set_error(MODIFF_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is not available");
  MODIFF_CHECK_ARG(w_corr == nullptr || with_sum_rows,
                   "w_corr given but the weight codes were packed without sum rows");
  Derived d = derive(*g);
  TcParams p;
  p.g = *g;
  p.d = d;
  p.bw = d.wo < 128 ? d.wo : 128;
  p.bh = (d.ho < 128 / p.bw) ? d.ho : 128 / p.bw;
  p.bn = 128 / (p.bw * p.bh);
  p.tiles_w = d.wo / p.bw;
  p.tiles_h = d.ho / p.bh;
  p.tiles_n = ceil_div(g->batch, p.bn);
  p.n_tiles = ceil_div(g->cout, 128);
  p.total_tiles = p.tiles_w * p.tiles_h * p.tiles_n * p.n_tiles;
  p.with_sum = with_sum_rows ? 1 : 0;
  p.umma_n = with_sum_rows ? 144 : 128;
  p.nseg = d.nseg;
  p.buf_cols = p.nseg * p.umma_n;
  p.nbuf = (2 * p.buf_cols <= 512) ? 2 : 1;
  int cols = p.nbuf * p.buf_cols;
  p.tmem_cols = 32;
  while (p.tmem_cols < cols) p.tmem_cols *= 2;
  p.cbeg[0] = 0;
  p.cbeg[1] = g->split;
  const int c_seg0 = p.nseg == 2 ? g->split : g->cin;
  p.chunks[0] = ceil_div(c_seg0, kChunkK);
  p.chunks[1] = p.nseg == 2 ? ceil_div(g->cin - g->split, kChunkK) : 0;
  p.accumulate = accumulate;
  p.per_sample = per_sample;
  p.x_scale = x_scale;
  p.w_scale = w_scale;
  p.w_corr = w_corr;
  p.x_zp = x_zp;
  p.w_csum = w_csum;
  p.bias = bias;
  p.o_hat = o_hat;
  p.acc_out = acc_out;

  static int sm_count = 0;
  if (!sm_count) {
    int dev = 0;
    MODIFF_CUDA(cudaGetDevice(&dev));
    MODIFF_CUDA(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev));
  }
  // The bulk-copy epilogue needs full-width row tiles of at least 4 pixels per image, per-tensor
  // scales, no bias and no accumulator dump.
  const int tile_px = p.bh * p.bw;
  // Linear layers (one pixel per row, output [rows][cout]): the same ring, filled and drained by
  // 2-D copies of 128 rows x 32 channels with the 128-byte swizzle.
  const bool row_epi_u = !per_sample && !bias && !acc_out && d.ho * d.wo == 1 && g->cout % 4 == 0 &&
                         g->batch >= 128 && (((uintptr_t)o_hat & 15) == 0);
  const bool tma_epi_u = row_epi_u ||
                         (!per_sample && !bias && !acc_out && tile_px >= 4 && p.bw == d.wo &&
                          (d.ho * d.wo) % 4 == 0 && (((uintptr_t)o_hat & 15) == 0));
  // Few tiles and a long K range: clusters of 2 / 4 / 8 CTAs share each tile's K iterations, as
  // long as the grid still fits the SMs at once and every CTA keeps at least three iterations.
  p.ksplit = 1;
  {
    const char* e = getenv("MODIFF_TC_KSPLIT");     // 1 switches the split off (tests compare)
    const int allow = e ? atoi(e) : 8;
    const int iters = d.taps * p.chunks[0];
    // (token-major layers keep the bulk-copy epilogue: a split one's touches 4 bytes of a row at a time.
    // Where the rule below would split them, us whole / split: 5120 -> 1280 of 128 rows 16.4 / 19.4, 256
    // rows 16.7 / 20.4, 308 rows 16.9 / 22.2, 512 rows 16.9 / 29.1; 4096 -> 4096 of 128 rows 14.7 / 20.5.  Below 128
    // rows there is no such epilogue and the split stays: 64 rows, 5120 -> 1280 19.3 / 16.4.)
    if (p.nseg == 1 && !row_epi_u)
      while (p.ksplit * 2 <= allow && p.ksplit < 8 && p.total_tiles * p.ksplit * 2 <= sm_count &&
             iters >= 6 * p.ksplit * 2)
        p.ksplit *= 2;
    // the cluster's barriers and the exchange of partial sums cost about what 20 K iterations do
    if (iters * (p.ksplit - 1) < 20 * p.ksplit) p.ksplit = 1;
  }

  // what the layer would take without the K split decides how the split epilogue rounds
  p.fused_round = (row_epi_u || (tma_epi_u && g->cout >= 128)) ? 1 : 0;
  const bool row_epi = row_epi_u && p.ksplit == 1;
  const bool tma_epi = tma_epi_u && p.ksplit == 1;
  p.row_epi = row_epi ? 1 : 0;
  const uint32_t b_tile = ((uint32_t)p.umma_n * kChunkK + 1023u) & ~1023u;
  const uint32_t stage_bytes = kATileBytes + b_tile;
  const uint32_t o_ring = tma_epi ? (uint32_t)kOSlots * kOHalfBytes : 0u;
  p.stages = (int)((224u * 1024u - o_ring) / stage_bytes);
  if (p.stages > kMaxStages) p.stages = kMaxStages;
  const size_t smem = (size_t)p.stages * stage_bytes + o_ring;

  // Activation codes: [batch][planes][hp][wp][cp] int8, innermost first.
  CUtensorMap map_a, map_b;
  {
    cuuint64_t dims[5] = {(cuuint64_t)d.cp, (cuuint64_t)d.wp, (cuuint64_t)d.hp,
                          (cuuint64_t)d.nplanes, (cuuint64_t)g->batch};
    cuuint64_t strides[4] = {(cuuint64_t)d.cp, (cuuint64_t)d.wp * d.cp,
                             (cuuint64_t)d.hp * d.wp * d.cp,
                             (cuuint64_t)d.nplanes * d.hp * d.wp * d.cp};
    // The image extent of the box never exceeds the batch; rows of the tile that no copy
    // fills belong to images >= batch and are masked in the epilogue.
    const int bn_box = p.bn < g->batch ? p.bn : g->batch;
    p.a_bytes = kChunkK * p.bw * p.bh * bn_box;
    cuuint32_t box[5] = {(cuuint32_t)kChunkK, (cuuint32_t)p.bw, (cuuint32_t)p.bh, 1u,
                         (cuuint32_t)bn_box};
    cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    CUresult r = encode(&map_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, (void*)codes, dims, strides, box,
                        estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
      return set_error(MODIFF_ERR_CUDA, "cuTensorMapEncodeTiled(activation codes) failed: %d", (int)r);
  }
  {
    const int rows = modiff_wcodes_rows(g, with_sum_rows);
    cuuint64_t dims[2] = {(cuuint64_t)d.taps * d.kp, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)d.taps * d.kp};
    cuuint32_t box[2] = {(cuuint32_t)kChunkK, (cuuint32_t)p.umma_n};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode(&map_b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)wcodes, dims, strides, box,
                        estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
      return set_error(MODIFF_ERR_CUDA, "cuTensorMapEncodeTiled(weight codes) failed: %d", (int)r);
  }

  CUtensorMap map_o = map_b;   // placeholder when the bulk-copy epilogue is off
  p.o_bytes = 0;
  if (row_epi) {
    // Cached output of a linear layer: [rows][cout] fp32; boxes of 128 rows x 32 channels.
    // Channels and rows beyond the tensor are filled with zeros on the way in and dropped on
    // the way out, so ragged channel counts and row counts need no special case.
    cuuint64_t dims[2] = {(cuuint64_t)g->cout, (cuuint64_t)g->batch};
    cuuint64_t strides[1] = {(cuuint64_t)g->cout * 4};
    cuuint32_t box[2] = {32u, 128u};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode(&map_o, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)o_hat, dims, strides, box,
                        estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
      return set_error(MODIFF_ERR_CUDA, "cuTensorMapEncodeTiled(cached output rows) failed: %d", (int)r);
    p.o_bytes = kOHalfBytes;
  } else if (tma_epi) {
    // Cached output: [batch][cout][ho*wo] fp32, innermost first.
    const int bn_box = p.bn < g->batch ? p.bn : g->batch;
    const int c_box = g->cout < 128 ? g->cout : 128;
    cuuint64_t dims[3] = {(cuuint64_t)(d.ho * d.wo), (cuuint64_t)g->cout, (cuuint64_t)g->batch};
    cuuint64_t strides[2] = {(cuuint64_t)d.ho * d.wo * 4, (cuuint64_t)g->cout * d.ho * d.wo * 4};
    cuuint32_t box[3] = {(cuuint32_t)tile_px, 64u, (cuuint32_t)bn_box};
    cuuint32_t estr[3] = {1, 1, 1};
    // the shared-memory tile is addressed as [image][128][tile_px]: boxes narrower than 128
    // channels would change that pitch, so they use the generic epilogue instead
    if (c_box == 128) {
      CUresult r = encode(&map_o, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void*)o_hat, dims, strides,
                          box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
      if (r != CUDA_SUCCESS)
        return set_error(MODIFF_ERR_CUDA, "cuTensorMapEncodeTiled(cached output) failed: %d", (int)r);
      p.o_bytes = tile_px * 64 * bn_box * 4;
    }
  }
  const bool use_tma_epi = tma_epi && p.o_bytes > 0;

  if (p.ksplit > 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.total_tiles * p.ksplit));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.ksplit;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (p.with_sum) {
      static SmemLimit smem_limit;
      MODIFF_CUDA(raise_smem_limit(igemm_tc_kernel<1, true, false, true>, smem, smem_limit));
      MODIFF_CUDA(cudaLaunchKernelEx(&cfg, igemm_tc_kernel<1, true, false, true>, map_a, map_b,
                                     map_o, p));
    } else {
      static SmemLimit smem_limit;
      MODIFF_CUDA(raise_smem_limit(igemm_tc_kernel<1, false, false, true>, smem, smem_limit));
      MODIFF_CUDA(cudaLaunchKernelEx(&cfg, igemm_tc_kernel<1, false, false, true>, map_a, map_b,
                                     map_o, p));
    }
    MODIFF_LAUNCH_CHECK("igemm_tc_kernel (K split across a cluster)");
    return MODIFF_OK;
  }
  const int grid = p.total_tiles < sm_count ? p.total_tiles : sm_count;
  const int variant = (p.nseg == 2 ? 4 : 0) | (p.with_sum ? 2 : 0) | (use_tma_epi ? 1 : 0);
#define MODIFF_TC_LAUNCH(NSEG, SUM, EPI)                                                       \
  {                                                                                            \
    static SmemLimit smem_limit;                                                               \
    MODIFF_CUDA(raise_smem_limit(igemm_tc_kernel<NSEG, SUM, EPI>, smem, smem_limit));          \
    igemm_tc_kernel<NSEG, SUM, EPI><<<grid, kThreads, smem, s>>>(map_a, map_b, map_o, p);      \
  }
  switch (variant) {
    case 0: MODIFF_TC_LAUNCH(1, false, false) break;
    case 1: MODIFF_TC_LAUNCH(1, false, true) break;
    case 2: MODIFF_TC_LAUNCH(1, true, false) break;
    case 3: MODIFF_TC_LAUNCH(1, true, true) break;
    case 4: MODIFF_TC_LAUNCH(2, false, false) break;
    case 5: MODIFF_TC_LAUNCH(2, false, true) break;
    case 6: MODIFF_TC_LAUNCH(2, true, false) break;
    default: MODIFF_TC_LAUNCH(2, true, true) break;
  }
#undef MODIFF_TC_LAUNCH
  MODIFF_LAUNCH_CHECK("igemm_tc_kernel");
  return MODIFF_OK;
}

int read_device_status_bf16(int* status, int reset);   // gemm_bf16_tc.cu
int read_device_status_halo(int* status, int reset);   // igemm_halo.cu
int read_device_status_attention(int* status, int reset);   // attention_tc.cu
int read_device_status_modq(int* status, int reset);        // modq.cu
int read_device_status_probe(int* status, int reset);       // i8_probe.cu
int read_device_status_pair(int* status, int reset);        // igemm_pair.cu
int read_device_status_attention_i8(int* status, int reset);   // attention_i8.cu
int read_device_status_conv_f32(int* status, int reset);       // conv_f32_tc.cu
bool pair_supported(const modiff_conv_geom* g, int with_sum_rows, int per_sample, const float* bias,
                    const int32_t* acc_out, const float* o_hat);
int launch_igemm_pair(const int8_t* codes, const int8_t* wcodes, int with_sum_rows,
                      const float* x_scale, const float* w_scale, const int32_t* w_corr,
                      float* o_hat, int accumulate, const modiff_conv_geom* g, cudaStream_t s,
                      const float* residual, float* sum_out, const float* x_zp,
                      const int32_t* w_csum);
bool halo_supported(const modiff_conv_geom* g, int with_sum_rows, int per_sample, const float* bias,
                    const int32_t* acc_out, const float* o_hat);
int launch_igemm_halo(const int8_t* codes, const int8_t* wcodes, int with_sum_rows,
                      const float* x_scale, const float* w_scale, const int32_t* w_corr,
                      float* o_hat, int accumulate, const modiff_conv_geom* g, cudaStream_t s,
                      const float* residual, float* sum_out, const float* x_zp,
                      const int32_t* w_csum, const float* packed_w_zp);

// MODIFF_IGEMM_PAIR=1 sends 3x3 layers to the two-SM kernel (cta_group::2, igemm_pair.cu): same
// results, measured slower than the single-CTA kernel at every layer of the covered models, so
// it is off unless asked for
static bool pair_enabled() {
  const char* e = getenv("MODIFF_IGEMM_PAIR");   // read per call: tests switch it at run time
  return e && e[0] == '1';
}

// MODIFF_IGEMM_HALO=0 keeps 3x3 layers on the one-copy-per-tap kernel (debug aid, same results)
static bool halo_enabled() {
  const char* e = getenv("MODIFF_IGEMM_HALO");   // read per call: tests switch it at run time
  return !(e && e[0] == '0');
}

int read_device_status(int* status, int reset) {
  int a = 0, b = 0, c = 0;
  int rc = read_status_this_unit(&a, reset);
  if (rc) return rc;
  rc = read_device_status_bf16(&b, reset);
  if (rc) return rc;
  rc = read_device_status_halo(&c, reset);
  if (rc) return rc;
  int d = 0;
  rc = read_device_status_attention(&d, reset);
  if (rc) return rc;
  int e = 0;
  rc = read_device_status_modq(&e, reset);
  if (rc) return rc;
  int f = 0;
  rc = read_device_status_probe(&f, reset);
  if (rc) return rc;
  int h = 0;
  rc = read_device_status_pair(&h, reset);
  if (rc) return rc;
  int i8 = 0;
  rc = read_device_status_attention_i8(&i8, reset);
  if (rc) return rc;
  int f32 = 0;
  rc = read_device_status_conv_f32(&f32, reset);
  if (rc) return rc;
  *status = a | b | c | d | e | f | h | i8 | f32;
  return MODIFF_OK;
}

}  // namespace modiff

using namespace modiff;

static int igemm_conv_impl(const int8_t* codes, const int8_t* wcodes, int with_sum_rows,
                           const float* x_scale, const float* w_scale, const int32_t* w_corr,
                           float* o_hat, int accumulate, const float* bias,
                           const modiff_conv_geom* g, int per_sample, int impl, int32_t* acc_out,
                           const float* residual, float* sum_out, const float* x_zp,
                           const int32_t* w_csum, void* stream) {
  int rc = validate_geom(g);
  if (rc) return rc;
  MODIFF_CHECK_ARG(codes && wcodes && x_scale && w_scale && o_hat, "NULL pointer argument");
  MODIFF_CHECK_ARG((((uintptr_t)codes | (uintptr_t)wcodes) & 15) == 0,
                   "code buffers must be 16-byte aligned");
  MODIFF_CHECK_ARG(!(per_sample && g->split > 0), "per-sample scales cannot be combined with split");
  MODIFF_CHECK_ARG((x_zp == nullptr) == (w_csum == nullptr), "x_zp and w_csum go together");
  MODIFF_CHECK_ARG(!(x_zp && per_sample), "offset codes have one zero point per scale segment");
  cudaStream_t s = (cudaStream_t)stream;
  const char* why = "";
  const bool tc_ok = tc_supported(g, per_sample, &why);
  if (impl == MODIFF_IMPL_TCGEN05 && !tc_ok)
    return set_error(MODIFF_ERR_UNSUPPORTED, "tcgen05 path does not cover this layer: %s", why);
  if (impl == MODIFF_IMPL_SIMT || !tc_ok) {
    const int rc1 = launch_igemm_simt(codes, wcodes, with_sum_rows, x_scale, w_scale, w_corr, o_hat,
                                      accumulate, bias, g, per_sample, acc_out, s, x_zp, w_csum);
    if (rc1 || !residual) return rc1;
    const Derived ds = derive(*g);
    return modiff_add(residual, o_hat, sum_out, g->batch, g->cout, ds.ho * ds.wo, 0, stream);
  }
  MODIFF_CHECK_ARG(impl == MODIFF_IMPL_AUTO || impl == MODIFF_IMPL_TCGEN05, "unknown impl %d", impl);
  if (pair_enabled() && halo_enabled() &&
      pair_supported(g, with_sum_rows, per_sample, bias, acc_out, o_hat))
    return launch_igemm_pair(codes, wcodes, with_sum_rows, x_scale, w_scale, w_corr, o_hat, accumulate,
                             g, s, residual, sum_out, x_zp, w_csum);
  if (halo_enabled() && halo_supported(g, with_sum_rows, per_sample, bias, acc_out, o_hat))
    return launch_igemm_halo(codes, wcodes, with_sum_rows, x_scale, w_scale, w_corr, o_hat, accumulate,
                             g, s, residual, sum_out, x_zp, w_csum, nullptr);
  int rc2 = launch_igemm_tc(codes, wcodes, with_sum_rows, x_scale, w_scale, w_corr, o_hat, accumulate,
                            bias, g, per_sample, acc_out, s, x_zp, w_csum);
  if (rc2 || !residual) return rc2;
  const Derived dd = derive(*g);
  return modiff_add(residual, o_hat, sum_out, g->batch, g->cout, dd.ho * dd.wo, 0, stream);
}

extern "C" int modiff_igemm_conv(const int8_t* codes, const int8_t* wcodes, int with_sum_rows,
                                 const float* x_scale, const float* w_scale,
                                 const int32_t* w_corr, float* o_hat, int accumulate,
                                 const float* bias, const modiff_conv_geom* g, int per_sample,
                                 int impl, int32_t* acc_out, void* stream) {
  return igemm_conv_impl(codes, wcodes, with_sum_rows, x_scale, w_scale, w_corr, o_hat, accumulate,
                         bias, g, per_sample, impl, acc_out, nullptr, nullptr, nullptr, nullptr,
                         stream);
}

extern "C" int modiff_igemm_conv_add(const int8_t* codes, const int8_t* wcodes, int with_sum_rows,
                                     const float* x_scale, const float* w_scale,
                                     const int32_t* w_corr, float* o_hat, int accumulate,
                                     const modiff_conv_geom* g, int impl, const float* residual,
                                     float* sum_out, void* stream) {
  MODIFF_CHECK_ARG(residual && sum_out, "NULL pointer argument");
  MODIFF_CHECK_ARG((((uintptr_t)residual | (uintptr_t)sum_out) & 15) == 0,
                   "residual and sum must be 16-byte aligned");
  return igemm_conv_impl(codes, wcodes, with_sum_rows, x_scale, w_scale, w_corr, o_hat, accumulate,
                         nullptr, g, 0, impl, nullptr, residual, sum_out, nullptr, nullptr, stream);
}

extern "C" int modiff_igemm_conv_offset(const int8_t* codes, const int8_t* wcodes, int with_sum_rows,
                                        const float* x_scale, const float* x_zp,
                                        const float* w_scale, const int32_t* w_corr,
                                        const int32_t* w_csum, float* o_hat, int accumulate,
                                        const float* bias, const modiff_conv_geom* g, int impl,
                                        const float* residual, float* sum_out, void* stream) {
  MODIFF_CHECK_ARG(x_zp && w_csum, "NULL pointer argument");
  MODIFF_CHECK_ARG((residual == nullptr) == (sum_out == nullptr), "residual and sum go together");
  MODIFF_CHECK_ARG((((uintptr_t)residual | (uintptr_t)sum_out) & 15) == 0,
                   "residual and sum must be 16-byte aligned");
  return igemm_conv_impl(codes, wcodes, with_sum_rows, x_scale, w_scale, w_corr, o_hat, accumulate,
                         bias, g, 0, impl, nullptr, residual, sum_out, x_zp, w_csum, stream);
}

extern "C" int modiff_igemm_conv_packed4(const uint8_t* codes4, const uint8_t* wcodes4,
                                         const float* w_zp, const float* x_scale,
                                         const float* w_scale, float* o_hat, int accumulate,
                                         const modiff_conv_geom* g, const float* residual,
                                         float* sum_out, void* stream) {
  int rc = validate_geom(g);
  if (rc) return rc;
  MODIFF_CHECK_ARG(codes4 && wcodes4 && w_zp && x_scale && w_scale && o_hat, "NULL pointer argument");
  MODIFF_CHECK_ARG((((uintptr_t)codes4 | (uintptr_t)wcodes4) & 15) == 0,
                   "code buffers must be 16-byte aligned");
  MODIFF_CHECK_ARG((residual == nullptr) == (sum_out == nullptr), "residual and sum go together");
  if (!halo_supported(g, 0, 0, nullptr, nullptr, o_hat) || g->cin % 128 != 0 || g->cout % 128 != 0)
    return set_error(MODIFF_ERR_UNSUPPORTED,
                     "packed 4-bit operands cover 3x3 stride-1 pad-1 layers with cin and cout "
                     "multiples of 128 and at least 128 pixels per image in rows of 16..64");
  return launch_igemm_halo(reinterpret_cast<const int8_t*>(codes4),
                           reinterpret_cast<const int8_t*>(wcodes4), 0, x_scale, w_scale, nullptr,
                           o_hat, accumulate, g, (cudaStream_t)stream, residual, sum_out, nullptr,
                           nullptr, w_zp);
}

extern "C" int modiff_device_status(int* status, int reset) {
  MODIFF_CHECK_ARG(status != nullptr, "status is NULL");
  return read_device_status(status, reset);
}
