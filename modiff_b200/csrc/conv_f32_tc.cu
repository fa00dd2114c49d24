// fp32 convolution on the 5th-generation tensor cores (sm_100a) at fp32 precision: the plain
// layers of the first-stage decoder (ldm/modules/diffusionmodules/model.py:465-573) and every
// other stride-1 convolution of an unquantised QuantModule (qdiff/quant_layer.py:309-311).
//
// An fp32 value is the sum of three bf16 values h + m + l (8 + 8 + 8 significand bits, |m| <= 2^-8
// and |l| <= 2^-17 of the value): exactly from 2^-103 on; of smaller values, parts below bf16's
// normal range (2^-126) may be lost.  A product of two is nine bf16 products; the six largest (hh,
// hm, mh, mm, hl, lh) are taken, and ml, lm, ll, together at most 2^-24 of the product, are not.
// tcgen05.mma kind::f16 adds the six, per 64-channel chunk, into tensor memory (small products
// first) with the tensor core's rounding of its accumulator; every chunk's 24 instructions are then
// drained and added to fp32 registers with ordinary rounding, so that only the sums inside a chunk
// meet that rounding.  What this gives is measured, not proven: against 64 bits the rms error is
// 0.14 - 0.73 of conv_fp32_kernel's on 25 shapes from 32 channels 1x1 to 768 channels 3x3, with
// operands of both signs and with positive ones (32 channels 1x1: 5.9e-8 against 1.0e-7, positive
// 6.5e-8 against 8.9e-8; 512 channels 3x3: 1.7e-7 against 1.2e-6).
//
// Operands: activation planes [image][part][h][w][cp] written by split3_kernel, which evaluates
// GroupNorm + SiLU on the way and repeats the pixels of a nearest x2 upsampling, so neither
// tensor is written in fp32; weight planes [part][cout][taps][kb].  Padding is the copy
// engine's zero fill (planes hold no halo).  The epilogue adds bias and an optional residual.
#include "common.cuh"
#include "tc_common.cuh"

namespace modiff {

int read_device_status_conv_f32(int* status, int reset) { return read_status_this_unit(status, reset); }

namespace {

constexpr int kTileM = 128;
constexpr int kChunk = 64;                      // channels per stage: one 128-byte swizzled row
constexpr int kAPart = kTileM * kChunk * 2;     // bytes of one part of the A tile
constexpr int kEpiWarps = 8;
constexpr int kThreads = 64 + 32 * kEpiWarps;   // TMA warp, MMA warp, epilogue warps
constexpr int kMaxStages = 4;
constexpr int kSmemBudget = 221184;

struct ConvParams {
  int batch, cin, cout, h, w, kw, taps, pad_t, pad_l, ho, wo;
  int cp, kb;                     // channel pitch of the planes, K pitch of a weight tap
  int bw, bh, bn;                 // box of output pixels forming one M tile
  int bn_box;                     // images one copy delivers (bn, or the batch when smaller)
  int tiles_w, tiles_h, n_tiles, total_tiles;
  int chunks, stages;
  const uint16_t* planes;
  const uint16_t* wplanes;
  const float* bias;              // [cout] or NULL
  const float* residual;          // fp32 [batch][cout][ho*wo] or NULL
  float* out;
};

__device__ inline uint16_t bf16_nearest(float x) {   // round to nearest even; finite stays finite
  uint32_t u = __float_as_uint(x);
  if ((u & 0x7f800000u) == 0x7f800000u) return (uint16_t)(u >> 16) | ((u & 0x7fffffu) ? 0x40u : 0u);
  const uint32_t r = u + 0x7fffu + ((u >> 16) & 1u);
  return (uint16_t)(((r & 0x7f800000u) == 0x7f800000u ? u : r) >> 16);
}
__device__ inline float bf16_value(uint16_t h) { return __uint_as_float((uint32_t)h << 16); }

// x = p[0] + p[1] + p[2], exactly from 2^-103 on; an infinity or NaN sits in p[0] alone.
__device__ inline void split3(float x, uint16_t (&p)[3]) {
  p[0] = bf16_nearest(x);
  const bool special = (__float_as_uint(x) & 0x7f800000u) == 0x7f800000u;
  const float r = special ? 0.0f : x - bf16_value(p[0]);
  p[1] = bf16_nearest(r);
  p[2] = bf16_nearest(r - bf16_value(p[1]));
}

// The plain fp32 sum of one output element over (channel, tap), operands put together again from
// their planes.  Called where the tensor-core sum is not finite: an infinity times the small parts
// of the other operand is not what the infinity times their sum is.
__device__ __noinline__ float plain_sum(const ConvParams& p, int n, int co, int y, int x) {
  const size_t part = (size_t)p.h * p.w * p.cp;
  const size_t wpart = (size_t)p.cout * p.taps * p.kb;
  float acc = 0.0f;
  for (int c = 0; c < p.cin && !isnan(acc); ++c)
    for (int t = 0; t < p.taps; ++t) {
      const int yy = y - p.pad_t + t / p.kw, xx = x - p.pad_l + t % p.kw;
      float a = 0.0f;
      if (yy >= 0 && yy < p.h && xx >= 0 && xx < p.w) {
        const uint16_t* s = p.planes + (size_t)n * 3 * part + ((size_t)yy * p.w + xx) * p.cp + c;
        a = (bf16_value(s[0]) + bf16_value(s[part])) + bf16_value(s[2 * part]);
      }
      const uint16_t* s = p.wplanes + ((size_t)co * p.taps + t) * p.kb + c;
      acc = fmaf(a, (bf16_value(s[0]) + bf16_value(s[wpart])) + bf16_value(s[2 * wpart]), acc);
    }
  return acc;
}

// Bound: tensor pipe (24 MMAs of M = 128, N, K = 16 per 64-channel chunk) and, close behind, the
// L2 -> shared-memory feed of 48 KB + 384 N bytes per chunk.  Both operands' three parts are
// loaded once per chunk and meet in six products.  Measured, decoder of 8 latents of 32x32 (5.0
// TFLOP): 293 ms in conv_fp32_kernel -> 26.7 ms here, 190 TFLOP/s of fp32 products = 1.14 PFLOP/s of
// bf16 (0.82 of a cuBLAS GEMM's sustained 1.385 PFLOP/s, 0.70 of its 1.634 in a burst); error of the
// decoded image against 64 bits 7.3e-6 -> 2.6e-6 (one 512x512 image: 1.2e-5 -> 1.0e-5).
template <int N>
__global__ void __launch_bounds__(kThreads, 1)
conv_f32_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                   const __grid_constant__ ConvParams p) {
  constexpr int kBPart = N * kChunk * 2;
  constexpr int kStageBytes = 3 * (kAPart + kBPart);
  constexpr int kCols = N < 32 ? 32 : N;             // tensor-memory columns of one accumulator
  constexpr int kHalf = N >= 64 ? N / 2 : 32;        // columns an epilogue warp owns
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[kMaxStages];
  __shared__ __align__(8) uint64_t bar_empty[kMaxStages];
  __shared__ __align__(8) uint64_t bar_tmem_full[2];
  __shared__ __align__(8) uint64_t bar_tmem_empty[2];
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  volatile int* abort_flag = &abort_sh;
  const uint32_t ring = smem_u32(smem_raw);

  if (threadIdx.x == 0) {
    abort_sh = 0;
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&bar_tmem_full[b]), 1);
      mbar_init(smem_u32(&bar_tmem_empty[b]), kEpiWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base_sh)),
                 "r"((uint32_t)(2 * kCols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_sh;
  const int iters = p.taps * p.chunks;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      const uint32_t bytes = (uint32_t)(3 * (kChunk * 2 * p.bw * p.bh * p.bn_box + kBPart));
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < p.total_tiles && ok; tile += gridDim.x) {
        const int nt = tile % p.n_tiles;
        int m = tile / p.n_tiles;
        const int x0 = (m % p.tiles_w) * p.bw - p.pad_l;
        m /= p.tiles_w;
        const int y0 = (m % p.tiles_h) * p.bh - p.pad_t;
        const int img = (m / p.tiles_h) * p.bn;
        for (int tap = 0; tap < p.taps && ok; ++tap) {
          const int dy = tap / p.kw, dx = tap % p.kw;
          for (int ch = 0; ch < p.chunks; ++ch) {
            ok = mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1u, abort_flag);
            if (!ok) break;
            const uint32_t full = smem_u32(&bar_full[stage]);
            const uint32_t a_dst = ring + stage * kStageBytes;
            const uint32_t b_dst = a_dst + 3 * kAPart;
            mbar_arrive_expect_tx(full, bytes);
#pragma unroll
            for (int part = 0; part < 3; ++part) {
              tma_load_5d(a_dst + part * kAPart, &map_a, full, ch * kChunk, x0 + dx, y0 + dy, part, img);
              tma_load_3d(b_dst + part * kBPart, &map_b, full, tap * p.kb + ch * kChunk, nt * N, part);
            }
            if (++stage == p.stages) { stage = 0; phase ^= 1u; }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t idesc = make_idesc_bf16(kTileM, N);
    int stage = 0, buf = 0;
    uint32_t phase = 0, bphase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < p.total_tiles && ok; tile += gridDim.x) {
      for (int it = 0; it < iters; ++it) {
        ok = mbar_wait(smem_u32(&bar_tmem_empty[buf]), bphase ^ 1u, abort_flag);
        if (!ok) break;
        ok = mbar_wait(smem_u32(&bar_full[stage]), phase, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(buf * kCols);
        const uint32_t a_src = ring + stage * kStageBytes;
        const uint64_t adesc = make_smem_desc(a_src);
        const uint64_t bdesc = make_smem_desc(a_src + 3 * kAPart);
        if (elect_one()) {
          constexpr int pa[6] = {1, 2, 0, 1, 0, 0}, pb[6] = {1, 0, 2, 0, 1, 0};
#pragma unroll
          for (int pr = 0; pr < 6; ++pr)
#pragma unroll
            for (int k = 0; k < kChunk / 16; ++k)
              tc_mma_bf16(d_tmem, adesc + (uint64_t)(pa[pr] * (kAPart >> 4) + 2 * k),
                          bdesc + (uint64_t)(pb[pr] * (kBPart >> 4) + 2 * k), idesc,
                          (pr > 0 || k > 0) ? 1u : 0u);
          tc_commit(smem_u32(&bar_empty[stage]));
          tc_commit(smem_u32(&bar_tmem_full[buf]));
        }
        __syncwarp();
        if (++stage == p.stages) { stage = 0; phase ^= 1u; }
        if (++buf == 2) { buf = 0; bphase ^= 1u; }
      }
    }
  } else {
    // ------------------------------------------------------------ accumulate + epilogue
    const int quarter = warp & 3;
    const int col0 = ((warp - 2) >> 2) * kHalf;
    const int row = quarter * 32 + lane;
    const int tile_px = p.bh * p.bw;
    const int ni = row / tile_px, pl = row % tile_px;
    const int hi = pl / p.bw, wi = pl % p.bw;
    const int howo = p.ho * p.wo;
    int buf = 0;
    uint32_t bphase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < p.total_tiles; tile += gridDim.x) {
      float acc[kHalf];
#pragma unroll
      for (int j = 0; j < kHalf; ++j) acc[j] = 0.0f;
      for (int it = 0; it < iters; ++it) {
        ok = mbar_wait(smem_u32(&bar_tmem_full[buf]), bphase, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * kCols + col0);
        if (col0 < N) {
#pragma unroll
          for (int q = 0; q < kHalf / 32; ++q) {
            int v[32];
            tc_ld32(t_row + 32 * q, v);
            tc_wait_ld();
            if (q == kHalf / 32 - 1) {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(smem_u32(&bar_tmem_empty[buf]));
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[32 * q + j] += __int_as_float(v[j]);
          }
        } else {
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bar_tmem_empty[buf]));
        }
        if (++buf == 2) { buf = 0; bphase ^= 1u; }
      }
      if (!ok) break;
      const int nt = tile % p.n_tiles;
      int m = tile / p.n_tiles;
      const int x = (m % p.tiles_w) * p.bw + wi;
      m /= p.tiles_w;
      const int y = (m % p.tiles_h) * p.bh + hi;
      const int n = (m / p.tiles_h) * p.bn + ni;
      const int co0 = nt * N + col0;
      const int ncols = min(min(kHalf, N - col0), p.cout - co0);
      if (n < p.batch && y < p.ho && x < p.wo && ncols > 0) {
        const size_t base = ((size_t)n * p.cout + co0) * howo + (size_t)y * p.wo + x;
#pragma unroll
        for (int j = 0; j < kHalf; ++j)
          if (j < ncols) {
            float v = acc[j];
            if (!isfinite(v)) v = plain_sum(p, n, co0 + j, y, x);
            if (p.bias) v += __ldg(p.bias + co0 + j);
            if (p.residual) v = __ldg(p.residual + base + (size_t)j * howo) + v;
            p.out[base + (size_t)j * howo] = v;
          }
      }
    }
  }

  // ---------------------------------------------------------------- teardown
  __syncwarp();
  if (abort_sh) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);   // let copies in flight land
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"((uint32_t)(2 * kCols))
                 : "memory");
  }
}

// ---------------------------------------------------------------- GroupNorm statistics
// One (image, group) slab is contiguous; it is cut into pieces of 8192 floats, one block each
// (the decoder's 512x512 level has 32 slabs of 4 MB, which one block per slab would leave to 32
// SMs).  A block holds its piece in registers and takes mean and squared deviations in two steps;
// gn_pieces_kernel puts the pieces of a slab together.  Bound: HBM, 4 bytes per element.
constexpr int kPiece = 8192;

__global__ void __launch_bounds__(256)
gn_piece_kernel(const float* __restrict__ x, float2* __restrict__ pieces, int64_t count, int npieces,
                int vec) {
  __shared__ float sh[32];
  const int64_t slab = blockIdx.x / npieces;
  const int64_t beg = (int64_t)(blockIdx.x % npieces) * kPiece;
  const int len = (int)(count - beg < kPiece ? count - beg : kPiece);
  const float* s = x + slab * count + beg;
  float v[kPiece / 256];
  if (vec) {
#pragma unroll
    for (int i = 0; i < kPiece / 1024; ++i) {
      const int e = 4 * ((int)threadIdx.x + 256 * i);
      const float4 f = e < len ? __ldg(reinterpret_cast<const float4*>(s + e)) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < kPiece / 1024; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int e = 4 * ((int)threadIdx.x + 256 * i) + j;
        v[4 * i + j] = e < len ? __ldg(s + e) : 0.0f;
      }
  }
  float a = 0.0f;
#pragma unroll
  for (int i = 0; i < kPiece / 256; ++i) a += v[i];
  const float mean = block_sum(a, sh) / (float)len;
  float q = 0.0f;
#pragma unroll
  for (int i = 0; i < kPiece / 256; ++i) {
    const int e = 4 * ((int)threadIdx.x + 256 * (i / 4)) + i % 4;
    const float d = v[i] - mean;
    q += e < len ? d * d : 0.0f;
  }
  q = block_sum(q, sh);
  if (threadIdx.x == 0) pieces[blockIdx.x] = make_float2(mean, q);
}

// (mean, 1 / sqrt(var + eps)) of every slab from its pieces; one warp per slab.
__global__ void __launch_bounds__(32)
gn_pieces_kernel(const float2* __restrict__ pieces, float2* __restrict__ stats, int64_t count, int npieces,
                 float eps) {
  const float2* s = pieces + (size_t)blockIdx.x * npieces;
  float a = 0.0f;
  for (int i = threadIdx.x; i < npieces; i += 32) {
    const int64_t left = count - (int64_t)i * kPiece;
    a += s[i].x * ((float)(left < kPiece ? left : kPiece) / (float)count);
  }
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  float q = 0.0f;
  for (int i = threadIdx.x; i < npieces; i += 32) {
    const int64_t left = count - (int64_t)i * kPiece;
    const float d = s[i].x - a;
    q += s[i].y + d * d * (float)(left < kPiece ? left : kPiece);
  }
  for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
  if (threadIdx.x == 0) stats[blockIdx.x] = make_float2(a, 1.0f / sqrtf(q / (float)count + eps));
}

// ---------------------------------------------------------------- operand planes
constexpr int kTileC = 64, kTileP = 64;

struct SplitParams {
  const float* x;                 // [batch][c][h*w]
  const float2* stats;            // [batch][groups] or NULL (no GroupNorm)
  const float* gamma;
  const float* beta;
  uint16_t* out;                  // [batch][3][pixels][cp]
  int c, w, hw, cp, cpg, silu, pb, cb, total;
};

// NCHW fp32 -> three NHWC bf16 planes through a shared-memory transpose of 64 channels x 64
// pixels.  Bound: HBM, 4 + 6 bytes per element (4 + 24 with UP2, which writes a pixel four times).
template <bool VEC, bool UP2>
__global__ void __launch_bounds__(256)
split3_kernel(const SplitParams p) {
  __shared__ uint32_t tile_sh[3][kTileP][kTileC / 2 + 1];
  const int cg = threadIdx.x >> 4;   // channel group: 4 channels
  const int pq = threadIdx.x & 15;   // pixel quad
  const size_t part = (size_t)p.hw * p.cp * (UP2 ? 4 : 1);
  for (int tile = blockIdx.x; tile < p.total; tile += gridDim.x) {
    const int n = tile / (p.pb * p.cb);
    const int rem = tile % (p.pb * p.cb);
    const int c0 = (rem / p.pb) * kTileC;
    const int p0 = (rem % p.pb) * kTileP;
    const int px0 = p0 + 4 * pq;
    float v[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = c0 + 4 * cg + i;
      const float* src = p.x + ((size_t)n * p.c + c) * p.hw + px0;
      if (VEC) {
        const float4 f = (c < p.c && px0 < p.hw) ? __ldg(reinterpret_cast<const float4*>(src))
                                                 : make_float4(0.f, 0.f, 0.f, 0.f);
        v[i][0] = f.x; v[i][1] = f.y; v[i][2] = f.z; v[i][3] = f.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i][j] = (c < p.c && px0 + j < p.hw) ? __ldg(src + j) : 0.0f;
      }
    }
    if (p.stats) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = c0 + 4 * cg + i;
        if (c < p.c) {
          const float2 st = __ldg(p.stats + (size_t)n * (p.c / p.cpg) + c / p.cpg);
          const float ga = p.gamma[c] * st.y, be = p.beta[c];
#pragma unroll
          for (int j = 0; j < 4; ++j) v[i][j] = gn_apply(v[i][j], st.x, ga, be);
        }
      }
    }
    if (p.silu) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i][j] = silu_f(v[i][j]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint16_t s[4][3];
#pragma unroll
      for (int i = 0; i < 4; ++i) split3(v[i][j], s[i]);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        tile_sh[q][4 * pq + j][2 * cg] = (uint32_t)s[0][q] | ((uint32_t)s[1][q] << 16);
        tile_sh[q][4 * pq + j][2 * cg + 1] = (uint32_t)s[2][q] | ((uint32_t)s[3][q] << 16);
      }
    }
    __syncthreads();
    // 4 threads per pixel; each writes 16 channels (32 bytes) of every part
    const int px = threadIdx.x >> 2;
    const int piece = threadIdx.x & 3;
    const int pp = p0 + px;
    const int cbase = c0 + 16 * piece;
    if (pp < p.hw && cbase < p.cp) {
      const int y = pp / p.w, x = pp % p.w;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const uint32_t* t = &tile_sh[q][px][8 * piece];
        const uint4 lo = make_uint4(t[0], t[1], t[2], t[3]);
        const uint4 hi = make_uint4(t[4], t[5], t[6], t[7]);
#pragma unroll
        for (int r = 0; r < (UP2 ? 4 : 1); ++r) {
          const size_t pix = UP2 ? (size_t)(2 * y + (r >> 1)) * (2 * p.w) + 2 * x + (r & 1) : (size_t)pp;
          uint16_t* dst = p.out + ((size_t)n * 3 + q) * part + pix * p.cp + cbase;
          *reinterpret_cast<uint4*>(dst) = lo;
          if (cbase + 8 < p.cp) *reinterpret_cast<uint4*>(dst + 8) = hi;   // cp is a multiple of 8
        }
      }
    }
    __syncthreads();
  }
}

// w[cout][cin][taps] fp32 -> out[3][cout][taps][kb], zeros beyond cin.
__global__ void __launch_bounds__(256)
split3_weights_kernel(const float* __restrict__ w, uint16_t* __restrict__ out, int cout, int cin, int taps,
                      int kb) {
  const int64_t part = (int64_t)cout * taps * kb;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < part; i += stride) {
    const int c = (int)(i % kb);
    const int64_t row = i / kb;                       // co * taps + tap
    const int64_t co = row / taps, tap = row % taps;
    uint16_t s[3];
    split3(c < cin ? __ldg(w + (co * cin + c) * taps + tap) : 0.0f, s);
#pragma unroll
    for (int q = 0; q < 3; ++q) out[q * part + i] = s[q];
  }
}

inline int plane_pitch(int cin) { return round_up(cin, 8); }
inline int weight_pitch(int cin) { return round_up(cin, kChunk); }

// widest power of two that divides the extent when that is at least 8 (no masked pixels), else
// the smallest one that covers it; at most 128
inline int box_width(int extent) {
  int b = extent & -extent;
  if (b < 8 && b < extent) {
    b = 1;
    while (b < extent && b < 128) b *= 2;
  }
  return b < 128 ? b : 128;
}

template <int N>
int launch_conv(const CUtensorMap& ma, const CUtensorMap& mb, ConvParams& p, int sms, cudaStream_t s) {
  const int stage = 3 * (kAPart + N * kChunk * 2);
  p.stages = kSmemBudget / stage < kMaxStages ? kSmemBudget / stage : kMaxStages;
  const size_t smem = (size_t)p.stages * stage;
  static SmemLimit limit;
  MODIFF_CUDA(raise_smem_limit(conv_f32_tc_kernel<N>, smem, limit));
  conv_f32_tc_kernel<N><<<p.total_tiles < sms ? p.total_tiles : sms, kThreads, smem, s>>>(ma, mb, p);
  MODIFF_LAUNCH_CHECK("conv_f32_tc_kernel");
  return MODIFF_OK;
}

}  // namespace
}  // namespace modiff

using namespace modiff;

extern "C" int64_t modiff_f32_planes_bytes(const modiff_conv_geom* g) {
  return g ? (int64_t)g->batch * 6 * g->h * g->w * plane_pitch(g->cin) : 0;
}

extern "C" int64_t modiff_f32_weights_bytes(const modiff_conv_geom* g) {
  return g ? 6ll * g->cout * g->kh * g->kw * weight_pitch(g->cin) : 0;
}

extern "C" int64_t modiff_f32_norm_bytes(const modiff_conv_geom* g, int groups) {
  if (!g || groups <= 0) return 0;
  const int64_t count = (int64_t)(g->cin / groups) * g->h * g->w;   // g->h x g->w covers upsampled inputs too
  return 8ll * g->batch * groups * (1 + ceil_div64(count, kPiece));
}

extern "C" int modiff_f32_split_weights(const float* w, uint16_t* out, const modiff_conv_geom* g,
                                        void* stream) {
  int rc = validate_geom(g);
  if (rc) return rc;
  MODIFF_CHECK_ARG(w && out && ((uintptr_t)out & 15) == 0, "NULL or misaligned pointer argument");
  const int64_t n = modiff_f32_weights_bytes(g) / 6;
  const int64_t blocks = ceil_div64(n, 256);
  split3_weights_kernel<<<(int)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, (cudaStream_t)stream>>>(
      w, out, g->cout, g->cin, g->kh * g->kw, weight_pitch(g->cin));
  MODIFF_LAUNCH_CHECK("split3_weights_kernel");
  return MODIFF_OK;
}

extern "C" int modiff_f32_split(const float* x, const modiff_conv_geom* g, int up2, const float* gamma,
                                const float* beta, int groups, float eps, int silu, void* work,
                                uint16_t* planes, void* stream) {
  int rc = validate_geom(g);
  if (rc) return rc;
  MODIFF_CHECK_ARG(x && planes && ((uintptr_t)planes & 15) == 0, "NULL or misaligned pointer argument");
  MODIFF_CHECK_ARG(!up2 || (g->h % 2 == 0 && g->w % 2 == 0), "an upsampled input has even sides");
  MODIFF_CHECK_ARG(groups == 0 || (gamma && beta && work && groups > 0 && g->cin % groups == 0),
                   "bad GroupNorm argument");
  cudaStream_t s = (cudaStream_t)stream;
  SplitParams p;
  p.x = x;
  p.c = g->cin;
  p.w = up2 ? g->w / 2 : g->w;
  p.hw = p.w * (up2 ? g->h / 2 : g->h);
  p.cp = plane_pitch(g->cin);
  p.gamma = gamma;
  p.beta = beta;
  p.stats = nullptr;
  p.cpg = groups ? g->cin / groups : 1;
  p.silu = silu;
  p.out = planes;
  if (groups) {
    const int64_t count = (int64_t)p.cpg * p.hw;
    const int64_t np = ceil_div64(count, kPiece), slabs = (int64_t)g->batch * groups;
    MODIFF_CHECK_ARG(np * slabs < (1ll << 31), "tensor too large");
    float2* stats = (float2*)work;
    float2* pieces = stats + slabs;
    const int vec = count % 4 == 0 && ((uintptr_t)x & 15) == 0;
    gn_piece_kernel<<<(unsigned)(np * slabs), 256, 0, s>>>(x, pieces, count, (int)np, vec);
    MODIFF_LAUNCH_CHECK("gn_piece_kernel");
    gn_pieces_kernel<<<(unsigned)slabs, 32, 0, s>>>(pieces, stats, count, (int)np, eps);
    MODIFF_LAUNCH_CHECK("gn_pieces_kernel");
    p.stats = stats;
  }
  p.pb = ceil_div(p.hw, kTileP);
  p.cb = ceil_div(g->cin, kTileC);
  const int64_t total = (int64_t)p.pb * p.cb * g->batch;
  MODIFF_CHECK_ARG(total < (1ll << 31), "tensor too large");
  p.total = (int)total;
  const int blocks = total < 148 * 8 ? (int)total : 148 * 8;
  const bool vec = p.hw % 4 == 0 && ((uintptr_t)x & 15) == 0;
  if (up2) {
    if (vec) split3_kernel<true, true><<<blocks, 256, 0, s>>>(p);
    else split3_kernel<false, true><<<blocks, 256, 0, s>>>(p);
  } else {
    if (vec) split3_kernel<true, false><<<blocks, 256, 0, s>>>(p);
    else split3_kernel<false, false><<<blocks, 256, 0, s>>>(p);
  }
  MODIFF_LAUNCH_CHECK("split3_kernel");
  return MODIFF_OK;
}

extern "C" int modiff_conv_f32_tc(const uint16_t* planes, const uint16_t* wplanes, const float* bias,
                                  const float* residual, float* out, const modiff_conv_geom* g,
                                  void* stream) {
  int rc = validate_geom(g);
  if (rc) return rc;
  MODIFF_CHECK_ARG(planes && wplanes && out, "NULL pointer argument");
  MODIFF_CHECK_ARG((((uintptr_t)planes | (uintptr_t)wplanes) & 15) == 0, "planes must be 16-byte aligned");
  if (g->stride != 1 || g->split != 0)
    return set_error(MODIFF_ERR_UNSUPPORTED, "the tensor-core fp32 convolution has stride 1 and no split");
  const Derived d = derive(*g);
  EncodeTiledFn encode = get_encode_fn();
  if (!encode) return set_error(MODIFF_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is not available");
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    MODIFF_CUDA(cudaGetDevice(&dev));
    MODIFF_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  }
  ConvParams p;
  p.batch = g->batch; p.cin = g->cin; p.cout = g->cout; p.h = g->h; p.w = g->w;
  p.kw = g->kw; p.taps = d.taps; p.pad_t = g->pad_t; p.pad_l = g->pad_l;
  p.ho = d.ho; p.wo = d.wo;
  p.cp = plane_pitch(g->cin);
  p.kb = weight_pitch(g->cin);
  p.chunks = p.kb / kChunk;
  p.bw = box_width(d.wo);
  p.bh = 1;
  while (p.bh * 2 * p.bw <= kTileM && p.bh < d.ho) p.bh *= 2;
  p.bn = kTileM / (p.bw * p.bh);
  p.bn_box = p.bn < g->batch ? p.bn : g->batch;
  p.tiles_w = ceil_div(d.wo, p.bw);
  p.tiles_h = ceil_div(d.ho, p.bh);
  const int64_t m_tiles = (int64_t)p.tiles_w * p.tiles_h * ceil_div(g->batch, p.bn);
  // Columns per tile: 128, or 64 where that fills the SMs better - a tile of 64 columns takes about
  // three quarters of the time of one of 128 (the A tile's copies stay the same).
  int n = 128;
  if (g->cout <= 64) {
    n = g->cout <= 16 ? 16 : (g->cout <= 32 ? 32 : 64);
  } else {
    const int64_t w128 = ceil_div64(m_tiles * ceil_div(g->cout, 128), sms);
    const int64_t w64 = ceil_div64(m_tiles * ceil_div(g->cout, 64), sms);
    if (3 * w64 < 4 * w128) n = 64;
  }
  p.n_tiles = ceil_div(g->cout, n);
  MODIFF_CHECK_ARG(m_tiles * p.n_tiles < (1ll << 31), "tensor too large");
  p.total_tiles = (int)(m_tiles * p.n_tiles);
  p.planes = planes; p.wplanes = wplanes; p.bias = bias; p.residual = residual; p.out = out;

  CUtensorMap ma, mb;
  {
    const cuuint64_t row = (cuuint64_t)p.cp * 2;
    cuuint64_t dims[5] = {(cuuint64_t)p.cp, (cuuint64_t)g->w, (cuuint64_t)g->h, 3, (cuuint64_t)g->batch};
    cuuint64_t strides[4] = {row, row * g->w, row * g->w * g->h, 3 * row * g->w * g->h};
    cuuint32_t box[5] = {(cuuint32_t)kChunk, (cuuint32_t)p.bw, (cuuint32_t)p.bh, 1u, (cuuint32_t)p.bn_box};
    cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    CUresult r = encode(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, (void*)planes, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
      return set_error(MODIFF_ERR_CUDA, "cuTensorMapEncodeTiled(activation planes) failed: %d", (int)r);
  }
  {
    const cuuint64_t row = (cuuint64_t)p.taps * p.kb * 2;
    cuuint64_t dims[3] = {(cuuint64_t)p.taps * p.kb, (cuuint64_t)g->cout, 3};
    cuuint64_t strides[2] = {row, row * g->cout};
    cuuint32_t box[3] = {(cuuint32_t)kChunk, (cuuint32_t)n, 1u};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = encode(&mb, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void*)wplanes, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
      return set_error(MODIFF_ERR_CUDA, "cuTensorMapEncodeTiled(weight planes) failed: %d", (int)r);
  }
  cudaStream_t s = (cudaStream_t)stream;
  switch (n) {
    case 16: return launch_conv<16>(ma, mb, p, sms, s);
    case 32: return launch_conv<32>(ma, mb, p, sms, s);
    case 64: return launch_conv<64>(ma, mb, p, sms, s);
    default: return launch_conv<128>(ma, mb, p, sms, s);
  }
}
