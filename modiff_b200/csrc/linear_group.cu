// Several small quantised linear layers that read the SAME activation codes, in one launch.
//
// Every residual block projects the same swish(temb) (ddim/models/diffusion.py:121-123, 297-301;
// ldm/modules/diffusionmodules/openaimodel.py:236-262): ~20 GEMMs of batch x 512 x 256 per
// step, each far too small to fill the GPU and dominated by launch and prologue time.  The
// residual codes are shared already (one quantisation per step); this kernel also shares the
// launch: a block owns 16 output channels of one layer (its weight rows sit in shared memory) and
// up to 256 batch rows, accumulating with dp4a.  With few rows the chain of dp4a along the input
// channels is what bounds it, so the threads that the rows leave over share a row: KS lanes take
// every KS-th 16-byte piece of it (and, with one or two rows, four warps take four channels
// each), and their integer sums are added by shuffles.  Measured, one row per thread -> shared
// rows: 2 rows, cin 1280, 22 layers 40.7 -> 13.7 us; 8 rows, cin 512 11.7 -> 6.1 us; 154 rows, cin 768,
// 2 x 320 channels 21.8 -> 9.3 us; 256 rows, cin 512 49 -> 41 us.
//
// Arithmetic per layer: out = o_hat + (sum codes * (q - zp)) * delta_x * delta_w[c]
// (qdiff/quant_layer.py:345-365), integer part exact.
#include "common.cuh"

namespace modiff {
namespace {

constexpr int kGroupChannels = 16;
constexpr int kGroupThreads = 256;

// A thread owns CPT of the block's channels for one row and every 2^lg_ks-th piece of it; the
// lanes of a row are neighbours.  Four blocks a SM: with the 70 registers that the compiler takes
// otherwise only three fit, and a grid of 445 - 592 blocks runs twice (64 rows, 3 x 320: 7.8 -> 12.6 us).
template <int CPT>
__global__ void __launch_bounds__(kGroupThreads, CPT == kGroupChannels ? 4 : 0)
linear_group_kernel(const int8_t* __restrict__ codes, const float* __restrict__ x_scale, int rows,
                    int cin, int kp, int lg_ks, const modiff_linear_item* __restrict__ items,
                    const int32_t* __restrict__ block_map) {
  extern __shared__ __align__(16) int8_t w_sh[];   // [16][kp]
  const int layer = block_map[2 * blockIdx.x];
  const int c0 = block_map[2 * blockIdx.x + 1];
  const modiff_linear_item it = items[layer];
  const int pieces = kp / 16;
  for (int idx = threadIdx.x; idx < kGroupChannels * pieces; idx += blockDim.x) {
    const int r = idx / pieces, piece = idx - r * pieces;
    const int co = c0 + r;
    int4 v = make_int4(0, 0, 0, 0);
    if (co < it.cout) {
      const size_t slot = it.with_sum_rows ? (size_t)(co / 128) * 144 + (co % 128) : (size_t)co;
      v = __ldg(reinterpret_cast<const int4*>(it.wcodes + slot * kp) + piece);
    }
    reinterpret_cast<int4*>(w_sh)[idx] = v;
  }
  __syncthreads();
  constexpr int kChanGroups = kGroupChannels / CPT;
  constexpr int kGroupSize = kGroupThreads / kChanGroups;     // threads per channel group (whole warps)
  const int cg0 = ((int)threadIdx.x / kGroupSize) * CPT;
  const int slot = (int)threadIdx.x % kGroupSize;
  const int ks = 1 << lg_ks, kpart = slot & (ks - 1);
  const int n = blockIdx.y * (kGroupSize >> lg_ks) + (slot >> lg_ks);
  int acc[CPT];
#pragma unroll
  for (int c = 0; c < CPT; ++c) acc[c] = 0;
  int rsum = 0;
  if (n < rows) {
    const int4* arow = reinterpret_cast<const int4*>(codes + (size_t)n * cin);
    for (int k = kpart; k < cin / 16; k += ks) {
      const int4 a = __ldg(arow + k);
      rsum = __dp4a(a.x, 0x01010101, rsum);
      rsum = __dp4a(a.y, 0x01010101, rsum);
      rsum = __dp4a(a.z, 0x01010101, rsum);
      rsum = __dp4a(a.w, 0x01010101, rsum);
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        const int4 w = reinterpret_cast<const int4*>(w_sh + (size_t)(cg0 + c) * kp)[k];
        int s = acc[c];
        s = __dp4a(a.x, w.x, s);
        s = __dp4a(a.y, w.y, s);
        s = __dp4a(a.z, w.z, s);
        s = __dp4a(a.w, w.w, s);
        acc[c] = s;
      }
    }
  }
  for (int o = ks >> 1; o > 0; o >>= 1) {           // integer sums: any order gives the same bits
    rsum += __shfl_xor_sync(0xffffffffu, rsum, o);
#pragma unroll
    for (int c = 0; c < CPT; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
  }
  if (n >= rows) return;
  const float xs = x_scale[0];
  float* orow = it.o_hat + (size_t)n * it.cout + c0 + cg0;
#pragma unroll
  for (int c = 0; c < CPT; ++c) {
    const int co = c0 + cg0 + c;
    if (co < it.cout && (c & (ks - 1)) == kpart) {   // the row's lanes share the channels
      int iv = acc[c];
      if (it.w_corr) iv += it.w_corr[co] * rsum;
      orow[c] = fmaf((float)iv, __fmul_rn(xs, it.w_scale[co]), orow[c]);
    }
  }
}

}  // namespace
}  // namespace modiff

using namespace modiff;

extern "C" int modiff_linear_group(const int8_t* codes, const float* x_scale, int rows, int cin,
                                   const modiff_linear_item* items, const int32_t* block_map,
                                   int n_blocks, void* stream) {
  MODIFF_CHECK_ARG(codes && x_scale && items && block_map, "NULL pointer argument");
  MODIFF_CHECK_ARG(rows > 0 && n_blocks > 0, "empty group");
  MODIFF_CHECK_ARG(cin > 0 && cin % 16 == 0 && cin <= 4096, "cin %d must be a multiple of 16 <= 4096",
                   cin);
  MODIFF_CHECK_ARG((((uintptr_t)codes | (uintptr_t)items) & 15) == 0, "buffers must be 16-byte aligned");
  const int kp = round_up(cin, 128);
  const size_t smem = (size_t)kGroupChannels * kp;
  const int cpt = rows <= 2 ? 4 : kGroupChannels;
  const int slots = kGroupThreads * cpt / kGroupChannels;      // threads per channel group
  // Lanes per row: two, and further doublings where the rows leave the lanes over in one block or the
  // grid stays below 2.75 blocks a SM: each doubling adds blocks along the rows, every block loads its 16
  // weight rows again, and four of them are resident.  A row is cut into at most 16 pieces (one row
  // alone into 32).  us for 1, 2, 4 .. 32 lanes, (rows, input channels, layers):
  //   8, 512, 22 of 128 / 256     11.9  9.5  7.3  6.2  6.1  6.7     (one thread a row, 56 registers: 11.7)
  //   64, 320, 3 x 320            10.3  8.4  7.4  6.2  6.6  7.8     (10.1)
  //   96, 1280, 3 x 1280          35.9 30.0 34.1 28.4 33.2 45.4     (35.4)
  //   154, 768, 2 x 640           24.7 19.4 15.5 13.6 16.3 22.5     (23.5)
  //   192, 1280, 22 of 320 - 1280 178  158  187  197  250  380      (180)
  //   256, 512, 22 of 128 / 256   50.1 40.7 44.0 50.8 65.6 98.7     (49.0)
  //   512, 320, 3 x 320           17.2 17.7 18.7 20.3 27.5 38.8     (16.9)
  const int max_lg = rows == 1 ? 5 : 4;
  const int64_t max_blocks = 11 * device_sms() / 4;
  int lg_ks = 1;
  while (lg_ks < max_lg && ((rows << (lg_ks + 1)) <= slots ||
                            (int64_t)n_blocks * ceil_div(rows, slots >> (lg_ks + 1)) <= max_blocks))
    ++lg_ks;
  dim3 grid(n_blocks, ceil_div(rows, slots >> lg_ks));
  cudaStream_t s = (cudaStream_t)stream;
  if (cpt == 4) {
    static SmemLimit smem_limit;
    MODIFF_CUDA(raise_smem_limit(linear_group_kernel<4>, smem, smem_limit));
    linear_group_kernel<4><<<grid, kGroupThreads, smem, s>>>(codes, x_scale, rows, cin, kp, lg_ks, items,
                                                             block_map);
  } else {
    static SmemLimit smem_limit;
    MODIFF_CUDA(raise_smem_limit(linear_group_kernel<kGroupChannels>, smem, smem_limit));
    linear_group_kernel<kGroupChannels><<<grid, kGroupThreads, smem, s>>>(codes, x_scale, rows, cin, kp,
                                                                          lg_ks, items, block_map);
  }
  MODIFF_LAUNCH_CHECK("linear_group_kernel");
  return MODIFF_OK;
}
