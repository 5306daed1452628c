// 3 x 3 convolutions for the flexure warm-start U-Net: implicit GEMM on the tensor cores, BF16
// operands, FP32 accumulation.
//
// Layout: activations NHWC (channels innermost), BF16; a tensor is addressed by a pixel stride
// (channels per pixel of the buffer) and a channel offset, so a layer can read or write a slice
// of a concatenated buffer. Padding is periodic in x (the raster wraps east-west) and zero in y,
// which makes the gradient with respect to the input the same kernel run on the output gradient
// with the taps mirrored and the weight matrix transposed.
//
// Forward / input-gradient: out[p][co] = sum_{tap, ci} in[p + off(tap)][ci] W[tap][ci][co], a GEMM
// with M = pixels, N = output channels, K = 9 x input channels (k_conv3x3_res, and k_conv3x3_line where
// that one's larger blocks are too few or do not fit). Fragments are loaded with
// ldmatrix (x4 for A, x4.trans for B from XOR-swizzled shared memory) and multiplied with
// mma.sync.m16n8k16.row.col.f32.bf16.bf16.f32.
//
// Weight gradient: dW[tap][ci][co] = sum_p in[p + off(tap)][ci] g[p][co], a GEMM with M = input
// channels, N = output channels, K = pixels; each block reduces a chunk of the pixels for all nine
// taps and writes a partial tile, and a second pass sums the partials in a fixed order (deterministic).
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"

namespace dt {

typedef __nv_bfloat16 bf16;

struct Tensor4 {
  bf16* p;      // base of the buffer
  int stride;   // channels per pixel of the buffer
  int off;      // first channel of this tensor
  int c;        // channels of this tensor
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  unsigned s = smem_addr(smem);
  int n = valid ? 16 : 0;  // zero-fill when the source is padding
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void ldmatrix_x4(unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3, const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3, const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(smem_addr(p)));
}

__device__ __forceinline__ void mma_bf16(float* d, const unsigned* a, const unsigned* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Swizzled offsets (in bf16 elements) of 16-byte chunk `chunk` of row `row`:
// A tiles are rows of 32 bf16 (4 chunks, 64 B); B tiles are rows of BN bf16 (BN/8 chunks).
__device__ __forceinline__ int swz_a(int row, int chunk) { return row * 32 + ((chunk ^ ((row >> 1) & 3)) << 3); }
template <int BN>
__device__ __forceinline__ int swz_b(int row, int chunk) {
  if (BN == 32) return row * 32 + ((chunk ^ ((row >> 1) & 3)) << 3);  // 64-byte rows, as swz_a
  return row * BN + ((chunk ^ (row & 7)) << 3);                       // 128-byte rows
}

enum { EPI_BIAS_RELU = 0, EPI_BIAS = 1, EPI_STORE = 2, EPI_MASK = 3 };

// Two neighbouring channels of a pixel's output: the bias and ReLU, or the producing ReLU's mask.
template <int EPI>
__device__ __forceinline__ void conv_store(bf16* dst, int col, float v0, float v1, const float* __restrict__ bias, int co0,
                                           const Tensor4& mask, size_t pix) {
  if (EPI == EPI_BIAS_RELU || EPI == EPI_BIAS) {
    v0 += bias[co0 + col];
    v1 += bias[co0 + col + 1];
  }
  if (EPI == EPI_BIAS_RELU) {
    v0 = fmaxf(v0, 0.f);
    v1 = fmaxf(v1, 0.f);
  }
  __nv_bfloat162* d2 = reinterpret_cast<__nv_bfloat162*>(dst + col);
  if (EPI == EPI_MASK) {
    // the gradient through the producing ReLU: zero where its output was zero
    __nv_bfloat162 m = *reinterpret_cast<const __nv_bfloat162*>(mask.p + pix * mask.stride + mask.off + co0 + col);
    if (!(__bfloat162float(m.x) > 0.f)) v0 = 0.f;
    if (!(__bfloat162float(m.y) > 0.f)) v1 = 0.f;
  }
  *d2 = __floats2bfloat162_rn(v0, v1);
}

// One 3 x 3 convolution (or its input gradient with mirrored, transposed weights): W is
// [9][Cin][Cout] bf16, tap = ky * 3 + kx reading in[y + ky - 1][x + kx - 1]. Image rows of width
// `w` (a multiple of 64), `h` rows, `nimg` images. A block takes 64 pixels of a row by BN output channels,
// its four warps 32 by BN / 2 each; a step stages one tap's pixels and weights of 32 channels, two steps
// in flight. Small blocks, so few pixels still reach many SMs; the pixels are staged nine times. Sums in
// k_conv3x3_res's order, so the same values.
template <int BN, int EPI>
__global__ void __launch_bounds__(128) k_conv3x3_line(int nimg, int h, int w, Tensor4 in, const bf16* __restrict__ W,
                                                 const float* __restrict__ bias, Tensor4 out, Tensor4 mask) {
  constexpr int BM = 64, BK = 32;
  __shared__ __align__(128) bf16 sA[2][BM * BK];
  __shared__ __align__(128) bf16 sB[2][BK * BN];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1;  // warp tile: rows wm*32.., cols wn*(BN/2)..
  const int tiles_x = w / BM;
  int bid = blockIdx.x;
  const int xt = bid % tiles_x;
  bid /= tiles_x;
  const int y = bid % h;
  const int n = bid / h;
  const int x0 = xt * BM;
  const int co0 = blockIdx.y * BN;
  const int cin = in.c;
  const int kchunks = 9 * (cin / BK);
  constexpr int NT = BN / 16;  // n8 tiles per warp
  float acc[2][NT][4];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < NT; ++b)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.f;

  auto load = [&](int kc, int stage) {
    int tap = kc / (cin / BK);
    int ci0 = (kc % (cin / BK)) * BK;
    int ky = tap / 3, kx = tap % 3;
    int yy = y + ky - 1;
    bool yok = yy >= 0 && yy < h;
    // A: 64 pixels x 32 channels = 256 chunks of 16 B; 2 a thread
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      int cidx = tid + q * 128;
      int row = cidx >> 2, ch = cidx & 3;
      int xx = x0 + row + kx - 1;
      xx = xx < 0 ? xx + w : (xx >= w ? xx - w : xx);
      const bf16* src = in.p + ((size_t)((size_t)n * h + (yok ? yy : 0)) * w + xx) * in.stride + in.off + ci0 + ch * 8;
      cp_async16(&sA[stage][swz_a(row, ch)], src, yok);
    }
    // B: 32 k-rows x BN channels
    constexpr int BCH = BK * BN / 8;
#pragma unroll
    for (int q = 0; q < (BCH + 127) / 128; ++q) {
      int cidx = tid + q * 128;
      if (cidx < BCH) {
        int row = cidx / (BN / 8), ch = cidx % (BN / 8);
        const bf16* src = W + ((size_t)tap * cin + ci0 + row) * out.c + co0 + ch * 8;
        cp_async16(&sB[stage][swz_b<BN>(row, ch)], src, true);
      }
    }
    cp_async_commit();
  };

  load(0, 0);
  for (int kc = 0; kc < kchunks; ++kc) {
    int stage = kc & 1;
    if (kc + 1 < kchunks) {
      load(kc + 1, stage ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      unsigned af[2][4];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        int row = wm * 32 + mt * 16 + (lane & 15);
        int chunk = (kk >> 3) + (lane >> 4);
        ldmatrix_x4(af[mt][0], af[mt][1], af[mt][2], af[mt][3], &sA[stage][swz_a(row, chunk)]);
      }
      unsigned bfr[NT][2];
#pragma unroll
      for (int nt = 0; nt < NT; nt += 2) {
        int krow = kk + (lane & 15);
        int chunk = (wn * (BN / 2) + nt * 8) / 8 + (lane >> 4);
        unsigned r0, r1, r2, r3;
        ldmatrix_x4_trans(r0, r1, r2, r3, &sB[stage][swz_b<BN>(krow, chunk)]);
        bfr[nt][0] = r0;
        bfr[nt][1] = r1;
        bfr[nt + 1][0] = r2;
        bfr[nt + 1][1] = r3;
      }
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) mma_bf16(acc[mt][nt], af[mt], bfr[nt]);
    }
    __syncthreads();
  }
  // epilogue: rows = pixels, cols = output channels
  const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      int row = wm * 32 + mt * 16 + g + half * 8;
      size_t pix = ((size_t)n * h + y) * w + x0 + row;
      bf16* dst = out.p + pix * out.stride + out.off + co0;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int col = wn * (BN / 2) + nt * 8 + t4 * 2;
        conv_store<EPI>(dst, col, acc[mt][nt][half * 2], acc[mt][nt][half * 2 + 1], bias, co0, mask, pix);
      }
    }
}

// The same with the pixels staged once. A block takes RY rows by 64 pixels of one image and BN output channels, its
// warps 32 pixels each of one row by all BN channels. The region's (RY + 2) x 66 pixels of every input
// channel are copied once into shared memory (padding and wrap in the copies) and the nine taps read them
// at shifted addresses; the weights come a tap and 32 channels at a time through a ring of STAGES.
// Products are summed by tap, then channel, 16 at a time. A pixel's channels are spaced by 16 bytes
// more than their own, which puts the eight rows of an ldmatrix in distinct banks.
// 2 RY x COW warps of 32 pixels by NC channels each, BN = NC COW.
// Bound by the legacy tensor path's issue (mma.sync) and its ldmatrix loads: 16 x 512 x 256 pixels, warm,
// 32 -> 32 channels 166 us (232 TFLOP/s; the line kernel 238), the gradient 32 -> 96 502 (690), a
// masked gradient 32 -> 32 178 (254), 64 -> 64 at half the size 139 (161).
__host__ __device__ constexpr size_t conv_res_smem(int cin, int ry, int bn, int stages) {
  return (size_t)(ry + 2) * 66 * (cin * 2 + 16) + (size_t)stages * 32 * bn * 2;
}
template <int NC, int COW, int RY, int STAGES, int EPI>
__global__ void __launch_bounds__(64 * RY * COW) k_conv3x3_res(int nimg, int h, int w, Tensor4 in, const bf16* __restrict__ W,
                                                         const float* __restrict__ bias, Tensor4 out, Tensor4 mask) {
  constexpr int BN = NC * COW, NTH = 64 * RY * COW, BK = 32, NT = NC / 8;
  extern __shared__ __align__(128) unsigned char conv_smem[];
  const int cin = in.c, pitch = cin * 2 + 16;  // bytes a pixel
  bf16* const sB = reinterpret_cast<bf16*>(conv_smem);
  unsigned char* const sA = conv_smem + (size_t)STAGES * BK * BN * 2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row = (warp >> 1) % RY, px0 = (warp & 1) * 32,
            nc0 = warp / (2 * RY) * NC;
  const int tiles_x = w / 64, tiles_y = (h + RY - 1) / RY;
  int bid = blockIdx.x;
  const int x0 = (bid % tiles_x) * 64;
  bid /= tiles_x;
  const int y0 = (bid % tiles_y) * RY, n = bid / tiles_y;
  const int co0 = blockIdx.y * BN, cchunks = cin / BK, steps = 9 * cchunks;
  auto load_b = [&](int s) {
    if (s < steps) {
      const int tap = s / cchunks, ci0 = (s - tap * cchunks) * BK;
      bf16* dst = sB + (s % STAGES) * BK * BN;
      for (int c = tid; c < BK * BN / 8; c += NTH) {
        const int r = c / (BN / 8), ch = c % (BN / 8);
        cp_async16(dst + swz_b<BN>(r, ch), W + ((size_t)tap * cin + ci0 + r) * out.c + co0 + ch * 8, true);
      }
    }
    cp_async_commit();
  };
  {
    const int per = cin / 8, total = (RY + 2) * 66 * per;
    for (int c = tid; c < total; c += NTH) {
      const int px = c / per, ch = c - px * per, ry = px / 66, rx = px - ry * 66;
      const int yy = y0 + ry - 1;
      int xx = x0 + rx - 1;
      xx = xx < 0 ? xx + w : (xx >= w ? xx - w : xx);
      const bool ok = yy >= 0 && yy < h;
      cp_async16(sA + px * pitch + ch * 16, in.p + ((size_t)((size_t)n * h + (ok ? yy : 0)) * w + xx) * in.stride + in.off + ch * 8, ok);
    }
  }
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) load_b(s);  // the region's copies are in the first group
  float acc[2][NT][4];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < NT; ++b)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.f;
  int tap = 0, ci0 = 0;
  for (int s = 0; s < steps; ++s) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();  // step s's weights are there, and step s - 1's stage is read
    load_b(s + STAGES - 1);
    const bf16* b = sB + (s % STAGES) * BK * BN;
    const int ky = tap / 3, kx = tap - 3 * ky;
    const unsigned char* a = sA + ((row + ky) * 66 + px0 + kx + (lane & 15)) * pitch + (ci0 + (lane >> 4) * 8) * 2;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      unsigned af[2][4], bfr[NT][2];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) ldmatrix_x4(af[mt][0], af[mt][1], af[mt][2], af[mt][3], a + mt * 16 * pitch + kk * 2);
#pragma unroll
      for (int nt = 0; nt < NT; nt += 2) {
        unsigned r0, r1, r2, r3;
        ldmatrix_x4_trans(r0, r1, r2, r3, b + swz_b<BN>(kk + (lane & 15), nc0 / 8 + nt + (lane >> 4)));
        bfr[nt][0] = r0;
        bfr[nt][1] = r1;
        bfr[nt + 1][0] = r2;
        bfr[nt + 1][1] = r3;
      }
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) mma_bf16(acc[mt][nt], af[mt], bfr[nt]);
    }
    ci0 += BK;
    if (ci0 == cin) {
      ci0 = 0;
      ++tap;
    }
  }
  cp_async_wait<0>();
  if (y0 + row >= h) return;
  const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const size_t pix = ((size_t)n * h + y0 + row) * w + x0 + px0 + mt * 16 + g + half * 8;
      bf16* dst = out.p + pix * out.stride + out.off + co0;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int col = nc0 + nt * 8 + t4 * 2;
        conv_store<EPI>(dst, col, acc[mt][nt][half * 2], acc[mt][nt][half * 2 + 1], bias, co0, mask, pix);
      }
    }
}

// Weight gradient partials: a block takes all nine taps of 16 CIG input by 32 COG output channels
// over a chunk of the pixels, in order, 32 a tile; part[chunk][tap][ci][co] (FP32). A step's 64 pixels of
// the output gradient and the three rows of 66 they multiply are copied once into shared memory for all
// taps (WG_STAGES in flight), and a warp keeps TAPS taps (a row of three, or one) of 16 x 32 channels
// in registers, so an output-gradient fragment serves TAPS products. Pixels are spaced as in
// k_conv3x3_res. Each sum takes its chunk's pixels 16 at a time in raster order, whatever the tile
// of channels: spreading a step's rows over warps or finer chunks moves the FP32 sums of 32768
// pixels by 3e-5 of the gradient.
// Bound by its chain of 16-pixel products a warp (64 chunks leave one or two blocks an SM) and the
// ldmatrix loads. A block a tap, each staging the pixels anew, took 705 us for 32 -> 32 channels at
// 16 x 512 x 256 pixels (its 64-channel tile half empty), now 360; 96 -> 32 1325, now 701; 64 -> 64 at half
// the size 218, now 172; 384 -> 128 at a quarter 587, now 409.
constexpr int WG_STAGES = 4;
__host__ __device__ constexpr int wg_stage(int cig, int cog) { return 3 * 66 * (cig * 32 + 16) + 64 * (cog * 64 + 16); }
__host__ __device__ constexpr int wg_threads(int cig, int cog, int taps) { return 32 * 9 / taps * cig * cog; }
template <int CIG, int COG, int TAPS>
__global__ void __launch_bounds__(wg_threads(CIG, COG, TAPS), 2)
    k_conv3x3_wgrad(int nimg, int h, int w, Tensor4 in, Tensor4 g, int tiles_per_chunk, float* __restrict__ part) {
  constexpr int NTH = wg_threads(CIG, COG, TAPS), PA = CIG * 32 + 16, PB = COG * 64 + 16;
  constexpr int REGION = 3 * 66 * PA, STAGE = wg_stage(CIG, COG), TG = 9 / TAPS;
  extern __shared__ __align__(128) unsigned char conv_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tap0 = warp % TG * TAPS, ky = tap0 / 3, kx0 = tap0 % 3, cig = warp / TG % CIG, cog = warp / (TG * CIG);
  const int cin = in.c, cout = g.c, co_tiles = cout / (32 * COG);
  const int co0 = blockIdx.x % co_tiles * (32 * COG), ci0 = blockIdx.x / co_tiles * (16 * CIG);
  const int tiles_x = w / 64, total = nimg * h * (w / 32);
  const int t_begin = blockIdx.y * tiles_per_chunk, t_end = min(total, t_begin + tiles_per_chunk);
  const int s_begin = t_begin / 2, s_end = (t_end + 1) / 2;  // steps of two tiles, the first and last perhaps half
  float acc[TAPS][4][4];
#pragma unroll
  for (int a = 0; a < TAPS; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.f;
  auto load = [&](int s) {
    if (s < s_end) {
      unsigned char* const sA = conv_smem + (s - s_begin) % WG_STAGES * STAGE;
      const int x0 = s % tiles_x * 64, line = s / tiles_x, y = line % h;  // line = image * h + y
      for (int c = tid; c < 3 * 66 * CIG * 2; c += NTH) {
        const int px = c / (CIG * 2), ch = c % (CIG * 2), r = px / 66, yy = y + r - 1;
        int xx = x0 + px - r * 66 - 1;
        xx = xx < 0 ? xx + w : (xx >= w ? xx - w : xx);
        const bool ok = yy >= 0 && yy < h;
        cp_async16(sA + px * PA + ch * 16, in.p + ((size_t)(ok ? line + r - 1 : line) * w + xx) * in.stride + in.off + ci0 + ch * 8, ok);
      }
      for (int c = tid; c < 64 * COG * 4; c += NTH) {
        const int px = c / (COG * 4), ch = c % (COG * 4);
        cp_async16(sA + REGION + px * PB + ch * 16, g.p + ((size_t)line * w + x0 + px) * g.stride + g.off + co0 + ch * 8, true);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int q = 0; q < WG_STAGES - 1; ++q) load(s_begin + q);
  for (int s = s_begin; s < s_end; ++s) {
    cp_async_wait<WG_STAGES - 2>();
    __syncthreads();  // step s is there, and step s - 1's stage is read
    load(s + WG_STAGES - 1);
    const unsigned char* const sA = conv_smem + (s - s_begin) % WG_STAGES * STAGE;
    // A = in^T (rows input channels, columns pixels) from [pixel][ci], so loaded transposed
    const unsigned char* a = sA + (ky * 66 + kx0 + (lane & 7) + ((lane >> 4) << 3)) * PA + cig * 32 + ((lane >> 3) & 1) * 16;
    const unsigned char* b = sA + REGION + (lane & 15) * PB + cog * 64 + (lane >> 4) * 16;
    auto tile = [&](int x) {  // 32 pixels
#pragma unroll
      for (int px = 0; px < 32; px += 16) {
        unsigned bf[4][2], af[TAPS][4];
        ldmatrix_x4_trans(bf[0][0], bf[0][1], bf[1][0], bf[1][1], b + (x + px) * PB);
        ldmatrix_x4_trans(bf[2][0], bf[2][1], bf[3][0], bf[3][1], b + (x + px) * PB + 32);
#pragma unroll
        for (int k = 0; k < TAPS; ++k)
          ldmatrix_x4_trans(af[k][0], af[k][1], af[k][2], af[k][3], a + (x + px + k) * PA);
#pragma unroll
        for (int k = 0; k < TAPS; ++k)
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) mma_bf16(acc[k][nt], af[k], bf[nt]);
      }
    };
    if (2 * s >= t_begin && 2 * s + 1 < t_end) {
      tile(0);
      tile(32);
    } else {
      tile(2 * s >= t_begin ? 0 : 32);
    }
  }
  cp_async_wait<0>();
  const int gq = lane >> 2, t4 = lane & 3;
#pragma unroll
  for (int k = 0; k < TAPS; ++k)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int ci = ci0 + cig * 16 + gq + half * 8;
      float* dst = part + (((size_t)blockIdx.y * 9 + tap0 + k) * cin + ci) * cout + co0 + cog * 32 + t4 * 2;
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
        *reinterpret_cast<float2*>(dst + nt * 8) = make_float2(acc[k][nt][half * 2], acc[k][nt][half * 2 + 1]);
    }
}

}  // namespace dt
