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
// with M = pixels, N = output channels, K = 9 x input channels (k_conv3x3_res). Fragments are loaded with
// ldmatrix (x4 for A, x4.trans for B from XOR-swizzled shared memory) and multiplied with
// mma.sync.m16n8k16.row.col.f32.bf16.bf16.f32.
//
// Weight gradient: dW[tap][ci][co] = sum_p in[p + off(tap)][ci] g[p][co], a GEMM with M = input
// channels, N = output channels, K = pixels; each block reduces a chunk of pixel tiles and writes
// a partial tile, and a second pass sums the partials in a fixed order (deterministic).
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

enum { EPI_BIAS_RELU = 0, EPI_BIAS = 1, EPI_STORE = 2, EPI_ACCUM = 3, EPI_MASK = 4 };

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
  if (EPI == EPI_ACCUM) {
    __nv_bfloat162 prev = *d2;
    v0 += __bfloat162float(prev.x);
    v1 += __bfloat162float(prev.y);
  }
  *d2 = __floats2bfloat162_rn(v0, v1);
}

// One 3 x 3 convolution (or its input gradient with mirrored, transposed weights): W is [9][Cin][Cout]
// bf16, tap = ky * 3 + kx reading in[y + ky - 1][x + kx - 1]; image rows of width `w` (a multiple of 64),
// `h` rows, `nimg` images. A block takes RY rows by 64 pixels of one image and BN output channels, its
// warps 32 pixels each of one row by all BN channels. The region's (RY + 2) x 66 pixels of every input
// channel are copied once into shared memory (padding and wrap in the copies) and the nine taps read them
// at shifted addresses; the weights come a tap and 32 channels at a time through a ring of STAGES.
// Products are summed by tap, then channel, 16 at a time. A pixel's channels are spaced by 16 bytes
// more than their own, which puts the eight rows of an ldmatrix in distinct banks.
// 2 RY x COW warps of 32 pixels by NC channels each, BN = NC COW.
// Bound by the legacy tensor path's issue (mma.sync) and its ldmatrix loads. Staging every tap's 128
// pixels anew through shared memory (nine times the input traffic) took, at 16 x 512 x 256 cells,
// 357 us for 32 -> 32 channels (now 253, 153 TFLOP/s), 716 for the gradient 32 -> 96 (522), 265
// for a masked gradient 32 -> 32 (184), 492 for 64 -> 192 at half the size (430) and 875 for 384 -> 128
// at a quarter (552).
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

// Weight gradient partials: block (tap, ci tile of 64, co tile of BN) x chunk of pixel tiles.
// part[chunk][tap][ci][co] (FP32).
template <int BN>
__global__ void __launch_bounds__(128) k_conv3x3_wgrad(int nimg, int h, int w, Tensor4 in, Tensor4 g, int tiles_per_chunk,
                                                       float* __restrict__ part) {
  constexpr int BM = 64;  // input channels per block (GEMM M)
  constexpr int BK = 32;  // pixels per k step
  __shared__ __align__(128) bf16 sA[2][BK * BM];  // [pixel][ci] : 32 rows of 64 channels
  __shared__ __align__(128) bf16 sB[2][BK * BN];  // [pixel][co]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1;
  const int cin = in.c, cout = g.c;
  const int ci_tiles = (cin + BM - 1) / BM;
  int bx = blockIdx.x;
  const int co0 = (bx % (cout / BN)) * BN;
  bx /= cout / BN;
  const int ci0 = (bx % ci_tiles) * BM;
  const int tap = bx / ci_tiles;
  const int ky = tap / 3, kx = tap % 3;
  const int chunk = blockIdx.y;
  const int tiles_x = w / BK;
  const int total_tiles = nimg * h * tiles_x;
  constexpr int NT = BN / 16;
  float acc[2][NT][4];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < NT; ++b)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.f;
  const int t_begin = chunk * tiles_per_chunk;
  const int t_end = min(total_tiles, t_begin + tiles_per_chunk);

  auto load = [&](int t, int stage) {
    int xt = t % tiles_x;
    int rest = t / tiles_x;
    int y = rest % h, n = rest / h;
    int x0 = xt * BK;
    int yy = y + ky - 1;
    bool yok = yy >= 0 && yy < h;
    // A: 32 pixels x 64 channels (shifted by the tap) = 256 chunks
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      int cidx = tid + q * 128;
      int row = cidx >> 3, ch = cidx & 7;
      int xx = x0 + row + kx - 1;
      xx = xx < 0 ? xx + w : (xx >= w ? xx - w : xx);
      bool ok = yok && (ci0 + ch * 8 < cin);
      const bf16* src = in.p + ((size_t)((size_t)n * h + (yok ? yy : 0)) * w + xx) * in.stride + in.off + (ok ? ci0 + ch * 8 : 0);
      cp_async16(&sA[stage][swz_b<BM>(row, ch)], src, ok);
    }
    // B: 32 pixels x BN output-channel gradients
    constexpr int BCH = BK * BN / 8;
#pragma unroll
    for (int q = 0; q < (BCH + 127) / 128; ++q) {
      int cidx = tid + q * 128;
      if (cidx < BCH) {
        int row = cidx / (BN / 8), ch = cidx % (BN / 8);
        const bf16* src = g.p + ((size_t)((size_t)n * h + y) * w + x0 + row) * g.stride + g.off + co0 + ch * 8;
        cp_async16(&sB[stage][swz_b<BN>(row, ch)], src, true);
      }
    }
    cp_async_commit();
  };

  if (t_begin < t_end) {
    load(t_begin, 0);
    for (int t = t_begin; t < t_end; ++t) {
      int stage = (t - t_begin) & 1;
      if (t + 1 < t_end) {
        load(t + 1, stage ^ 1);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
#pragma unroll
      for (int kk = 0; kk < BK; kk += 16) {
        // A = in^T: rows ci, cols pixels; the tile is [pixel][ci], so load transposed
        unsigned af[2][4];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          // matrices: (ci 0-7, px 0-7), (ci 8-15, px 0-7), (ci 0-7, px 8-15), (ci 8-15, px 8-15)
          int prow = kk + (lane & 7) + ((lane >> 4) << 3);
          int chunk = (wm * 32 + mt * 16) / 8 + ((lane >> 3) & 1);
          ldmatrix_x4_trans(af[mt][0], af[mt][1], af[mt][2], af[mt][3], &sA[stage][swz_b<BM>(prow, chunk)]);
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
  }
  const int gq = lane >> 2, t4 = lane & 3;
  float* dst = part + ((size_t)chunk * 9 + tap) * cin * cout;
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      int ci = ci0 + wm * 32 + mt * 16 + gq + half * 8;
      if (ci >= cin) continue;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        int co = co0 + wn * (BN / 2) + nt * 8 + t4 * 2;
        dst[(size_t)ci * cout + co] = acc[mt][nt][half * 2];
        dst[(size_t)ci * cout + co + 1] = acc[mt][nt][half * 2 + 1];
      }
    }
}

}  // namespace dt
