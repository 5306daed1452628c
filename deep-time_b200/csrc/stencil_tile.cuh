// The 13-point operator of a PCG iteration over register tiles: y = A p with p.y (AP_DOT) and the two
// passes of the Jacobi sandwich (JAC_LEFT, JAC_FINAL), for any width, on the block or the row metric.
// k_apply's arithmetic, term for term.
//
// A block takes a region of 64 columns by R = FT_WARPS RPW rows, a lane two neighbouring columns of its
// warp's RPW rows, every array of those cells in registers, all loads issued first. m = d L u and then
// L m + c u: horizontal neighbours from the next lane by a shuffle, vertical ones from the lane's own
// rows, or for a warp's first and last row from the neighbouring warp's through shared memory (one
// barrier a Laplacian). The region's two outer rings, whose outer neighbours are missing, are not
// written: a tile is (64 - 4) x (R - 4) cells. Rows clamp: the raster's first row is its own northern
// neighbour and its last its own southern one, in u and in m alike. x wraps in the loads (region columns
// that repeat on a raster narrower than 64 compute the same values).
// VEC: an even width, so that a lane's two columns are one aligned word.
// Bound by HBM on large rasters: 16, 20 and 24 bytes a cell in FP32 (AP_DOT, JAC_LEFT, JAC_FINAL),
// twice that in FP64. A block walks over tiles, two blocks an SM, so that the reductions end once a
// block: with a block a tile AP_DOT at FP32 4096 x 2048 took 54 us. Against the tile stencils in shared
// memory it replaces (TMA-fed for widths of whole 64-column tiles, cp.async-fed else), L2 flushed, us
// (AP_DOT, JAC_LEFT, JAC_FINAL): FP32 4096 x 2048 39.3, 44.0, 54.0 -> 37.9, 37.7, 49.1; FP64 57.7, 75.6,
// 88.4 -> 59.2, 63.9, 81.9; FP64 1024 x 328 15.6, 14.1, 18.3 -> 13.3, 11.1, 15.3; FP64 1500 x 750 21.6,
// 19.8, 29.6 -> 17.9, 16.3, 23.5.
// The one loss, AP_DOT at FP64 4096 x 2048, is not felt: a mean-D iteration there, which has no other
// stencil, went from 327 to 321 us with the vector kernels' words.
// Included by flexure.cu after k_apply.
#pragma once

namespace dt {

constexpr int FT_H = 2, FT_TX = 64 - 2 * FT_H;
template <class T>
struct Duo {
  T v[2];
};
__device__ __forceinline__ float max_num(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double max_num(double a, double b) { return fmax(a, b); }
template <class T, bool VEC>
__device__ __forceinline__ Duo<T> ft_load(const T* __restrict__ a, size_t row, int c0, int c1, bool ok) {
  Duo<T> p;
  p.v[0] = p.v[1] = (T)0;
  if (!ok) return p;
  if constexpr (VEC) {
    using V = cplx<T>;
    const V t = *reinterpret_cast<const V*>(a + row + c0);
    p.v[0] = t.x;
    p.v[1] = t.y;
  } else {
    p.v[0] = a[row + c0];
    p.v[1] = a[row + c1];
  }
  return p;
}

template <class T, int MODE, bool MET, int FT_WARPS, int RPW, bool VEC>
__global__ void __launch_bounds__(32 * FT_WARPS, 2) k_flex_tile(int w, int h, T inv_dx2, const T* __restrict__ v,
                                                                const T* __restrict__ J, const T* __restrict__ part,
                                                                const T* __restrict__ d, const T* __restrict__ c,
                                                                T* __restrict__ y, double* partials, Scalars* S, int tiles_x,
                                                                int ntiles, const T* __restrict__ ma, const T* __restrict__ mb) {
  if (S->stop) {
    if (blockIdx.x == 0 && threadIdx.x == 0) set_cond(S, 0);
    return;
  }
  constexpr bool JAC = MODE == JAC_LEFT || MODE == JAC_FINAL;
  constexpr int R = FT_WARPS * RPW, TY = R - 2 * FT_H;
  __shared__ Duo<T> edge[2][2][FT_WARPS][32];  // [u, m][first, last row][warp][lane]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Acc<2> acc;
  acc.v[0] = acc.v[1] = 0.0;
  T most = (T)0;
  // a buffer of `edge` is written again only after the next barrier of its other one
#pragma unroll 1
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int ty = tile / tiles_x;
    const int raw = (tile - ty * tiles_x) * FT_TX - FT_H + 2 * lane, j0 = ty * TY - FT_H + warp * RPW;
    int c0 = raw % w;
    c0 += c0 < 0 ? w : 0;
    const int c1 = c0 + 1 == w ? 0 : c0 + 1;
    const bool tile_cols = lane >= FT_H / 2 && lane < 32 - FT_H / 2 && raw < w;
    Duo<T> u[RPW], rr[JAC ? RPW : 1], jj[MODE == JAC_FINAL ? RPW : 1], m[RPW], cc[RPW];
#pragma unroll
    for (int q = 0; q < RPW; ++q) {
      const int j = j0 + q;
      const bool in = j >= 0 && j < h;
      const size_t row = (size_t)(in ? j : 0) * w;
      u[q] = ft_load<T, VEC>(v, row, c0, c1, in);
      if constexpr (JAC) {
        const Duo<T> w_ = ft_load<T, VEC>(J, row, c0, c1, in);
        rr[q] = u[q];
        if constexpr (MODE == JAC_FINAL) {
          jj[q] = w_;
          u[q] = ft_load<T, VEC>(part, row, c0, c1, in);
        } else {
          u[q] = w_;
        }
      }
      m[q] = ft_load<T, VEC>(d, row, c0, c1, in);
      cc[q] = ft_load<T, VEC>(c, row, c0, c1, in && tile_cols);
    }
    if constexpr (JAC) {
      // the vector the mode forms: u = J r (+ part)
#pragma unroll
      for (int q = 0; q < RPW; ++q)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if constexpr (MODE == JAC_FINAL) {
            T t = jj[q].v[e] * rr[q].v[e];
            t += u[q].v[e];
            u[q].v[e] = t;
          } else {
            u[q].v[e] = u[q].v[e] * rr[q].v[e];
          }
        }
    }
    // L x at the lane's cells of row q; up / down: the rows beyond the lane's own
    auto lap = [&](const Duo<T>* x, int q, const Duo<T>& up, const Duo<T>& down) {
      const int j = j0 + q;
      const RowCoef<T, MET> k = row_coef<T, MET>(ma, mb, j, h);
      const Duo<T> self = x[q], north = j == 0 ? self : q ? x[q ? q - 1 : 0] : up,
                   south = j == h - 1 ? self : q + 1 < RPW ? x[q + 1 < RPW ? q + 1 : q] : down;
      const T right = __shfl_down_sync(0xffffffffu, self.v[0], 1), left = __shfl_up_sync(0xffffffffu, self.v[1], 1);
      Duo<T> o;
      o.v[0] = lap5<T, MET>(left, self.v[1], north.v[0], south.v[0], self.v[0], k, inv_dx2);
      o.v[1] = lap5<T, MET>(self.v[0], right, north.v[1], south.v[1], self.v[1], k, inv_dx2);
      return o;
    };
    auto meet = [&](int b, const Duo<T>* x, Duo<T>& up, Duo<T>& down) {
      edge[b][0][warp][lane] = x[0];
      edge[b][1][warp][lane] = x[RPW - 1];
      __syncthreads();
      up.v[0] = up.v[1] = down.v[0] = down.v[1] = (T)0;
      if (warp > 0) up = edge[b][1][warp - 1][lane];
      if (warp < FT_WARPS - 1) down = edge[b][0][warp + 1][lane];
    };
    Duo<T> up, down;
    meet(0, u, up, down);
#pragma unroll
    for (int q = 0; q < RPW; ++q) {
      const Duo<T> l = lap(u, q, up, down);
      m[q].v[0] = l.v[0] * m[q].v[0];
      m[q].v[1] = l.v[1] * m[q].v[1];
    }
    meet(1, m, up, down);
#pragma unroll
    for (int q = 0; q < RPW; ++q) {
      const Duo<T> l = lap(m, q, up, down);
      const int j = j0 + q, rw = warp * RPW + q;
      if (!tile_cols || rw < FT_H || rw >= R - FT_H || j >= h) continue;
      Duo<T> o;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const T uu = u[q].v[e], au = l.v[e] + cc[q].v[e] * uu;
        const bool on = VEC || e == 0 || raw + 1 < w;
        if constexpr (MODE == AP_DOT) {
          o.v[e] = au;
          if (on) acc.v[0] += (double)uu * (double)au;
        } else if constexpr (MODE == JAC_LEFT) {
          o.v[e] = rr[q].v[e] - au;
        } else {
          const T r = rr[q].v[e], z = uu + jj[q].v[e] * (r - au);
          o.v[e] = z;
          if (on) {
            acc.v[0] += (double)r * (double)z;
            most = max_num(most, fabs(z));
          }
        }
      }
      const size_t at = (size_t)j * w + raw;
      if constexpr (VEC) {
        *reinterpret_cast<cplx<T>*>(y + at) = mk<cplx<T>>(o.v[0], o.v[1]);
      } else {
        y[at] = o.v[0];
        if (raw + 1 < w) y[at + 1] = o.v[1];
      }
    }
  }
  if constexpr (MODE != JAC_LEFT) {
    const int kind[2] = {0, 1};
    const unsigned nb = gridDim.x;
    acc.v[1] = (double)most;
    constexpr int site = MODE == AP_DOT ? SITE_PAP : SITE_PRECOND;
    const bool last = MODE == JAC_FINAL ? reduce_partials<2>(acc, kind, partials, &S->ticket[site], nb)
                                        : reduce_partials<1>(*reinterpret_cast<Acc<1>*>(&acc), kind, partials, &S->ticket[site], nb);
    if (last && threadIdx.x == 0) {
      if (MODE == AP_DOT) finish_pap(S, acc.v[0]);
      if (MODE == JAC_FINAL) finish_precond(S, acc.v[0], acc.v[1]);
    }
  }
}

}  // namespace dt
