// The Jacobi-PCG kernels of the FP64 path for a product operator, (My + kyy Ky) (x)
// (Mx + kxx Kx): the mass matrix, or the TG3 matrix of an axis-parallel direction.
//
// A CTA takes up to 128 columns by RT rows of one system, one thread per column. The
// operand lands in shared memory with a halo of P; a thread forms the x pass of its
// column row by row from the assembled 1-D row it holds in registers and
// carries a sliding window of 2P + 1 of them through the y pass, whose rows have
// 2P + 1 (vertex) or P + 1 (interior) entries, known at compile time since tiles
// start at cell boundaries.
//
// The element-tile form of these kernels (k_cg_start / _p / _update, kept for the general
// TG3 and Laplace operators, strips, the solve without allocation, and the meshes on which
// it is the faster one) spends
// 160 instructions per node, most of them on index maps and staging, and leaves
// lanes idle in both passes; it was bound by issue and latency on L2-resident
// meshes (13.5 and 21.7 us per launch on 405 x 309 Q4 nodes, 8 systems, whose data
// take 5 us) and at 52 to 60% of the DRAM rate on large ones. At 1024^2 Q3 the start
// went from 766 to 687 us (67% of the measured rate) and the direction from 358 to
// 338 us; on 257^2 Q2 nodes and one system an iteration went from 27 to 20 us.
#pragma once

#include "operators.cuh"

namespace lbfem_gpu
{
  template <int P>
  struct ColShape
  {
    static constexpr int TX = 128;
    static constexpr int RT = P == 3 ? 18 : 16;             // rows, whole cells
    static constexpr int FX = TX + 2 * P, FY = RT + 2 * P; // staged operand
    static constexpr int K = 2 * P + 1;
    static constexpr int KP = K + 1; // pitch of the y rows (16-byte pairs)
    static constexpr int THREADS = TX + 32; // the last warp stages the halo's columns
    // CTAs per SM the registers are sized for: the direction, and the start and update (which
    // hold two cells' rows of b, or of x and r, in flight)
    static constexpr int CTAS_P = P <= 2 ? 6 : 5, CTAS = P <= 2 ? 6 : P == 3 ? 5 : 4;
    static_assert(RT % P == 0, "tiles of whole cells");
  };

  template <int P>
  constexpr size_t
  col_smem()
  {
    using S = ColShape<P>;
    return sizeof(double) * (size_t(S::FX) * S::FY + S::RT * S::KP + S::RT);
  }

  // Columns per CTA so that the CTAs of a row are equally wide.
  __host__ __device__ inline int
  col_width(int nfx)
  {
    const int n = (nfx + 127) / 128;
    return (nfx + n - 1) / n;
  }

  // The tile's tables and this thread's column.
  template <int P, bool SEP>
  struct ColTile
  {
    using S = ColShape<P>;
    double *u, *my, *iy; // staged operand; y rows and inverse y Jacobi factors of the own rows
    int gx0, gy0, tw, gx, rows_in;
    bool col_in, img_col;
    double mx[S::K], ix;

    __device__ __forceinline__ void
    init(const Geo &geo, const StreamCoef &sc, int s, unsigned char *sm)
    {
      const Grid &g = geo.g;
      const int tid = threadIdx.x;
      u = reinterpret_cast<double *>(sm);
      my = u + S::FX * S::FY;
      iy = my + S::RT * S::KP;
      tw = col_width(g.nfx);
      gx0 = blockIdx.x * tw;
      gy0 = blockIdx.y * S::RT;
      gx = gx0 + tid;
      rows_in = g.nfy - gy0;
      col_in = tid < tw && gx < g.nfx;
      img_col = g.px && gx == g.nux;
      const double kxx = SEP ? sc.kxx[s] : 0., kyy = SEP ? sc.kyy[s] : 0.;
      for (int t = tid; t < S::RT; t += S::THREADS)
        iy[t] = gy0 + t < g.nfy ? geo.ijy[gy0 + t] : 0.;
      for (int t = tid; t < S::RT * S::KP; t += S::THREADS)
        {
          const int i = t / S::KP, k = t - i * S::KP, gy = gy0 + i;
          const bool ok = k < S::K && gy < g.nfy && !(g.py && gy == g.nuy);
          double v = ok ? geo.rowy[(long long)gy * S::K + k] : 0.;
          if (SEP && ok)
            v = fma(kyy, geo.rowy[((long long)3 * g.nfy + gy) * S::K + k], v);
          my[t] = v;
        }
#pragma unroll
      for (int k = 0; k < S::K; ++k)
        {
          const bool ok = col_in && !img_col;
          mx[k] = ok ? geo.rowx[(long long)gx * S::K + k] : 0.;
          if (SEP && ok)
            mx[k] = fma(kxx, geo.rowx[((long long)3 * g.nfx + gx) * S::K + k], mx[k]);
        }
      ix = col_in ? (img_col ? 1. : geo.ijx[gx]) : 0.;
    }

    // u <- value(load(storage index), inverse Jacobi factors of the node) on the tile and its
    // halo, 0 outside the grid: a thread per staged column, B rows of loads in flight. Ends
    // with the barrier that also completes the tables.
    template <int B, bool JACOBI, typename Load, typename F>
    __device__ __forceinline__ void
    stage(const Geo &geo, Load &&load, F &&value)
    {
      const Grid &g = geo.g;
      const int c = threadIdx.x;
      if (c < tw + 2 * P)
        {
          const int col = wrap(gx0 - P + c, g.px, g.nux, g.nfx);
          const double ixc = JACOBI && col >= 0 ? geo.ijx[col] : 0.;
          // the mesh row of a staged row, stepped with the periodic wrap
          int row = g.py ? wrap(gy0 - P, 1, g.nuy, g.nfy) : gy0 - P;
#pragma unroll
          for (int q0 = 0; q0 < S::FY; q0 += B)
            {
              double2 v[B];
              double iyr[B];
#pragma unroll
              for (int k = 0; k < B; ++k)
                if (q0 + k < S::FY)
                  {
                    const bool ok = col >= 0 && row >= 0 && row < g.nfy;
                    v[k] = ok ? load(row * g.nfx + col) : make_double2(0., 0.);
                    iyr[k] = JACOBI && ok ? geo.ijy[row] : 0.;
                    ++row;
                    if (g.py && row == g.nuy)
                      row = 0;
                  }
#pragma unroll
              for (int k = 0; k < B; ++k)
                if (q0 + k < S::FY)
                  u[(q0 + k) * S::FX + c] = value(v[k], ixc, iyr[k]);
            }
        }
      __syncthreads();
    }

    // f(row, A u) for this thread's own rows, in order
    template <typename F>
    __device__ __forceinline__ void
    apply(F &&f) const
    {
      double t[S::FY];
#pragma unroll
      for (int q = 0; q < S::FY; ++q)
        {
          const double *w = u + q * S::FX + threadIdx.x; // columns gx - P .. gx + P
          double a0 = mx[0] * w[0], a1 = mx[1] * w[1];
#pragma unroll
          for (int k = 2; k < S::K; ++k)
            if (k & 1)
              a1 = fma(mx[k], w[k], a1);
            else
              a0 = fma(mx[k], w[k], a0);
          t[q] = a0 + a1;
          const int i = q - 2 * P;
          if (i >= 0)
            {
              const double *m = my + i * S::KP;
              // a vertex row couples to 2P + 1 rows, an interior one to its cell's P + 1
              const int a = i % P, k0 = a == 0 ? 0 : P - a, k1 = a == 0 ? 2 * P : 2 * P - a;
              double b0 = 0., b1 = 0.;
#pragma unroll
              for (int k = 0; k < S::K; ++k)
                if (k >= k0 && k <= k1)
                  {
                    if ((k - k0) & 1)
                      b1 = fma(m[k], t[i + k], b1);
                    else
                      b0 = fma(m[k], t[i + k], b0);
                  }
              f(i, b0 + b1);
            }
        }
    }

    __device__ __forceinline__ double
    own(int i) const
    {
      return u[(i + P) * S::FX + threadIdx.x + P];
    }
  };

  // r = b - A xg with xg = extrapolate ? 2 x_cur - x_prev (written to x) : x; sums b.b, r.r, r.D^{-1}r.
  template <int P, bool SEP>
  __global__ void __launch_bounds__(ColShape<P>::THREADS, ColShape<P>::CTAS)
    k_col_start(const Geo geo, const double *__restrict__ b, const double *__restrict__ x_cur,
                const double *__restrict__ x_prev, double *__restrict__ x, double *__restrict__ r, int extrapolate,
                double *__restrict__ partials, const StreamCoef sc, int skip, CgState *st, const CgFinish fin)
  {
    using S = ColShape<P>;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const Grid &g = geo.g;
    const int s = blockIdx.z, nt = gridDim.x * gridDim.y, tile = blockIdx.y * gridDim.x + blockIdx.x;
    if ((skip >> s) & 1)
      {
        if (threadIdx.x == 0 && tile == 0)
          {
            const double v[3] = {0., 0., 0.};
            cg_scalars(st, s, cg_system(st, s), v, 0, fin.cg_tol, fin.max_its);
            cg_system_done(st, fin, 0);
          }
        return;
      }
    const long long o = s * g.N;
    const double *bs = b + o, *xc = extrapolate ? x_cur + o : nullptr, *xp = extrapolate ? x_prev + o : nullptr;
    double *xs = x + o, *rs = r + o;
    ColTile<P, SEP> T;
    T.init(geo, sc, s, sm_raw);
    T.template stage<ColShape<P>::FY / 2, false>(
      geo, [&](int i) { return extrapolate ? make_double2(xc[i], xp[i]) : make_double2(xs[i], 0.); },
      [&](double2 v, double, double) { return extrapolate ? -v.y + 2. * v.x : v.x; });
    double part[3] = {0., 0., 0.};
    if (T.col_in)
      {
        double bv[2][P];
        auto fetch = [&](int c, double (&v)[P]) {
#pragma unroll
          for (int a = 0; a < P; ++a)
            v[a] = c * P + a < T.rows_in ? bs[(T.gy0 + c * P + a) * g.nfx + T.gx] : 0.;
        };
        fetch(0, bv[0]);
        T.apply([&](int i, double Ax) {
          if (i % P == 0 && i + P < S::RT)
            fetch(i / P + 1, bv[(i / P + 1) & 1]);
          if (i >= T.rows_in)
            return;
          const int gy = T.gy0 + i, idx = gy * g.nfx + T.gx;
          double xg = T.own(i), inv = T.ix * T.iy[i];
          if (T.img_col || (g.py && gy == g.nuy))
            {
              xg = extrapolate ? -xp[idx] + 2. * xc[idx] : xs[idx]; // identity rows
              Ax = xg;
              inv = 1.;
            }
          const double bb = bv[(i / P) & 1][i % P], rr = bb - Ax;
          if (extrapolate)
            xs[idx] = xg;
          rs[idx] = rr;
          part[0] += bb * bb;
          part[1] += rr * rr;
          part[2] += rr * (inv * rr);
        });
      }
    cg_finish<3, S::THREADS>(part, partials, st, s, tile, nt, 0, fin);
  }

  // p <- D^{-1} r + beta p (p <- D^{-1} r on the first iteration); sum p.Ap.
  template <int P, bool SEP>
  __global__ void __launch_bounds__(ColShape<P>::THREADS, ColShape<P>::CTAS_P)
    k_col_p(const Geo geo, const double *__restrict__ r, const double *__restrict__ p_in, double *__restrict__ p_out,
            CgState *st, double *__restrict__ partials, const StreamCoef sc, const CgFinish fin)
  {
    using S = ColShape<P>;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const Grid &g = geo.g;
    const int s = blockIdx.z, nt = gridDim.x * gridDim.y, tile = blockIdx.y * gridDim.x + blockIdx.x;
    if (!st->active[s])
      {
        if (tile == 0 && threadIdx.x == 0)
          cg_system_done(st, fin, 1);
        return;
      }
    const bool first = st->it[s] == 0;
    const double beta = st->beta[s];
    const long long o = s * g.N;
    const double *rs = r + o, *ps = p_in + o;
    double *po = p_out + o;
    ColTile<P, SEP> T;
    T.init(geo, sc, s, sm_raw);
    T.template stage<ColShape<P>::FY / 3, true>(
      geo, [&](int i) { return make_double2(rs[i], first ? 0. : ps[i]); },
      [&](double2 v, double ix, double iy) { return first ? ix * iy * v.x : fma(beta, v.y, ix * iy * v.x); });
    double part[1] = {0.};
    if (T.col_in)
      T.apply([&](int i, double Ap) {
        if (i >= T.rows_in)
          return;
        const int gy = T.gy0 + i, idx = gy * g.nfx + T.gx;
        double pn = T.own(i);
        if (T.img_col || (g.py && gy == g.nuy))
          {
            pn = first ? rs[idx] : fma(beta, ps[idx], rs[idx]); // identity rows
            Ap = pn;
          }
        po[idx] = pn;
        part[0] += pn * Ap;
      });
    cg_finish<1, S::THREADS>(part, partials, st, s, tile, nt, 1, fin);
  }

  // x += alpha p, r -= alpha A p; sums r.r, r.D^{-1}r.
  template <int P, bool SEP>
  __global__ void __launch_bounds__(ColShape<P>::THREADS, ColShape<P>::CTAS)
    k_col_update(const Geo geo, double *__restrict__ x, double *__restrict__ r, const double *__restrict__ p,
                 CgState *st, double *__restrict__ partials, const StreamCoef sc, const CgFinish fin)
  {
    using S = ColShape<P>;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const Grid &g = geo.g;
    const int s = blockIdx.z, nt = gridDim.x * gridDim.y, tile = blockIdx.y * gridDim.x + blockIdx.x;
    if (!st->active[s])
      {
        if (tile == 0 && threadIdx.x == 0)
          cg_system_done(st, fin, 2);
        return;
      }
    const double al = st->alpha[s];
    const long long o = s * g.N;
    const double *ps = p + o;
    double *xs = x + o, *rs = r + o;
    ColTile<P, SEP> T;
    T.init(geo, sc, s, sm_raw);
    T.template stage<ColShape<P>::FY / 2, false>(
      geo, [&](int i) { return make_double2(ps[i], 0.); }, [&](double2 v, double, double) { return v.x; });
    double part[2] = {0., 0.};
    if (T.col_in)
      {
        double xv[2][P], rv[2][P];
        auto fetch = [&](int c, double (&v)[P], double (&w)[P]) {
#pragma unroll
          for (int a = 0; a < P; ++a)
            {
              const int idx = (T.gy0 + c * P + a) * g.nfx + T.gx;
              const bool in = c * P + a < T.rows_in;
              v[a] = in ? xs[idx] : 0.;
              w[a] = in ? rs[idx] : 0.;
            }
        };
        fetch(0, xv[0], rv[0]);
        T.apply([&](int i, double Ap) {
          if (i % P == 0 && i + P < S::RT)
            fetch(i / P + 1, xv[(i / P + 1) & 1], rv[(i / P + 1) & 1]);
          if (i >= T.rows_in)
            return;
          const int gy = T.gy0 + i, idx = gy * g.nfx + T.gx;
          double pv = T.own(i), inv = T.ix * T.iy[i];
          if (T.img_col || (g.py && gy == g.nuy))
            {
              pv = ps[idx]; // identity rows
              Ap = pv;
              inv = 1.;
            }
          xs[idx] = xv[(i / P) & 1][i % P] + al * pv;
          const double rr = rv[(i / P) & 1][i % P] + -al * Ap;
          rs[idx] = rr;
          part[0] += rr * rr;
          part[1] += rr * (inv * rr);
        });
      }
    cg_finish<2, S::THREADS>(part, partials, st, s, tile, nt, 2, fin);
  }
} // namespace lbfem_gpu
