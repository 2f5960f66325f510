// Jacobi-PCG of the FP64 path on small meshes, with the whole solve in one launch.
//
// The loop of small kernels (start, p, sums, scalars, update, sums, scalars) pays
// its launches and the loop's conditional node on every iteration: about 25 us
// per iteration on meshes whose vectors take a few us to read. Here a system is
// one thread-block cluster. Its CTAs hold the search direction in shared memory
// and the residual in registers, and meet at the two sums of an iteration (p.Ap
// and r.r), so an iteration costs two cluster barriers (0.25 us each) and the
// FP64 products of a CTA's own rows. On 64^2 Q1 nodes an iteration takes 4 us
// (it took 25 us), bound by the latency of the two sums' chains, not by any unit.
//
// A system's mesh is cut into bands of whole cell rows, one per CTA. A band keeps
// copies of r and p on the P node rows below and the one above it, and updates
// them like its own: the neighbours pass their A p on those rows through
// distributed shared memory along with the partial sum p.Ap, so no third barrier
// is needed for p. The operator is the tensor-product mass matrix, or the product
// form of the TG3 matrix (My + kyy Ky) (x) (Mx + kxx Kx) of an axis-parallel
// direction. Sums are fixed-order: a warp's tree, then a tree over the warps of
// all CTAs, the same on every thread.
//
// A form with more CTAs than a cluster holds, meeting at counters in global memory,
// was measured and left out: a sum took 6 to 10 us there (the partial sums and
// halo rows are lines that every SM writes and reads), and its waits hold only if
// every CTA of the solve is resident, beside whatever else the GPU runs.
#pragma once

#include "operators.cuh"

#include <cooperative_groups.h>

namespace lbfem_gpu
{
  struct FusedArgs
  {
    const double *b, *x_cur, *x_prev;
    double *x;        // the solution; the start if not extrapolate
    CgState *st;
    DevStats *ds;     // counters of a graph-launched step, or null
    StreamCoef sc;
    int sys[NM];      // the systems solved, in cluster order
    int extrapolate;
    double cg_tol;
    int max_its;
  };

  // A thread holds r, A p and x of up to MAXT (column, cell row) pairs of P nodes: 8 to 12
  // nodes. More would spill, and a spilled value is fetched from L2 again after
  // every barrier.
  template <int P>
  struct FusedShape
  {
    static constexpr int THREADS = 512; // most threads of a CTA
    static constexpr int GROUP = 8;     // CTAs of a cluster: the largest portable size
    static constexpr int MAXT = P == 1 ? 10 : P == 2 ? 5 : P == 3 ? 4 : 2;
  };

  // The band of rank `rank` of `group`: cell rows [c0, c1), and in the last band also the
  // mesh's last node row (the upper boundary, or the periodic image row).
  __host__ __device__ inline void
  fused_band(int ncy, int group, int rank, int &c0, int &c1)
  {
    c0 = int((long long)ncy * rank / group);
    c1 = int((long long)ncy * (rank + 1) / group);
  }

  // Doubles of shared memory of a band of at most ncr cell rows: the direction with P halo
  // rows below and one above, the x-pass output, the halo rows of r and of the neighbours'
  // A p, the cell widths and the Jacobi factors.
  template <int P>
  __host__ __device__ inline long long
  fused_smem_doubles(int nfx, int ncx, int ncr)
  {
    const long long pitch = nfx | 1, own = (long long)ncr * P + 1;
    return pitch * ((own + P + 1) + (own + P) + 2 * (P + 1)) + 2LL * (ncx + 2) + nfx + 2LL * (ncr + 2) + own + P + 1;
  }

  // One row's x pass at cell c: the vertex of the cell and its interior nodes from
  // the row's values in the left cell (l) and in the cell itself (u).
  template <int P, bool SEP>
  __device__ __forceinline__ void
  fused_cell(const double (&l)[P + 1], const double (&u)[P + 1], double hl, double h, double kil, double ki,
             double (&out)[P])
  {
    double vl = ref<double, P, OP_M>(P, 0) * l[0];
#pragma unroll
    for (int b = 1; b <= P; ++b)
      vl = fma(ref<double, P, OP_M>(P, b), l[b], vl);
    double acc = hl * vl;
    if constexpr (SEP)
      {
        double kl = ref<double, P, OP_K>(P, 0) * l[0];
#pragma unroll
        for (int b = 1; b <= P; ++b)
          kl = fma(ref<double, P, OP_K>(P, b), l[b], kl);
        acc = fma(kil, kl, acc);
      }
#pragma unroll
    for (int a = 0; a < P; ++a)
      {
        double m = ref<double, P, OP_M>(a, 0) * u[0];
#pragma unroll
        for (int b = 1; b <= P; ++b)
          m = fma(ref<double, P, OP_M>(a, b), u[b], m);
        double v = a == 0 ? fma(h, m, acc) : h * m;
        if constexpr (SEP)
          {
            double k = ref<double, P, OP_K>(a, 0) * u[0];
#pragma unroll
            for (int b = 1; b <= P; ++b)
              k = fma(ref<double, P, OP_K>(a, b), u[b], k);
            v = fma(ki, k, v);
          }
        out[a] = v;
      }
  }

  template <int P, bool SEP>
  __global__ void __launch_bounds__(FusedShape<P>::THREADS, 1)
    k_cg_fused(const Geo geo, const FusedArgs A)
  {
    using S = FusedShape<P>;
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char sm_raw[];
    constexpr int MW = S::THREADS / 32;
    __shared__ double s_slot[4][S::GROUP * MW]; // the warps' partial sums of all CTAs of the cluster
    const Grid &g = geo.g;
    const int nt = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = nt / 32;
    constexpr int group = S::GROUP;
    const int s = A.sys[blockIdx.x / group], rank = blockIdx.x % group;
    const int nfx = g.nfx, ncx = g.ncx, pitch = nfx | 1;
    int c0, c1;
    fused_band(g.ncy, group, rank, c0, c1);
    const int ncr = c1 - c0, j0 = c0 * P;
    const bool last = rank == group - 1;
    const int own = ncr * P + (last ? 1 : 0); // own node rows
    const int TR = ncr * P + P + 1;           // x-pass rows: P below, own, one above
    const int crows = ncr + (last ? 1 : 0);   // y-pass cell rows (the last one: the row of the last vertex only)
    const int n_tasks = crows * nfx;
    const bool below = g.py || rank > 0, above = g.py || !last; // has neighbour rows
    // s_in: the neighbours' A p on the halo rows, P below and one above, and s_rh: r there;
    // at the same place in every CTA, since the neighbours write them.
    // s_p: row q of the band (q = -P .. own - 1) at (q + P) pitch, the row above at (own + P) pitch
    double *s_in = reinterpret_cast<double *>(sm_raw);
    double *s_rh = s_in + pitch * (P + 1);
    double *s_p = s_rh + pitch * (P + 1);
    double *s_t = s_p + pitch * (own + P + 1); // x-pass output, row q at (q + P) pitch
    double *s_hx = s_t + pitch * TR;           // [ncx + 2]: widths of cells -1 .. ncx
    double *s_kx = s_hx + ncx + 2;             // kxx / width
    double *s_ix = s_kx + ncx + 2;             // [nfx]
    double *s_hy = s_ix + nfx;                 // [ncr + 2]: cell rows c0 - 1 .. c1
    double *s_ky = s_hy + ncr + 2;
    double *s_iy = s_ky + ncr + 2;             // [own + P + 1], the rows of s_p
    const long long o = (long long)s * g.N;
    double *xs = A.x + o;
    const double kxx = SEP ? A.sc.kxx[s] : 0., kyy = SEP ? A.sc.kyy[s] : 0.;
    // the mesh row of row k of s_p (images read their source row)
    auto row_of = [&](int k) {
      int j = k < own + P ? j0 + k - P : j0 + ncr * P;
      if (g.py && k < P && j < 0)
        j += g.nuy;
      if (g.py && k == own + P && j >= g.nuy)
        j -= g.nuy;
      return j;
    };
    for (int t = tid; t < ncx + 2; t += nt)
      {
        const int c = wrap(t - 1, g.px, ncx, ncx);
        s_hx[t] = c < 0 ? 0. : geo.hx[c];
        s_kx[t] = c < 0 ? 0. : kxx * geo.hxi[c];
      }
    for (int t = tid; t < nfx; t += nt)
      s_ix[t] = geo.ijx[t];
    for (int t = tid; t < ncr + 2; t += nt)
      {
        const int c = wrap(c0 - 1 + t, g.py, g.ncy, g.ncy);
        s_hy[t] = c < 0 ? 0. : geo.hy[c];
        s_ky[t] = c < 0 ? 0. : kyy * geo.hyi[c];
      }
    for (int t = tid; t < own + P + 1; t += nt)
      {
        const int j = row_of(t);
        s_iy[t] = j >= 0 && j < g.nfy ? geo.ijy[j] : 0.;
      }

    // Sums over the system of v[q], on every thread: each warp's sum goes to every CTA.
    // Everything the CTAs wrote before it is visible after it. Slots sl0 .. sl0 + NQ - 1:
    // a slot is rewritten only after every CTA has read it and met the others again.
    auto sum = [&](auto NQC, double *v, int sl0) {
      constexpr int NQ = decltype(NQC)::value;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1)
#pragma unroll
        for (int q = 0; q < NQ; ++q)
          v[q] += __shfl_down_sync(0xffffffffu, v[q], d);
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        {
          const double w = __shfl_sync(0xffffffffu, v[q], 0);
          if (lane < group)
            *cl.map_shared_rank(&s_slot[sl0 + q][rank * nw + warp], lane) = w;
        }
      cl.sync();
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        v[q] = 0.;
      for (int k = lane; k < group * nw; k += 32)
#pragma unroll
        for (int q = 0; q < NQ; ++q)
          v[q] += s_slot[sl0 + q][k];
#pragma unroll
      for (int d = 16; d > 0; d >>= 1)
#pragma unroll
        for (int q = 0; q < NQ; ++q)
          v[q] += __shfl_xor_sync(0xffffffffu, v[q], d);
    };

    // ---- the operator's x pass: s_t row q = (Mx + kxx Kx) p on rows q = -P .. ncr P
    const int NCX = ncx + (g.px ? 0 : 1);
    auto xcell = [&](int tr, int c) {
      const int k = tr < ncr * P + P || (last && !g.py) ? tr : own + P;
      const double *row = s_p + k * pitch;
      double *trow = s_t + tr * pitch;
      const int v = c * P;
      const int lv = c > 0 ? v - P : g.px ? nfx - 1 - P : -1;
      double l[P + 1], u[P + 1], out[P];
#pragma unroll
      for (int b = 0; b <= P; ++b)
        {
          l[b] = 0.;
          u[b] = 0.;
        }
      u[0] = row[v]; // a periodic axis has no cell at its image column: v < nux there
      if (lv >= 0)
        {
#pragma unroll
          for (int b = 0; b < P; ++b)
            l[b] = row[lv + b];
          l[P] = u[0];
        }
      if (c < ncx)
        {
#pragma unroll
          for (int b = 1; b < P; ++b)
            u[b] = row[v + b];
          u[P] = row[g.px && c == ncx - 1 ? 0 : v + P];
        }
      fused_cell<P, SEP>(l, u, s_hx[c], s_hx[c + 1], s_kx[c], s_kx[c + 1], out);
      trow[v] = out[0];
      if (c < ncx)
        {
#pragma unroll
          for (int a = 1; a < P; ++a)
            trow[v + a] = out[a];
        }
    };
    auto xpass = [&]() {
      __syncthreads(); // the direction is in place
      if constexpr (P == 4)
        {
          // rows fastest: lanes over cells of 4 nodes would meet in 4 banks
          for (unsigned t = tid; t < unsigned(TR * NCX); t += nt)
            {
              const unsigned c = t / unsigned(TR);
              xcell(int(t - c * TR), int(c));
            }
        }
      else
        {
          // a warp takes 32 cells of a row
          int tr = warp % TR, ch = warp / TR;
          while (ch * 32 < NCX)
            {
              const int c = ch * 32 + lane;
              if (c < NCX)
                xcell(tr, c);
              tr += nw;
              while (tr >= TR)
                {
                  tr -= TR;
                  ++ch;
                }
            }
        }
      __syncthreads();
    };
    auto image = [&](int i, int q) { return (g.px && i == g.nux) || (g.py && j0 + q == g.nuy); };
    auto inv_diag = [&](int i, int q) { return image(i, q) ? 1. : s_ix[i] * s_iy[q + P]; };
    // the y pass at column i, cell row cr: A p on rows cr P .. cr P + P - 1
    auto ypass = [&](int i, int cr, double (&out)[P]) {
      const double *t = s_t + (cr * P) * pitch + i;
      double l[P + 1], u[P + 1];
#pragma unroll
      for (int k = 0; k <= P; ++k)
        {
          l[k] = t[k * pitch];
          u[k] = 0.;
        }
      u[0] = l[P];
      if (cr < ncr)
        {
#pragma unroll
          for (int k = 1; k <= P; ++k)
            u[k] = t[(P + k) * pitch];
        }
      fused_cell<P, SEP>(l, u, s_hy[cr], s_hy[cr + 1], s_ky[cr], s_ky[cr + 1], out);
#pragma unroll
      for (int a = 0; a < P; ++a)
        if ((a == 0 || cr < ncr) && image(i, cr * P + a))
          out[a] = s_p[(cr * P + a + P) * pitch + i]; // identity rows
    };
    // f(t, column, cell row) for this thread's tasks, in order
    const int cr_first = tid / nfx, i_first = tid - cr_first * nfx, dc = nt / nfx, di = nt - dc * nfx;
    auto tasks = [&](auto &&f) {
      int cr = cr_first, i = i_first;
#pragma unroll
      for (int t = 0; t < S::MAXT; ++t)
        {
          // opaque: or the unrolled tasks' indices are all computed once, outside the
          // iterations, and kept in (spilled) registers
          asm volatile("" : "+r"(cr), "+r"(i));
          if (t * nt >= n_tasks)
            break;
          if (cr < crows)
            f(t, i, cr);
          cr += dc;
          i += di;
          if (i >= nfx)
            {
              i -= nfx;
              ++cr;
            }
        }
    };
    // f(halo row h: 0 .. P - 1 below, P above; column; the row of s_p) for the halo nodes this thread updates
    auto halo = [&](auto &&f) {
      for (int t = tid; t < (P + 1) * nfx; t += nt)
        {
          const int h = t / nfx, i = t - h * nfx;
          if (h < P ? below : above)
            f(h, i, h < P ? h : own + P);
        }
    };
    // row q's value at column i to the neighbours that hold the row as a halo row, at `to`
    // (s_rh for r, s_in for A p: a neighbour may still read the one when it gets the other)
    auto push = [&](double *to, int q, int i, double v) {
      if (q == 0 && below)
        *cl.map_shared_rank(to + P * pitch + i, rank > 0 ? rank - 1 : group - 1) = v;
      if (q >= ncr * P - P && q < ncr * P && above)
        *cl.map_shared_rank(to + (q - (ncr * P - P)) * pitch + i, last ? 0 : rank + 1) = v;
    };

    // ---- start: r = b - A x0, with the sums b.b, r.r, r.D^-1 r
    double rr[S::MAXT][P]; // r of the own nodes
    {
      // x0 on s_p's rows, halo included
      const double *xc = A.x_cur + o, *xp = A.x_prev + o;
      for (int t = tid; t < (own + P + 1) * nfx; t += nt)
        {
          const int k = t / nfx, i = t - k * nfx;
          double x0 = 0.;
          if (k < P ? below : k < own + P ? true : above)
            {
              const int idx = row_of(k) * nfx + i;
              x0 = A.extrapolate ? -xp[idx] + 2. * xc[idx] : xs[idx];
            }
          s_p[k * pitch + i] = x0;
        }
    }
    cl.sync(); // every CTA runs, before its shared memory is written
    xpass();
    double v3[3] = {0., 0., 0.};
    tasks([&](int t, int i, int cr) {
      double Ax[P], bb[P];
#pragma unroll
      for (int a = 0; a < P; ++a)
        bb[a] = a == 0 || cr < ncr ? A.b[o + (j0 + cr * P + a) * nfx + i] : 0.;
      ypass(i, cr, Ax);
#pragma unroll
      for (int a = 0; a < P; ++a)
        if (a == 0 || cr < ncr)
          {
            const int q = cr * P + a;
            const double r = bb[a] - Ax[a];
            rr[t][a] = r;
            push(s_rh, q, i, r);
            v3[0] += bb[a] * bb[a];
            v3[1] += r * r;
            v3[2] += r * (inv_diag(i, q) * r);
          }
    });
    sum(std::integral_constant<int, 3>(), v3, 0);
    const double tol = A.cg_tol * sqrt(v3[0]);
    double res = sqrt(v3[1]), rz = v3[2], beta = 0.;
    const bool zero = v3[0] == 0.; // b = 0 exactly: x = 0, no iterations
    int status = isnan(res) ? 3 : 0, it = 0;
    bool active = !status && res > tol && !zero;
    tasks([&](int, int i, int cr) {
#pragma unroll
      for (int a = 0; a < P; ++a)
        if ((a == 0 || cr < ncr) && (zero || A.extrapolate))
          xs[(j0 + cr * P + a) * nfx + i] = zero ? 0. : s_p[(cr * P + a + P) * pitch + i];
    });

    // ---- iterations, in the order of updates of deal.II SolverCG (mass.h:204-211)
    while (active)
      {
        // p = D^-1 r + beta p on the own and the halo nodes
        tasks([&](int t, int i, int cr) {
#pragma unroll
          for (int a = 0; a < P; ++a)
            if (a == 0 || cr < ncr)
              {
                double *p = s_p + (cr * P + a + P) * pitch + i;
                const double z = inv_diag(i, cr * P + a) * rr[t][a];
                *p = it == 0 ? z : fma(beta, *p, z);
              }
        });
        halo([&](int h, int i, int k) {
          double *p = s_p + k * pitch + i;
          const double z = s_ix[i] * s_iy[k] * s_rh[h * pitch + i];
          *p = it == 0 ? z : fma(beta, *p, z);
        });
        xpass();
        double ap[S::MAXT][P], xv[S::MAXT][P], pap[1] = {0.};
        tasks([&](int t, int i, int cr) {
          ypass(i, cr, ap[t]);
#pragma unroll
          for (int a = 0; a < P; ++a)
            if (a == 0 || cr < ncr)
              {
                push(s_in, cr * P + a, i, ap[t][a]);
                pap[0] += s_p[(cr * P + a + P) * pitch + i] * ap[t][a];
              }
        });
        sum(std::integral_constant<int, 1>(), pap, 3);
        const double al = rz / pap[0];
        // r -= alpha A p on the own and the halo nodes; x is fetched here and updated after
        // the sums, off their path
        tasks([&](int t, int i, int cr) {
#pragma unroll
          for (int a = 0; a < P; ++a)
            xv[t][a] = a == 0 || cr < ncr ? xs[(j0 + cr * P + a) * nfx + i] : 0.;
        });
        double v2[2] = {0., 0.};
        tasks([&](int t, int i, int cr) {
#pragma unroll
          for (int a = 0; a < P; ++a)
            if (a == 0 || cr < ncr)
              {
                const double r = rr[t][a] + -al * ap[t][a];
                rr[t][a] = r;
                v2[0] += r * r;
                v2[1] += r * (inv_diag(i, cr * P + a) * r);
              }
        });
        halo([&](int h, int i, int) { s_rh[h * pitch + i] += -al * s_in[h * pitch + i]; });
        sum(std::integral_constant<int, 2>(), v2, 0);
        tasks([&](int t, int i, int cr) {
#pragma unroll
          for (int a = 0; a < P; ++a)
            if (a == 0 || cr < ncr)
              xs[(j0 + cr * P + a) * nfx + i] = xv[t][a] + al * s_p[(cr * P + a + P) * pitch + i];
        });
        ++it;
        res = sqrt(v2[0]);
        beta = v2[1] / rz;
        rz = v2[1];
        status = isnan(res) ? 3 : res > tol && it >= A.max_its ? 2 : 0;
        active = !status && res > tol;
      }
    if (tid == 0 && rank == 0)
      {
        CgState *st = A.st;
        st->tol[s] = tol;
        st->res[s] = res;
        st->it[s] = it;
        st->its_total[s] = it;
        st->zero[s] = zero ? 1 : 0;
        st->active[s] = 0;
        atomicAdd(&st->total_its, (unsigned long long)it);
        // a non-finite system (3) wins over the iteration cap (2), whichever ends first
        if (status)
          atomicMax(&st->status, status);
        if (A.ds)
          {
            __threadfence();
            if (atomicAdd(&st->systems_done, 1) == int(gridDim.x) / group - 1)
              {
                __threadfence();
                cg_fold(st, A.ds);
              }
          }
      }
  }
} // namespace lbfem_gpu
