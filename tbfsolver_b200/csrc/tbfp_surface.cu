// Surface tension on the grid: the interface cells, the height-function
// curvature and the face force that the projection reads as st (the reference's
// computeSurfaceTension, VOF.f90:1872-2002, with computeBlockCurvature and
// hfColumn, :2070-2290, after Popinet 2009).
//
// The reference works on per-bubble blocks; this is a grid-wide restatement:
//   * interface cells: mixed eps <= c <= 1-eps, full c >= 1-eps (VOF.f90:1094-1108);
//     a full cell with an empty 6-neighbour becomes mixed with c = 1-2 eps
//     (search_full_interface_cells, :672-726);
//   * curvature at a mixed cell: the height-function direction is the largest
//     component of a smoothed central-difference normal (then the second, then
//     the third); in that direction nine columns (the cell's 3x3 neighbourhood
//     across it) each walk at most kStColumn cells toward the full phase and
//     toward the empty phase; the column height is the sum of c times the cell
//     width between the two ends, the interface position is the full end's outer
//     face minus that height; with all nine columns valid the curvature is
//     s * div(grad f / sqrt(1 + |grad f|^2)) of the positions f by second-order
//     (non-uniform in y) differences, s the orientation of the column.  Columns
//     stop at the walls; a cell without a valid direction gets curvature 0 (the
//     reference fits a parabola through interface centroids there);
//   * face force: sigma * k_f * (c(Q) - c(P)) / dc, k_f the mean curvature of the
//     two cells if both are mixed, else the mixed one's, else 0 (computeBlockST,
//     :1904-1996); zero on the wall faces.
//
// Work split.  Only the interface cells (about 1 % of a bubbly channel) need
// more than their own class, so nothing dense is kept but one class byte per
// cell, and the curvature and the force run over a list:
//   1. k_st_classify: reads c once, writes the class bytes, appends the mixed
//      cells to a list (one atomic per block of rows) and, in every other block,
//      fills the three force arrays with zeros;
//   2. k_st_curvature: the listed cells, 32 per warp;
//   3. k_st_faces: the faces of the listed cells and their periodic images.
// Bound: HBM for the first (33 bytes per cell: c 8, class 1, st 24), loads and
// instructions per interface cell for the others.
// 512x384x256 with 200 bubbles: 0.289 + 0.173 + 0.041 ms (the first at 5.7 TB/s),
// where dense passes over all cells (classes with a copy of c, curvature, faces)
// took 0.44 + 10.6 + 2.09 ms.
// The decisions (the normal's ranking, the column sums) use adds and multiplies
// that the compiler does not contract, so they are those of the oracle's
// restatement in oracle/tbfp_oracle.py (surface_tension).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "tbfp_kernels.cuh"

namespace tbfp {

namespace {

constexpr int kStColumn = 6;
// class bits of a cell: mixed; full; promoted (a mixed cell whose c reads as
// 1 - 2 eps); wild (c is NaN, infinite or huge: its faces are evaluated in full
// although neither cell is mixed, so the NaN reaches the force)
constexpr unsigned kMixed = 1, kFull = 2, kPromoted = 4, kWild = 8;
constexpr int kRowWarps = 8;  // rows per block of the row kernels, one per warp

// Index into 0..n-1 of a periodic direction, for an index within two periods
// (columns and stencils leave the grid by at most 7 cells, and n >= 4 in x;
// nz may be 2, hence the loop form).
__device__ __forceinline__ int wrapn(int i, int n) {
  while (i < 0) i += n;
  while (i >= n) i -= n;
  return i;
}
__device__ __forceinline__ int clampj(const StGrid &g, int j) { return j < 0 ? 0 : (j >= g.ny ? g.ny - 1 : j); }
__device__ __forceinline__ long dix(const StGrid &g, int i, int j, int k) {  // dense index of cell (i, j, k)
  return (long)i + (long)g.nx * ((long)j + (long)g.ny * k);
}

// classes of the original field: mixed, full (both bits when c == 1-eps)
__device__ __forceinline__ unsigned cls0(double c, double eps) {
  return ((c >= 0.0 + eps && c <= 1.0 - eps) ? kMixed : 0u) | (c >= 1.0 - eps ? kFull : 0u);
}

// Zeros into elements e0..e1-1 of a (8-byte aligned), 16 bytes at a time.
__device__ __forceinline__ void fill_zero(double *__restrict__ a, long e0, long e1) {
  if (e0 >= e1) return;
  if (threadIdx.x == 0) a[e0] = a[e1 - 1] = 0.0;
  const long lead = (reinterpret_cast<uintptr_t>(a + e0) & 15) ? 1 : 0;
  double2 *v = reinterpret_cast<double2 *>(a + e0 + lead);
  const long n2 = (e1 - e0 - lead) / 2;
  for (long q = threadIdx.x; q < n2; q += blockDim.x) v[q] = make_double2(0.0, 0.0);
}

struct StOut {  // the three force arrays and their layouts
  double *s[3];
  Lay L[3];
  long n[3];
};

// Even blocks classify: a warp takes one row (j, k), four loads of 32 cells in
// flight; stretches of zeros (c = 0 away from the bubbles) are one vote and one
// store.  The row's listed cells are kept as one ballot per 32 cells in lane
// (chunk), which holds a row of nx <= 1024 cells (the x transform's limit; nx is
// a multiple of 4 there), and go to the list in one piece.  Odd blocks fill the
// force arrays, so that the stores run under the classification's latency.
__global__ void __launch_bounds__(32 * kRowWarps) k_st_classify(const double *__restrict__ c, Lay Lc, StGrid g,
                                                                double eps, unsigned char *__restrict__ fl,
                                                                int *__restrict__ list, int *__restrict__ count,
                                                                StOut out) {
  if (blockIdx.x & 1) {
    const long nb = gridDim.x / 2, b = blockIdx.x / 2;
#pragma unroll 1
    for (int d = 0; d < 3; ++d) {
      const long per = (out.n[d] + nb - 1) / nb;
      fill_zero(out.s[d], b * per, min((b + 1) * per, out.n[d]));
    }
    return;
  }
  __shared__ int cnt[kRowWarps], first[kRowWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long row = (long)(blockIdx.x / 2) * kRowWarps + warp;
  const bool live = row < (long)g.ny * g.nz;
  const int j = live ? (int)(row % g.ny) : 0, k = live ? (int)(row / g.ny) : 0;
  const double *cr = c + at(Lc, 1, j + 1, k + 1);
  unsigned char *fr = fl + row * g.nx;
  unsigned mine = 0;  // lane q: listed cells of chunk q
  int total = 0;
  if (live) {
    for (int b = 0; b < g.nx; b += 128) {
      double v[4];
      long long any = 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = b + 32 * u + lane;
        v[u] = i < g.nx ? cr[i] : 0.0;
        any |= __double_as_longlong(v[u]);
      }
      if (!__any_sync(0xffffffffu, any != 0)) {
        if (b + 4 * lane < g.nx) *reinterpret_cast<unsigned *>(fr + b + 4 * lane) = 0u;
        continue;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = b + 32 * u + lane;
        unsigned f = cls0(v[u], eps);
        if (i < g.nx && (f & kFull)) {  // a full cell next to an empty one is an interface cell
          auto cv = [&](int ii, int jj, int kk) { return c[at(Lc, ii + 1, jj + 1, kk + 1)]; };
          const bool empty_nb = cls0(cv(wrapn(i + 1, g.nx), j, k), eps) == 0 ||
                                cls0(cv(wrapn(i - 1, g.nx), j, k), eps) == 0 ||
                                cls0(cv(i, clampj(g, j + 1), k), eps) == 0 ||
                                cls0(cv(i, clampj(g, j - 1), k), eps) == 0 ||
                                cls0(cv(i, j, wrapn(k + 1, g.nz)), eps) == 0 ||
                                cls0(cv(i, j, wrapn(k - 1, g.nz)), eps) == 0;
          if (empty_nb) f = kMixed | kPromoted;
        }
        if (!(fabs(v[u]) <= 1e100)) f |= kWild;
        if (i < g.nx) fr[i] = (unsigned char)f;
        const unsigned m = __ballot_sync(0xffffffffu, i < g.nx && (f & (kMixed | kWild)));
        if (lane == (b >> 5) + u) mine = m;
        total += __popc(m);
      }
    }
  }
  if (lane == 0) cnt[warp] = total;
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int w = 0; w < kRowWarps; ++w) {
      first[w] = s;
      s += cnt[w];
    }
    const int base = s ? atomicAdd(count, s) : 0;
    for (int w = 0; w < kRowWarps; ++w) first[w] += base;
  }
  __syncthreads();
  if (total == 0) return;
  int pos = __popc(mine);  // exclusive prefix over the chunks
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, pos, o);
    if (lane >= o) pos += n;
  }
  pos += first[warp] - __popc(mine);
  for (unsigned m = mine; m; m &= m - 1) list[pos++] = (int)(row * g.nx) + 32 * lane + __ffs(m) - 1;
}

__device__ __forceinline__ double face_pos(const StGrid &g, int d, int q) {
  return d == 0 ? q * g.dx : (d == 2 ? q * g.dz : g.yf[q]);
}

// A warp takes 32 listed cells.  The normal and the curvature formula run one
// cell per lane; in between the cells' height columns (nine per cell) are dealt
// out to the lanes, whatever cell they belong to, 32 at a time, and leave their
// interface positions in shared memory; the eight around a cell's own column wait
// until that one has proved valid.  A cell without a valid first direction takes
// another round with its second and third.  The 13 class bytes of a column are
// loaded at once, so its two ends are bit scans and not walks of dependent loads.
// Sums are taken in the order of the restatement, so a rounding cannot turn a
// decision.  Bound: instructions of the columns and L1 misses on c's rows; one
// thread per grid cell with serial walks took 10.6 ms on 512x384x256 (0.9 % of
// the lanes busy), three cells per warp with the formula repeated by nine lanes
// 1.29 ms, this form 0.173 ms (0.169 with a cell's nine columns at once, which walks
// the eight in vain where its own is not valid).
constexpr int kCurvWarps = 4;
constexpr int kCurvBlocks = 6;  // blocks per SM
__global__ void __launch_bounds__(32 * kCurvWarps, kCurvBlocks) k_st_curvature(const double *__restrict__ c, Lay Lc,
                                                                  const unsigned char *__restrict__ fl, StGrid g,
                                                                  double eps, const int *__restrict__ list,
                                                                  const int *__restrict__ count,
                                                                  double *__restrict__ kap) {
  __shared__ double Fs[kCurvWarps][32][9];
  __shared__ int bad[kCurvWarps][32], slot[kCurvWarps][32];
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int n = *count;
  const int nwarps = (int)gridDim.x * kCurvWarps;
  for (long w0 = 32L * (blockIdx.x * kCurvWarps + wib); w0 < n; w0 += 32L * nwarps) {
    const int t = list[min(w0 + lane, (long)n - 1)];
    const bool live = w0 + lane < n && (fl[t] & kMixed);
    const int row = t / g.nx, k = row / g.ny;
    const int i = t - row * g.nx, j = row - k * g.ny;
    int ord, sgn;  // direction of each round, two bits each; bit d: the normal's component d is negative
    {
      const int xo[3] = {i > 0 ? i - 1 : g.nx - 1, i, i + 1 < g.nx ? i + 1 : 0};
      const int jo[3] = {clampj(g, j - 1), j, clampj(g, j + 1)};
      const int ko[3] = {k > 0 ? k - 1 : g.nz - 1, k, k + 1 < g.nz ? k + 1 : 0};
      double v[3][3][3];
#pragma unroll
      for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          const double *cr = c + at(Lc, 1, jo[b] + 1, ko[e] + 1);
          const unsigned char *fr = fl + dix(g, 0, jo[b], ko[e]);
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            const double x = cr[xo[a]];  // promoted full cells read as 1 - 2 eps
            v[a][b][e] = (x >= 1.0 - eps && (fr[xo[a]] & kPromoted)) ? 1.0 - 2.0 * eps : x;
          }
        }
      double sx = 0.0, sy = 0.0, sz = 0.0;
#pragma unroll
      for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const double w = (p == 1 ? 2.0 : 1.0) * (q == 1 ? 2.0 : 1.0);
          sx = __dadd_rn(sx, __dmul_rn(w, __dsub_rn(v[2][p][q], v[0][p][q])));
          sy = __dadd_rn(sy, __dmul_rn(w, __dsub_rn(v[p][2][q], v[p][0][q])));
          sz = __dadd_rn(sz, __dmul_rn(w, __dsub_rn(v[p][q][2], v[p][q][0])));
        }
      double ydist = 0.0;
      for (int J = jo[0] + 1; J <= jo[2]; ++J) ydist = __dadd_rn(ydist, g.dyc[J]);
      const double nx = sx / (2.0 * g.dx), ny = jo[2] > jo[0] ? sy / ydist : 0.0, nz = sz / (2.0 * g.dz);
      // maxloc: the first largest, then the first larger of the other two
      const double ax = fabs(nx), ay = fabs(ny), az = fabs(nz);
      int o0 = 0;
      if (ay > ax) o0 = 1;
      if (az > (o0 ? ay : ax)) o0 = 2;
      const int ra = o0 == 0 ? 1 : 0, rb = o0 == 2 ? 1 : 2;
      const bool sw = (rb == 1 ? ay : az) > (ra == 0 ? ax : ay);
      ord = o0 | (sw ? rb : ra) << 2 | (sw ? ra : rb) << 4;
      sgn = (nx >= 0.0 ? 0 : 1) | (ny >= 0.0 ? 0 : 2) | (nz >= 0.0 ? 0 : 4);
    }
    bool found = !live;
    double kv = 0.0;
    for (int r = 0; r < 3; ++r) {
      if (!__any_sync(all, !found)) break;
      bad[wib][lane] = 0;
      __syncwarp();
      int ncol = 0;  // columns of the passes after the first
      for (int pass = 0; pass == 0 || 32 * (pass - 1) < ncol; ++pass) {
        // the first pass walks every open cell's own column, the others the eight
        // around it of the cells where that one is valid
        const int q = 32 * (pass - 1) + lane, e = q & 7;
        const bool have = pass == 0 ? !found : q < ncol;
        const int own = pass == 0 ? lane : (have ? slot[wib][q >> 3] : 0), col = pass == 0 ? 4 : e + (e >= 4);
        const int oi = __shfl_sync(all, i, own), oj = __shfl_sync(all, j, own), ok_ = __shfl_sync(all, k, own);
        const int od = __shfl_sync(all, ord, own) >> (2 * r) & 3, os = __shfl_sync(all, sgn, own);
        if (have) {
          const int d = od, s = os >> d & 1 ? -1 : 1;
          // the column's start cell, one step across the direction
          const int da = col / 3 - 1, db = col % 3 - 1;
          int ci = oi + (d != 0 ? da : 0), cj = oj + (d == 0 ? da : (d == 2 ? db : 0)), ck = ok_ + (d != 2 ? db : 0);
          bool ok = cj >= 0 && cj < g.ny;
          ci = ci < 0 ? ci + g.nx : (ci >= g.nx ? ci - g.nx : ci);
          cj = clampj(g, cj);
          ck = ck < 0 ? ck + g.nz : (ck >= g.nz ? ck - g.nz : ck);
          const int q0 = d == 0 ? ci : (d == 1 ? cj : ck), nd = d == 0 ? g.nx : (d == 1 ? g.ny : g.nz);
          const int dd = d == 0 ? 1 : (d == 1 ? g.nx : g.nx * g.ny);
          const long cd = d == 0 ? 1 : (d == 1 ? Lc.sj : Lc.sk);
          const unsigned char *fr = fl + dix(g, ci, cj, ck);
          const double *cr = c + at(Lc, ci + 1, cj + 1, ck + 1);
          // class nibbles, the cell at -kStColumn steps (away from the full phase) lowest
          unsigned long long w = 0;
          const bool inside = q0 >= kStColumn && q0 + kStColumn < nd;
          if (inside) {
            const unsigned char *f0 = fr - (long)(s * kStColumn) * dd;
            const long sd = (long)s * dd;
            unsigned lo = 0, hi = 0;
  #pragma unroll
            for (int u = 0; u <= 2 * kStColumn; ++u) {
              if (u < 8) lo |= (unsigned)f0[u * sd] << (4 * u);
              else hi |= (unsigned)f0[u * sd] << (4 * (u - 8));
            }
            w = (unsigned long long)hi << 32 | lo;
          } else {  // near a wall, where columns stop, or across a periodic boundary
  #pragma unroll 1
            for (int u = 0; u <= 2 * kStColumn; ++u) {
              int x = q0 + s * (u - kStColumn);
              unsigned f = kMixed;  // beyond a wall: no end of the column
              if (d != 1 || (x >= 0 && x < nd)) {
                x = wrapn(x, nd);
                f = fr[(long)(x - q0) * dd];
              }
              w |= (unsigned long long)f << (4 * u);
            }
          }
          const unsigned long long ones = 0x1111111111111ull;
          // bit 4u: the cell u is full / empty
          const unsigned long long wf = (w >> 1 & ones) >> (4 * kStColumn);
          const unsigned long long we = (~(w | w >> 1) & ones) << (63 - 4 * kStColumn);
          const int tf = wf ? (__ffsll((long long)wf) - 1) >> 2 : -1;  // steps to the first full cell
          const int te = we ? __clzll((long long)we) >> 2 : -1;        // and back to the first empty one
          ok = ok && tf >= 0 && te >= 0;
          double f = 0.0;
          if (ok) {
            double hs = 0.0;
            if (inside && (w & (kPromoted * ones)) == 0) {
              const double *pc = cr - (long)(s * te) * cd;
              const double wd = d == 0 ? g.dx : g.dz;
              int x = q0 - s * te;
              for (int u = te + tf; u >= 0; --u, pc += s * cd, x += s)
                hs = __dadd_rn(hs, __dmul_rn(*pc, d == 1 ? g.dyf[x] : wd));
            } else {
              for (int u = -te; u <= tf; ++u) {
                int x = q0 + s * u;
                if (d != 1) x = wrapn(x, nd);
                const double v = (w >> (4 * (u + kStColumn)) & kPromoted) ? 1.0 - 2.0 * eps : cr[(x - q0) * cd];
                hs = __dadd_rn(hs, __dmul_rn(v, d == 0 ? g.dx : (d == 2 ? g.dz : g.dyf[x])));
              }
            }
            const int qf = q0 + s * tf;  // not wrapped: the nine columns share one frame
            const double xf = face_pos(g, d, s > 0 ? qf + 1 : qf);
            f = s > 0 ? __dsub_rn(xf, hs) : __dadd_rn(xf, hs);
          }
          Fs[wib][own][col] = f;
          if (!ok) bad[wib][own] = 1;
        }
        if (pass == 0) {
          __syncwarp();
          const bool open = !found && !bad[wib][lane];
          const unsigned m = __ballot_sync(all, open);
          if (open) slot[wib][__popc(m & ((1u << lane) - 1u))] = lane;
          ncol = 8 * __popc(m);
          __syncwarp();
        }
      }
      __syncwarp();
      if (!found && !bad[wib][lane]) {
        const int d = ord >> (2 * r) & 3;
        const double(&F)[9] = Fs[wib][lane];
        const double h1m = d != 0 ? g.dx : g.dyc[j], h1p = d != 0 ? g.dx : g.dyc[j + 1];  // across: x, or y
        const double h2m = d != 2 ? g.dz : g.dyc[j], h2p = d != 2 ? g.dz : g.dyc[j + 1];  // across: z, or y
        const double den1 = h1p * h1m * (h1p + h1m), den2 = h2p * h2m * (h2p + h2m);
        const double d1 = (h1m * h1m * F[7] - h1p * h1p * F[1] + (h1p * h1p - h1m * h1m) * F[4]) / den1;
        const double d11 = 2.0 * (h1m * F[7] - (h1p + h1m) * F[4] + h1p * F[1]) / den1;
        const double d2 = (h2m * h2m * F[5] - h2p * h2p * F[3] + (h2p * h2p - h2m * h2m) * F[4]) / den2;
        const double d22 = 2.0 * (h2m * F[5] - (h2p + h2m) * F[4] + h2p * F[3]) / den2;
        const double d12 = (F[8] - F[6] - F[2] + F[0]) / ((h1p + h1m) * (h2p + h2m));
        const double num = d11 * (1.0 + d2 * d2) + d22 * (1.0 + d1 * d1) - 2.0 * d1 * d2 * d12;
        const double gg = 1.0 + d1 * d1 + d2 * d2;
        kv = ((sgn >> d & 1) ? -1 : 1) * num / (gg * sqrt(gg));
        found = true;
      }
      __syncwarp();  // the round's positions are read before the next round's are written
    }
    if (live) kap[t] = kv;
  }
}

// sigma * k_f * grad c of the face between cells p and q (dense indices, c at
// cp_ and cq_): k_f the mean of two mixed cells' curvatures, else the mixed
// one's, else 0.
__device__ __forceinline__ double face_force(double sigma, unsigned fp, unsigned fq, const double *__restrict__ kap,
                                             long p, long q, double cp, double cq, double dc, double eps) {
  const bool mp = fp & kMixed, mq = fq & kMixed;
  const double kp = mp ? kap[p] : 0.0, kq = mq ? kap[q] : 0.0;
  if (fp & kPromoted) cp = 1.0 - 2.0 * eps;
  if (fq & kPromoted) cq = 1.0 - 2.0 * eps;
  return sigma * ((mp && mq) ? 0.5 * (kq + kp) : (mq ? kq : kp)) * ((cq - cp) / dc);
}

// A face value into its element of component D and the element's periodic
// images in x and z (halos included).
template <int D>
__device__ __forceinline__ void put_face(const StOut &o, const StGrid &g, int hd, int i, int j, int k, double v) {
  const Lay &L = o.L[D];
  const int ihi = g.nx + hd, khi = g.nz + hd;
  int i0 = i, k0 = k;
  while (i0 - g.nx >= L.ilo) i0 -= g.nx;
  while (k0 - g.nz >= L.klo) k0 -= g.nz;
  for (int kk = k0; kk <= khi; kk += g.nz)
    for (int ii = i0; ii <= ihi; ii += g.nx) o.s[D][at(L, ii, j, kk)] = v;
}

// The faces of the listed cells, one cell per thread: its upper faces, and the
// lower ones where the cell below is not listed itself.  Every other face was
// filled with zeros (component d, face index along d in Fortran counting 0..n,
// the other two indices wrap periodically; y faces 0 and ny and the y ghost rows
// stay zero).  A pass over all faces that read the class bytes and computed the
// force where it met an interface took 0.35 ms on 512x384x256: one or two lanes
// of a warp had a force to compute.  This one takes 0.041 ms, and the
// fill hides under the classification.
__global__ void __launch_bounds__(256) k_st_faces(const double *__restrict__ c, Lay Lc,
                                                  const unsigned char *__restrict__ fl,
                                                  const double *__restrict__ kap, StGrid g, double eps, double sigma,
                                                  const int *__restrict__ list, const int *__restrict__ count, int hd,
                                                  StOut o) {
  const int n = *count;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) {
    const int t = list[e], row = t / g.nx, k = row / g.ny, i = t - row * g.nx, j = row - k * g.ny;
    const int im = i > 0 ? i - 1 : g.nx - 1, ip = i + 1 < g.nx ? i + 1 : 0;
    const int km = k > 0 ? k - 1 : g.nz - 1, kp = k + 1 < g.nz ? k + 1 : 0;
    const unsigned f0 = fl[t];
    const double c0 = c[at(Lc, i + 1, j + 1, k + 1)];
    auto upper = [&](int ii, int jj, int kk, double dc) {
      const long q = dix(g, ii, jj, kk);
      return face_force(sigma, f0, fl[q], kap, t, q, c0, c[at(Lc, ii + 1, jj + 1, kk + 1)], dc, eps);
    };
    auto lower = [&](int ii, int jj, int kk, double dc, double *v) {
      const long p = dix(g, ii, jj, kk);
      const unsigned f = fl[p];
      if (f & (kMixed | kWild)) return false;
      *v = face_force(sigma, f, f0, kap, p, t, c[at(Lc, ii + 1, jj + 1, kk + 1)], c0, dc, eps);
      return true;
    };
    double v;
    // Fortran: face i lies between the cells i and i+1
    put_face<0>(o, g, hd, i + 1, j + 1, k + 1, upper(ip, j, k, g.dx));
    if (lower(im, j, k, g.dx, &v)) put_face<0>(o, g, hd, i, j + 1, k + 1, v);
    if (j + 1 < g.ny) put_face<1>(o, g, hd, i + 1, j + 1, k + 1, upper(i, j + 1, k, g.dyc[j + 1]));
    if (j > 0 && lower(i, j - 1, k, g.dyc[j], &v)) put_face<1>(o, g, hd, i + 1, j, k + 1, v);
    put_face<2>(o, g, hd, i + 1, j + 1, k + 1, upper(i, j, kp, g.dz));
    if (lower(i, j, km, g.dz, &v)) put_face<2>(o, g, hd, i + 1, j + 1, k, v);
  }
}

// curvature as a cell field with the layout of c: interior, x/z ghosts periodic, y ghosts 0
__global__ void k_st_kappa_out(const double *__restrict__ kap, const unsigned char *__restrict__ fl, StGrid g,
                               double *__restrict__ out, Lay L, long n) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) {
    const int i = (int)(e % L.sj) + L.ilo, j = (int)((e / L.sj) % (L.sk / L.sj)) + L.jlo, k = (int)(e / L.sk) + L.klo;
    double v = 0.0;
    if (j >= 1 && j <= g.ny) {
      const long t = dix(g, wrapn(i - 1, g.nx), j - 1, wrapn(k - 1, g.nz));
      if (fl[t] & kMixed) v = kap[t];
    }
    out[e] = v;
  }
}

int grid_blocks(long n, int threads) {
  long b = (n + threads - 1) / threads;
  return (int)(b < 148 * 32 ? (b < 1 ? 1 : b) : 148 * 32);
}

}  // namespace

void launch_surface_tension(const double *c, Lay Lc, const StGrid &g, double eps, double sigma, unsigned char *fl,
                            double *kap, int *list, int *count, double *kap_out, Lay Lk, long nk, int hd, double *sx,
                            Lay Lx, long nsx, double *sy, Lay Ly, long nsy, double *sz, Lay Lz, long nsz,
                            cudaStream_t st) {
  const long rows = (long)g.ny * g.nz, most = rows * g.nx;  // most: the longest list
  const StOut o{{sx, sy, sz}, {Lx, Ly, Lz}, {nsx, nsy, nsz}};
  cudaMemsetAsync(count, 0, sizeof(int), st);
  k_st_classify<<<2 * (unsigned)((rows + kRowWarps - 1) / kRowWarps), 32 * kRowWarps, 0, st>>>(c, Lc, g, eps, fl, list,
                                                                                               count, o);
  // the list's length is on the device: grids that fill the chip stride over it
  const unsigned cb = (unsigned)std::min<long>(148 * kCurvBlocks, (most + 32 * kCurvWarps - 1) / (32 * kCurvWarps));
  k_st_curvature<<<cb, 32 * kCurvWarps, 0, st>>>(c, Lc, fl, g, eps, list, count, kap);
  k_st_faces<<<(unsigned)std::min<long>(148 * 6, (most + 255) / 256), 256, 0, st>>>(c, Lc, fl, kap, g, eps, sigma, list,
                                                                                    count, hd, o);
  if (kap_out) k_st_kappa_out<<<grid_blocks(nk, 256), 256, 0, st>>>(kap, fl, g, kap_out, Lk, nk);
}

}  // namespace tbfp
