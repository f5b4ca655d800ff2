// nudge_kernels.cu -- temperature nudging toward values stored along
// trajectories.
//
// Box mode (the reference, Nudging/code/tempvel_nudge.c:1380-1781 read_prtcl):
//   every step each observation's position and temperature are advanced by
//   linear interpolation in time between files written every ntempread steps
//   (with the periodic-x and wall-y jump handling of :1489-1552, :1688-1720);
//   then every node inside the 7x7 box around (round x, round y) gets the
//   running mean tempreadint = (tempreadint*n + T)/(n+1), n = nudge_vol, in
//   the reference's contribution order: observation index k ascending, and
//   per k the main box, then its left and right periodic images.
//   The per-node order is reproduced exactly (FP64 bit-identical): the
//   contributions are binned into 8x8-node cells, each cell sorts its
//   contribution keys (3k + image), and each node walks its cell's sorted
//   list.  Only cells that hold contributions, or held some the step before,
//   touch memory: two launches a step, one that advances the observations and
//   bins them into a few places per cell (and lists the cells it touches),
//   one over the listed cells of this step and the last.  (1680x840, 1600
//   observations: the box launches take 14 us of a step; with a count, a
//   one-block scan of all cells, a fill and a block for every cell they took
//   45, the scan alone 17.)
// Bilinear mode (no reference counterpart): innovation
//   d = alpha (T_obs - T(x_obs)) spread to the 4 cell corners with bilinear
//   weights; contributions are summed in 2^-40 fixed point with integer
//   atomics, so the result does not depend on their order, then added to the
//   post-collision g as w_k * S.
#include <algorithm>

#include "lbrb_internal.cuh"
#include "nudge_dev.cuh"

namespace lbrb {

constexpr int CELL = 8;

// per-observation double arrays in Handle::nb, each of length nobs
enum { NB_OX = 0, NB_OY, NB_OT, NB_FX, NB_FY, NB_FT, NB_XINT, NB_YINT, NB_TINT, NB_DX, NB_DY,
       NB_DT, NB_COUNT };
// per-observation int arrays in Handle::nbi
enum { NBI_CHK = 0, NBI_BC, NBI_XIDX, NBI_YIDX, NBI_COUNT };

// Contributions of a cell: the first BOX_SLOTS in the cell's own slots, the
// rest in BOX_CHAINS chains of the cell, by turns, linked through `link` (a
// contribution's place there: 4 key + its cell's number in its box, at most
// 2 x 2 cells).  A chain's length follows from the cell's count, so heads and
// links are never cleared, and a chain is read by a thread of its own: work in
// proportion to a cell's own contributions, however many all cells have.
// (A whole step with 100,000 observations: 123 us on 512x256 and 196 on
// 1680x840; with one list for all cells, which every full cell searched, 1314
// and 4228; with a count, a scan and a fill of all cells 149 and 204.)
// A step's lists and counters are one of three sets, by `seq` (a count of
// steps, from 1): this step's, the last one's, and the one that this step
// leaves cleared for the next.  The count is in device memory, so that replays
// of a captured step go on from the step before them, whichever it was.  Each
// of its two words is written by the kernel that does not read it.
constexpr int BOX_SLOTS = 8, BOX_CHAINS = 16;
enum { BOX_NCELLS = 0, BOX_NSORT, BOX_NCOUNT = 4 };
enum { BOX_PLACED = 3 * BOX_NCOUNT, BOX_PLACING, BOX_HEAD = 16 };  // words after the counters: steps done, begun

struct BoxView {
  double* nb;
  int* nbi;
  // ny: the handle's rows (of nudge_vol, tempreadint and the cells); nyT:
  // the whole domain's rows (positions and boxes); j0: the handle's first
  // row in the domain (0 unless a y-slab)
  int n, nx, ny, nt, istep, nyT, j0;
  int ncx, ncell;
  int* cnt;      // [3][BOX_NCOUNT], BOX_PLACED, BOX_PLACING
  int* count;    // [ncell] contributions of a cell this step (0 between steps)
  int* stamp;    // [ncell] the last step that touched a cell
  int* slots;    // [ncell][BOX_SLOTS]
  int* cells;    // [3][lcap] cells touched
  int* head;     // [ncell][BOX_CHAINS] newest entry of a chain
  int* link;     // [12 n] the entry before it in its chain
  int* scratch;  // [2][12 n]
  int lcap;
  int* nudge_vol;
  double* tempreadint;
  int pitch;
};

__device__ __forceinline__ double* NB(const BoxView& B, int a) { return B.nb + (size_t)a * B.n; }
__device__ __forceinline__ int* NBI(const BoxView& B, int a) { return B.nbi + (size_t)a * B.n; }

// time interpolation of observation i (read_prtcl's three branches)
__device__ __forceinline__ void box_interp(const BoxView& B, int i) {
  const int nx = B.nx, ny = B.nyT, nt = B.nt;
  double *ox = NB(B, NB_OX), *oy = NB(B, NB_OY), *oT = NB(B, NB_OT);
  double *fx = NB(B, NB_FX), *fy = NB(B, NB_FY), *fT = NB(B, NB_FT);
  double *xint = NB(B, NB_XINT), *yint = NB(B, NB_YINT), *Tint = NB(B, NB_TINT);
  double *dxs = NB(B, NB_DX), *dys = NB(B, NB_DY), *dTs = NB(B, NB_DT);
  int *chk = NBI(B, NBI_CHK), *bc = NBI(B, NBI_BC), *xidx = NBI(B, NBI_XIDX), *yidx = NBI(B, NBI_YIDX);
  const int ph = B.istep % nt;
  if (ph == 1) {
    const int c = chk[i];
    int bci = 0;
    double xread = fx[c];
    double yread = fy[c];
    dxs[i] = (xread - xint[i]) / ((double)nt);
    if (abs((int)(xread - xint[i])) > ((double)nx / 2.0)) {
      if (xread > xint[i]) {
        xread = xread - (double)nx;
        dxs[i] = (xread - xint[i]) / ((double)nt);
      } else {
        xread = xread + (double)nx;
        dxs[i] = (xread - xint[i]) / ((double)nt);
      }
    }
    double xposnow = xint[i] + dxs[i];
    if (xposnow > (double)nx) xposnow = xposnow - (double)nx;
    if (xposnow < 0.0) xposnow = xposnow + (double)nx;
    xint[i] = xposnow;
    dys[i] = (yread - yint[i]) / ((double)nt);
    if (abs((int)(yread - yint[i])) > ((double)ny / 2.0)) {
      bci = 1;
      if (yread > yint[i]) {
        yread = yread - (double)ny + 1.0;
        dys[i] = (yread - yint[i]) / ((double)nt);
      } else {
        yread = yread + (double)ny - 1.0;
        dys[i] = (yread - yint[i]) / ((double)nt);
      }
    }
    double yposnow = yint[i] + dys[i];
    if (yposnow > (double)ny) { yposnow = yposnow - (double)ny + 1.0; bci = 2; }
    if (yposnow < 1.0) { yposnow = yposnow + (double)ny - 1.0; bci = 2; }
    yint[i] = yposnow;
    xidx[i] = (int)round(xposnow);
    yidx[i] = (int)round(yposnow);
    const double Tread = fT[c];
    dTs[i] = (Tread - Tint[i]) / ((double)nt);
    double Tnow = Tint[i] + dTs[i];
    if (bci == 1) Tnow = Tint[i];
    if (bci == 2) { Tnow = fT[c]; bci = 1; }
    Tint[i] = Tnow;
    bc[i] = bci;
    // the loaded file becomes the "last file" (read by the other branches only)
    ox[i] = fx[i];
    oy[i] = fy[i];
    oT[i] = fT[i];
  } else if (ph == 0) {
    const int c = chk[i];
    xint[i] = ox[c];
    yint[i] = oy[c];
    Tint[i] = oT[c];
    xidx[i] = (int)round(ox[c]);
    yidx[i] = (int)round(oy[c]);
  } else {
    double xposnow = xint[i] + dxs[i];
    if (xposnow > (double)nx) xposnow = xposnow - (double)nx;
    if (xposnow < 0.0) xposnow = xposnow + (double)nx;
    xint[i] = xposnow;
    int bci = bc[i];
    double yposnow = yint[i] + dys[i];
    if (yposnow > (double)ny) { yposnow = yposnow - (double)ny + 1.0; bci = 2; }
    if (yposnow < 1.0) { yposnow = yposnow + (double)ny - 1.0; bci = 2; }
    yint[i] = yposnow;
    xidx[i] = (int)round(xposnow);
    yidx[i] = (int)round(yposnow);
    double Tnow = Tint[i] + dTs[i];
    if (bci == 1) Tnow = Tint[i];
    if (bci == 2) { Tnow = oT[chk[i]]; bci = 1; }
    Tint[i] = Tnow;
    bc[i] = bci;
  }
}

// node box of contribution (k, img), reference 1-based node coordinates of
// the whole domain, clipped to its interior; false when empty.  img 0: main 7x7 box; img 1:
// left periodic image (xidx < 4); img 2: right periodic image (xidx > nx-2).
__device__ __forceinline__ bool contrib_box(const BoxView& B, int k, int img, int& xa, int& xb,
                                            int& ya, int& yb) {
  const int xi = NBI(B, NBI_XIDX)[k], yi = NBI(B, NBI_YIDX)[k];
  if (img == 0) {
    xa = xi - 3; xb = xi + 3;
  } else if (img == 1) {
    if (!(xi < 4)) return false;
    xa = B.nx + xi - 3; xb = B.nx + xi;
  } else {
    if (!(xi > B.nx - 2)) return false;
    xa = xi - B.nx; xb = xi - B.nx + 3;
  }
  ya = yi - 3; yb = yi + 3;
  if (xa < 1) xa = 1;
  if (xb > B.nx) xb = B.nx;
  if (ya < 1) ya = 1;
  if (yb > B.nyT) yb = B.nyT;
  return xa <= xb && ya <= yb;
}

// one thread per observation: its new position and temperature, then its
// contributions into the cells they reach
__global__ void __launch_bounds__(32) box_bin_kernel(const BoxView B) {
  pdl_wait();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= B.n) return;
  const int seq = B.cnt[BOX_PLACED] + 1;
  if (k == 0) B.cnt[BOX_PLACING] = seq;
  box_interp(B, k);
  const int set = seq % 3;
  int* cnt = B.cnt + set * BOX_NCOUNT;
  for (int img = 0; img < 3; img++) {
    int xa, xb, ya, yb;
    if (!contrib_box(B, k, img, xa, xb, ya, yb)) continue;
    // the rows of this handle (a y-slab bins only what reaches its rows)
    ya = max(ya, B.j0 + 1);
    yb = min(yb, B.j0 + B.ny);
    if (ya > yb) continue;
    const int ca = (xa - 1) / CELL, cb = (xb - 1) / CELL;
    const int ra = (ya - 1 - B.j0) / CELL, rb = (yb - 1 - B.j0) / CELL;
    for (int cy = ra; cy <= rb; cy++)
      for (int cx = ca; cx <= cb; cx++) {
        const int c = cy * B.ncx + cx, key = 3 * k + img;
        const int at = atomicAdd(&B.count[c], 1);
        if (at == 0) {
          B.stamp[c] = seq;
          B.cells[(size_t)set * B.lcap + atomicAdd(&cnt[BOX_NCELLS], 1)] = c;
        }
        if (at < BOX_SLOTS) {
          B.slots[(size_t)c * BOX_SLOTS + at] = key;
        } else {
          const int e = 4 * key + 2 * (cy - ra) + (cx - ca);
          B.link[e] = atomicExch(&B.head[(size_t)c * BOX_CHAINS + (at - BOX_SLOTS) % BOX_CHAINS], e);
        }
      }
  }
}

// one block of CELL*CELL threads per listed cell: sort the cell's keys, then
// every node applies the running mean in key order; cells of the last step
// that this one did not touch are cleared
__global__ void __launch_bounds__(CELL * CELL) box_cells_kernel(const BoxView B) {
  pdl_wait();
  constexpr int NT = CELL * CELL;
  __shared__ int keys[BOX_SLOTS];
  __shared__ int base;
  const int tid = threadIdx.x;
  // (the three sets' counts loaded with the step, not after it)
  const int seq = B.cnt[BOX_PLACING];
  const int n0 = B.cnt[BOX_NCELLS], n1 = B.cnt[BOX_NCOUNT + BOX_NCELLS], n2 = B.cnt[2 * BOX_NCOUNT + BOX_NCELLS];
  const int set = seq % 3, last = (seq + 2) % 3, next = (seq + 1) % 3;
  const int ncur = set == 0 ? n0 : (set == 1 ? n1 : n2), nlast = last == 0 ? n0 : (last == 1 ? n1 : n2);
  if (blockIdx.x == 0 && tid < BOX_NCOUNT) B.cnt[next * BOX_NCOUNT + tid] = 0;
  if (blockIdx.x == 0 && tid == 0) B.cnt[BOX_PLACED] = seq;
  const double* Tint = NB(B, NB_TINT);
  for (int it = blockIdx.x; it < ncur + nlast; it += gridDim.x) {
    const bool now = it < ncur;
    const int c = now ? B.cells[(size_t)set * B.lcap + it] : B.cells[(size_t)last * B.lcap + it - ncur];
    if (!now && B.stamp[c] == seq) continue;  // (listed in this step too)
    const int cx = c % B.ncx, cy = c / B.ncx;
    const int i = cx * CELL + (tid % CELL) + 1;  // reference node coordinates (of the domain)
    const int j = B.j0 + cy * CELL + (tid / CELL) + 1;
    int nv = 0;
    double tri = 0.0;
    if (now) {
      const int cnt = B.count[c];
      const int* list = keys;
      if (cnt <= BOX_SLOTS) {
        // rank sort (keys are unique)
        if (tid < cnt) {
          const int key = B.slots[(size_t)c * BOX_SLOTS + tid];
          int rank = 0;
          for (int b = 0; b < cnt; b++) rank += (B.slots[(size_t)c * BOX_SLOTS + b] < key);
          keys[rank] = key;
        }
        __syncthreads();
      } else {
        // more than the slots hold: the cell's keys into scratch, then ranked there
        if (tid == 0) base = atomicAdd(&B.cnt[set * BOX_NCOUNT + BOX_NSORT], cnt);
        __syncthreads();
        int* raw = B.scratch + base;
        int* sorted = raw + (size_t)12 * B.n;
        if (tid < BOX_SLOTS) raw[tid] = B.slots[(size_t)c * BOX_SLOTS + tid];
        if (tid < BOX_CHAINS) {
          int e = B.head[(size_t)c * BOX_CHAINS + tid];
          for (int a = BOX_SLOTS + tid; a < cnt; a += BOX_CHAINS) {
            raw[a] = e >> 2;
            e = B.link[e];
          }
        }
        __syncthreads();
        for (int a = tid; a < cnt; a += NT) {
          const int key = raw[a];
          int rank = 0;
          for (int b = 0; b < cnt; b++) rank += (raw[b] < key);
          sorted[rank] = key;
        }
        __syncthreads();
        list = sorted;
      }
      for (int a = 0; a < cnt; a++) {
        const int key = list[a];
        const int k = key / 3, img = key - 3 * k;
        int xa, xb, ya, yb;
        if (!contrib_box(B, k, img, xa, xb, ya, yb)) continue;
        if (i >= xa && i <= xb && j >= ya && j <= yb) {
          tri = (tri * (double)nv + Tint[k]) / ((double)nv + 1.0);
          nv = nv + 1;
        }
      }
      __syncthreads();  // (every thread has the count and the keys)
      if (tid == 0) B.count[c] = 0;
    }
    if (i <= B.nx && j <= B.j0 + B.ny) {
      const size_t q = (size_t)(j - 1 - B.j0) * B.pitch + (i - 1);
      B.nudge_vol[q] = nv;
      B.tempreadint[q] = tri;
    }
  }
}

// ints of the cell lists for n observations over ncell cells: counters,
// counts, stamps, slots, chain heads, three lists, links, scratch
static size_t box_lcap(int n, int ncell) { return std::min((size_t)ncell, (size_t)12 * n); }
size_t box_cell_ints(int n, int ncell) {
  return BOX_HEAD + (size_t)ncell * (2 + BOX_SLOTS + BOX_CHAINS) + 3 * box_lcap(n, ncell) + (size_t)3 * 12 * n;
}

// `work`: box_cell_ints ints, zero at the start of the run
cudaError_t launch_box_nudge(double* nb, int* nbi, int n, int nx, int ny, int ny_total, int j0, int nt, int istep,
                             int ncx, int ncy, int* work, int* nudge_vol, double* tempreadint, int pitch,
                             cudaStream_t s, bool pdl) {
  const int ncell = ncx * ncy;
  const size_t lcap = box_lcap(n, ncell);
  BoxView B{nb, nbi, n, nx, ny, nt, istep, ny_total, j0, ncx, ncell};
  B.cnt = work;
  B.link = work + BOX_HEAD;
  B.scratch = B.link + (size_t)12 * n;
  B.count = B.scratch + (size_t)2 * 12 * n;
  B.stamp = B.count + ncell;
  B.slots = B.stamp + ncell;
  B.head = B.slots + (size_t)ncell * BOX_SLOTS;
  B.cells = B.head + (size_t)ncell * BOX_CHAINS;
  B.lcap = (int)lcap;
  B.nudge_vol = nudge_vol;
  B.tempreadint = tempreadint;
  B.pitch = pitch;
  // (32 threads a block: a few thousand observations still reach most SMs)
  const cudaError_t e = launch_k(box_bin_kernel, (n + 31) / 32, 32, 0, s, pdl, B);
  if (e != cudaSuccess) return e;
  const int blocks = (int)std::min((size_t)2 * lcap, (size_t)148 * 16);
  return launch_k(box_cells_kernel, blocks, CELL * CELL, 0, s, pdl, B);
}

// ------------------------------------------------------------ bilinear mode
template <typename Real>
__global__ void obs_scatter_kernel(const Real* __restrict__ T, int nx, int ny, int pitch,
                                   const double* __restrict__ ox, const double* __restrict__ oy,
                                   const double* __restrict__ oT, int nobs, double alpha,
                                   unsigned long long* __restrict__ acc, unsigned* dflags) {
  pdl_wait();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nobs) return;
  obs_scatter_one(T, nx, ny, pitch, ox[p], oy[p], oT[p], alpha, acc, dflags);
}

template <typename Real>
__global__ void obs_apply_kernel(Real* __restrict__ g, size_t plane, int nx, int ny, int pitch,
                                 const double* __restrict__ ox, const double* __restrict__ oy,
                                 int nobs, unsigned long long* __restrict__ acc) {
  pdl_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 4 * nobs) return;
  const int p = t >> 2;
  obs_apply_one(g, plane, nx, ny, pitch, ox[p], oy[p], t & 3, acc);
}

// Two-step launch of a nudged run: step n's innovations before the launch
// (four threads per observation, obs_pre_corner in nudge_dev.cuh), and the
// clearing of their sums and mask bits after it
template <typename Real>
__global__ void __launch_bounds__(128) obs_pre4_kernel(const LBView<Real> V, const double* __restrict__ ox,
                                                       const double* __restrict__ oy, const double* __restrict__ oT,
                                                       int nobs, double alpha, unsigned long long* __restrict__ acc,
                                                       unsigned* __restrict__ mask, unsigned* dflags) {
  pdl_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int p = t >> 2;
  const bool live = p < nobs;
  obs_pre_corner(V, live, live ? ox[p] : 0.0, live ? oy[p] : 0.0, live ? oT[p] : 0.0, alpha, t & 3, acc, mask,
                 dflags);
}

// after a nudged two-step launch: step n+1's apply pass (acc) and the
// clearing of step n's in-launch sums and mask bits (acc2, mask) in one
// launch -- corner t & 3 of observation t >> 2 of each step
template <typename Real>
__global__ void obs_apply_clear_kernel(Real* __restrict__ g, size_t plane, int nx, int ny, int pitch,
                                       const double* __restrict__ ox2, const double* __restrict__ oy2, int nobs,
                                       unsigned long long* __restrict__ acc, const double* __restrict__ ox1,
                                       const double* __restrict__ oy1, unsigned long long* __restrict__ acc2,
                                       unsigned* __restrict__ mask) {
  pdl_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 4 * nobs) return;
  const int p = t >> 2;
  const double x1 = ox1[p], y1 = oy1[p], x2 = ox2[p], y2 = oy2[p];
  obs_clear_one(nx, ny, pitch, x1, y1, t & 3, acc2, mask);
  obs_apply_one(g, plane, nx, ny, pitch, x2, y2, t & 3, acc);
}

cudaError_t launch_obs_pre_fp32(const LBView<float>& V, const double* ox, const double* oy, const double* oT,
                                int nobs, double alpha, long long* acc, unsigned* mask, unsigned* dflags,
                                cudaStream_t s, bool pdl) {
  if (nobs <= 0) return cudaSuccess;
  return launch_k(obs_pre4_kernel<float>, (4 * nobs + 127) / 128, 128, 0, s, pdl, V, ox, oy, oT, nobs, alpha,
                  reinterpret_cast<unsigned long long*>(acc), mask, dflags);
}
cudaError_t launch_obs_pre_fp64(const LBView<double>& V, const double* ox, const double* oy, const double* oT,
                                int nobs, double alpha, long long* acc, unsigned* mask, unsigned* dflags,
                                cudaStream_t s, bool pdl) {
  if (nobs <= 0) return cudaSuccess;
  return launch_k(obs_pre4_kernel<double>, (4 * nobs + 127) / 128, 128, 0, s, pdl, V, ox, oy, oT, nobs, alpha,
                  reinterpret_cast<unsigned long long*>(acc), mask, dflags);
}
cudaError_t launch_bilinear_nudge_clear(void* T, void* g, bool fp32, size_t plane, int nx, int ny, int pitch,
                                        const double* ox, const double* oy, const double* oT, int nobs, double alpha,
                                        long long* acc, const double* ox1, const double* oy1, long long* acc2,
                                        unsigned* mask, unsigned* dflags, cudaStream_t s, bool pdl) {
  if (nobs <= 0) return cudaSuccess;
  const int tb = 128;
  unsigned long long* a = reinterpret_cast<unsigned long long*>(acc);
  unsigned long long* a2 = reinterpret_cast<unsigned long long*>(acc2);
  auto go = [&](auto zero) -> cudaError_t {
    using Real = decltype(zero);
    cudaError_t e = launch_k(obs_scatter_kernel<Real>, (nobs + tb - 1) / tb, tb, 0, s, pdl, (const Real*)T, nx, ny,
                             pitch, ox, oy, oT, nobs, alpha, a, dflags);
    if (e != cudaSuccess) return e;
    return launch_k(obs_apply_clear_kernel<Real>, (4 * nobs + tb - 1) / tb, tb, 0, s, pdl, (Real*)g, plane, nx, ny,
                    pitch, ox, oy, nobs, a, ox1, oy1, a2, mask);
  };
  return fp32 ? go(0.f) : go(0.0);
}

// y-slab: the observations' innovations read T of the whole domain through
// a table of row pointers (one per global row); the slab scatters to and
// applies at the corners in its own rows only
template <typename Real>
__global__ void obs_scatter_slab_kernel(const Real* const* __restrict__ Trow, int nx, int ny_total, int pitch,
                                        const double* __restrict__ ox, const double* __restrict__ oy,
                                        const double* __restrict__ oT, int nobs, double alpha,
                                        unsigned long long* __restrict__ acc, unsigned* dflags, int j0, int nyl) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nobs) return;
  obs_scatter_rows([&](int j, int i) { return Trow[j][i]; }, nx, ny_total, pitch, ox[p], oy[p], oT[p], alpha, acc,
                   dflags, j0, nyl);
}

template <typename Real>
__global__ void obs_apply_slab_kernel(Real* __restrict__ g, size_t plane, int nx, int ny_total, int pitch,
                                      const double* __restrict__ ox, const double* __restrict__ oy, int nobs,
                                      unsigned long long* __restrict__ acc, int j0, int nyl) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 4 * nobs) return;
  const int p = t >> 2;
  obs_apply_one(g, plane, nx, ny_total, pitch, ox[p], oy[p], t & 3, acc, j0, nyl);
}

cudaError_t launch_bilinear_nudge_slab(const void* Trows, void* g, bool fp32, size_t plane, int nx, int ny_total,
                                       int j0, int nyl, int pitch, const double* ox, const double* oy,
                                       const double* oT, int nobs, double alpha, long long* acc, unsigned* dflags,
                                       cudaStream_t s) {
  if (nobs <= 0) return cudaSuccess;
  const int tb = 128;
  unsigned long long* a = reinterpret_cast<unsigned long long*>(acc);
  auto go = [&](auto zero) {
    using Real = decltype(zero);
    obs_scatter_slab_kernel<Real><<<(nobs + tb - 1) / tb, tb, 0, s>>>(
        (const Real* const*)Trows, nx, ny_total, pitch, ox, oy, oT, nobs, alpha, a, dflags, j0, nyl);
    obs_apply_slab_kernel<Real><<<(4 * nobs + tb - 1) / tb, tb, 0, s>>>((Real*)g, plane, nx, ny_total, pitch, ox,
                                                                       oy, nobs, a, j0, nyl);
  };
  if (fp32) go(0.f);
  else go(0.0);
  return cudaGetLastError();
}

cudaError_t launch_bilinear_nudge(void* T, void* g, bool fp32, size_t plane, int nx, int ny,
                                  int pitch, const double* ox, const double* oy, const double* oT,
                                  int nobs, double alpha, long long* acc, unsigned* dflags,
                                  cudaStream_t s, bool pdl) {
  if (nobs <= 0) return cudaSuccess;
  const int tb = 128;
  unsigned long long* a = reinterpret_cast<unsigned long long*>(acc);
  auto go = [&](auto zero) -> cudaError_t {
    using Real = decltype(zero);
    cudaError_t e = launch_k(obs_scatter_kernel<Real>, (nobs + tb - 1) / tb, tb, 0, s, pdl, (const Real*)T, nx, ny,
                             pitch, ox, oy, oT, nobs, alpha, a, dflags);
    if (e != cudaSuccess) return e;
    return launch_k(obs_apply_kernel<Real>, (4 * nobs + tb - 1) / tb, tb, 0, s, pdl, (Real*)g, plane, nx, ny, pitch,
                    ox, oy, nobs, a);
  };
  return fp32 ? go(0.f) : go(0.0);
}

}  // namespace lbrb
