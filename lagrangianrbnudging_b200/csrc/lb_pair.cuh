// lb_pair.cuh -- device code of the two-step launches shared by the
// single-run kernels (lb_kernels.cu: lb_pair_kernel, lb_wave2_kernel, lb_wave4_kernel) and
// the ensemble's two-step kernels (ensemble_kernels.cu): the ghost rows of a
// y-slab, the nudging sums of a nudged run, one tile block and one marching
// block.
//
// Reference semantics: as lb_kernels.cu (temppart_dump.c:744-1341, the loop
// body :1674-1759); two steps here equal two single steps bit for bit.
#pragma once

#include <type_traits>

#include "lb_node.cuh"

namespace lbrb {

// On a y-slab, the ring row outside the slab (row -1 or ny) is the
// neighbour's boundary row r1: its populations of step n-1 come from the
// ghost block (SLAB_GH2_PLANES planes: r1's crossing populations, its k = 0,
// 1, 3, its F, then the crossing populations of the row r2 beyond), except
// those it pulls from this slab's own boundary row.  Neither r1 nor r2 is a
// wall row (slabs hold at least three rows).
template <typename Real, typename Off>
__device__ __forceinline__ void pull_ghost_row(const LBView<Real>& V, bool lo, int x, Real* fs, Real* gs, Real& Fy) {
  const Real* G = lo ? V.gh2_lo : V.gh2_hi;
  const int nx = V.nx;
  const int xl = (x == 0) ? nx - 1 : x - 1, xr = (x == nx - 1) ? 0 : x + 1;
  const Off pl = (Off)V.plane, own = (Off)(lo ? 0 : V.ny - 1) * (Off)V.pitch;
  static_for<NPOP>([&](auto kc) {
    constexpr int k = decltype(kc)::value;
    const int xs = icx(k) == 1 ? xl : (icx(k) == -1 ? xr : x);
    if constexpr (icy(k) == 0) {
      constexpr int m = k == 0 ? 0 : (k == 1 ? 1 : 2);
      fs[k] = G[(size_t)(6 + m) * nx + xs];
      gs[k] = G[(size_t)(9 + m) * nx + xs];
    } else {
      // from this slab's boundary row (k moving away from it), else from r2
      const bool from_own = lo ? icy(k) == -1 : icy(k) == 1;
      constexpr int slot = (k == 2 || k == 4) ? 0 : ((k == 5 || k == 7) ? 1 : 2);
      if (from_own) {
        fs[k] = V.fsrc[(Off)k * pl + own + (Off)xs];
        gs[k] = V.gsrc[(Off)k * pl + own + (Off)xs];
      } else {
        fs[k] = G[(size_t)(13 + slot) * nx + xs];
        gs[k] = G[(size_t)(16 + slot) * nx + xs];
      }
    }
  });
  Fy = G[(size_t)12 * nx + x];
}

// A bilinear-nudged run's two-step launch: the nudging sum of step n at
// node (y, x) (element offset o), 0 where the mask has no bit or the sum is
// 0 (the apply pass of a single step skips those nodes too)
template <typename Real>
__device__ __forceinline__ long long pair_nudge_sum(const LBView<Real>& V, int y, int x, size_t o) {
  if (!V.nmask || y < 0 || y >= V.ny) return 0;
  const unsigned w = V.nmask[(size_t)y * (size_t)(V.pitch >> 5) + (size_t)(x >> 5)];
  if (!((w >> (x & 31)) & 1u)) return 0;
  return (long long)V.nacc[o];
}

// ------------------------------------------------ two steps per launch, tile
// Temporal blocking of two steps n, n+1 (Dirichlet walls, no ghost rows, no
// nudging in between).  A block owns a TX x TY tile.  Phase 1 computes step n
// at the tile and a one-node ring around it (x wrapped, rows outside the
// domain skipped) from HBM, exactly as lb_update_node does, and keeps the
// post-collision populations in shared memory; at the tile it also stores
// u^n, v^n (and T^n on a record step) to HBM through V1, and keeps the next
// buoyancy F^{n+1} in shared memory.  Phase 2 computes step n+1 at the tile,
// pulling from shared memory with the same wall rules as pull_node (bounce-back
// from the node's own opposite population, anti-bounce-back for g), and
// stores through V2.  Populations and F cross HBM once per two steps; the
// ring is recomputed (34 x 10 nodes for a 32 x 8 tile).  The per-node
// arithmetic is lb_update_node's, so two steps here equal two launches of
// lb_node_kernel bit for bit.
// On a y-slab the ring rows beyond an inner boundary come from the ghost
// blocks (pull_ghost_row).

// shared memory of tile_block: the ring of step-n populations, then F^{n+1}
template <typename Real, int TX, int TY>
constexpr size_t tile_smem_bytes() {
  return ((size_t)2 * NPOP * (TX + 2) * (TY + 2) + (size_t)TX * TY) * sizeof(Real);
}

// One block's tile [x0, x0 + TX) x [y0, y0 + TY); smem: tile_smem_bytes<Real,
// TX, TY>() of shared memory.  NT threads per block: TX * TY (phase 1 takes
// the region in passes), or one per region node rounded to whole warps
// (phase 1 in one pass; phase 2 leaves the rest idle)
template <typename Real, int TX, int TY, int NT, typename Off>
__device__ __forceinline__ void tile_block(const LBView<Real>& V1, const LBView<Real>& V2, int x0, int y0,
                                           unsigned char* smem) {
  constexpr int RX = TX + 2, RY = TY + 2, RN = RX * RY;
  Real* S = reinterpret_cast<Real*>(smem);  // [2 * NPOP][RY][RX]: f then g of step n
  Real* SF = S + 2 * NPOP * RN;             // [TY][TX]: F^{n+1} at the tile
  const int nx = V1.nx, ny = V1.ny;
  const int ncols = min(TX, nx - x0), nrows = min(TY, ny - y0);
  const Off pitch = (Off)V1.pitch;
  // y-slab: the rows beyond an inner boundary are computed from ghost blocks
  const bool glo = V1.gh2_lo != nullptr, ghi = V1.gh2_hi != nullptr;
  // FP64: a full tile whose ring, and the ring's pulls, lie strictly inside
  // the domain (no x wrap, no wall row, no slab ghost row) in a run without
  // in-launch nudging sums takes phase 1 by fixed offsets from each node:
  // the values pull_node's interior path reads, without its bounds, wrap and
  // wall logic (block-uniform).  (In FP32 the second copy of the phase made
  // the launch 10% slower, so FP32 keeps the one general phase.)
  const bool fast = ncols == TX && nrows == TY && x0 >= 2 && x0 + TX + 1 <= nx - 1 && y0 >= 2 &&
                    y0 + TY + 1 <= ny - 1 && !V1.nmask;
  auto phase1 = [&](auto fastc) {
    constexpr bool FAST = decltype(fastc)::value;
    for (int q = threadIdx.x; q < RN; q += NT) {
      const int lx = q % RX, ly = q / RX;
      const int jg = y0 - 1 + ly;
      Real fs[NPOP], gs[NPOP];
      Real Fy, r, u, v, t;
      Off o;
      long long nsum = 0;
      double nsv = 0.0;
      if constexpr (FAST) {
        const int xg = x0 - 1 + lx;
        o = (Off)jg * pitch + (Off)xg;
        const Off pl = (Off)V1.plane;
        static_for<NPOP>([&](auto kc) {
          constexpr int k = decltype(kc)::value;
          const Off src = (Off)k * pl + o + (Off)(-icy(k) * V1.pitch - icx(k));  // (modular: a negative shift wraps)
          fs[k] = __ldcs(V1.fsrc + src);
          gs[k] = __ldcs(V1.gsrc + src);
        });
        Fy = V1.Fin[o];
      } else {
        if (lx > ncols + 1 || ly > nrows + 1 || jg < (glo ? -1 : 0) || jg > (ghi ? ny : ny - 1)) continue;
        int xg = x0 - 1 + lx;
        if (xg < 0) xg += nx;
        else if (xg >= nx) xg -= nx;
        o = (Off)(jg < 0 ? 0 : (jg >= ny ? ny - 1 : jg)) * pitch + (Off)xg;  // (ring rows of a slab: no stores)
        if (jg < 0 || jg >= ny) {
          pull_ghost_row<Real, Off>(V1, jg < 0, xg, fs, gs, Fy);
        } else {
          pull_node<Real, LBRB_TWALL_DIRICHLET, Off, true>(V1, jg, xg, fs, gs);
          dirichlet_walls(V1, jg, gs);
          Fy = V1.Fin[o];
        }
        // (nudged run: step n's sums join g after the collision, as the apply pass does)
        if (V1.nmask) {
          nsum = pair_nudge_sum(V1, jg, xg, (size_t)o);
          if (nsum != 0) nsv = (double)nsum * (1.0 / FIX_SCALE);
        }
      }
      lb_collide<Real, false>(
          V1, (size_t)o, fs, gs, Fy, r, u, v, t, [&](int k, Real val) { S[(k * RY + ly) * RX + lx] = val; },
          [&](int k, Real val) {
            if (!FAST && nsum != 0) val = val + nudge_increment<Real>(k, nsv);
            S[((NPOP + k) * RY + ly) * RX + lx] = val;
          });
      if (lx >= 1 && lx <= ncols && ly >= 1 && ly <= nrows) {
        SF[(ly - 1) * TX + (lx - 1)] = Fy;
        if (V1.write_F) V1.Fout[o] = Fy;
        if (V1.write_uv) {
          V1.u[o] = u;
          V1.v[o] = v;
        }
        if (V1.write_rt & 1) V1.T[o] = t;
        if (V1.write_rt & 2) V1.rho[o] = r;
      }
    }
  };
  if constexpr (std::is_same<Real, double>::value) {
    if (fast) phase1(std::true_type{});
    else phase1(std::false_type{});
  } else {
    phase1(std::false_type{});
  }
  __syncthreads();
  if (threadIdx.x >= TX * TY) return;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  if (tx >= ncols || ty >= nrows) return;
  const int x = x0 + tx, j = y0 + ty;
  Real fs[NPOP], gs[NPOP];
  // a tile whose rows and their neighbours all lie in the domain (or beyond
  // an inner slab edge) pulls with no wall rule (block-uniform)
  const bool inner = (y0 > 0 || glo) && (y0 + nrows < ny || ghi);
  if (inner) {
    static_for<NPOP>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      const int lx = tx + 1 - icx(k), ly = ty + 1 - icy(k);
      fs[k] = S[(k * RY + ly) * RX + lx];
      gs[k] = S[((NPOP + k) * RY + ly) * RX + lx];
    });
  } else {
    static_for<NPOP>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      const int js = j - icy(k);
      if ((js < 0 && !glo) || (js >= ny && !ghi)) {
        fs[k] = S[(opp(k) * RY + ty + 1) * RX + tx + 1];
        gs[k] = Real(0);
      } else {
        const int lx = tx + 1 - icx(k), ly = ty + 1 - icy(k);
        fs[k] = S[(k * RY + ly) * RX + lx];
        gs[k] = S[((NPOP + k) * RY + ly) * RX + lx];
      }
    });
    dirichlet_walls(V2, j, gs);
  }
  lb_finish_node<Real, false, Off>(V2, (Off)j * pitch + (Off)x, fs, gs, SF[ty * TX + tx]);
}

// -------------------------- S steps per launch, one warp per strip, two nodes per thread
// A warp owns a strip of up to WAVE_COLS<S> columns [x0, x0 + ncols) and a
// chunk of rows [ya, ya + Hc), and walks up it one row per iteration: level 1
// computes step n at row y, level 2 step n+1 at row y - 1, ..., level S step
// n+S-1 at row y - S + 1, which it stores.  No other warp takes part, so
// there is no block barrier.  Lane l holds a pair of columns at every level,
// (p, p + 1) with p = x0 - (S - s) + 2l at level s: a level's pair starts one
// column right of the level's before it, so of the populations streaming
// into it those with c_x = +1 come from the lane's own pair of the level
// before, those with c_x = -1 from lane l + 1's pair, and those with c_x = 0
// one from each.  In y, populations with c_y = -1 come from the row the level
// before has just computed (registers, shuffles), c_y = 0 from the row before
// it and c_y = +1 from the one before that: those wait in the warp's shared
// memory (1 and 2 rows deep).  Level s has 32 - s lanes, so a strip is
// 2 (32 - S) columns, and recomputes S - s rows beyond each end of its chunk.
// Level 1's inputs come through D stages of shared memory filled by 16-byte
// asynchronous copies: a row's 64 columns from x0 - S (a multiple of 4, so x0
// is 2 mod 4 for S = 2 and 0 mod 4 for S = 4), each population from the row
// it streams out of; in FP32 one instruction copies a population of f (lanes
// 0-15) and of g (lanes 16-31).  Strips wrap around in x, pair by pair.
// FP32 collides the pair in two-lane arithmetic (node_shift2), FP64 one node
// after the other in the reference's order (node_ref).
// Wall rows bounce back from the node's own populations: at row 0 the slot
// of row -1 takes the level's f4, f7, f8 instead (read at the node's own
// columns); at the top the c_y = +1 populations of the row itself are there.
// Rows outside the domain, and a level's iterations before its first inputs,
// run on whatever is in their places: nothing of them is stored, and no row of
// the domain reads them (a level skips the arithmetic of the latter).
// Level 1 takes the domain's first and last row, and the ghost rows of a
// y-slab (S = 2), by pull_node / pull_ghost_row instead of a stage.
template <int S>
constexpr int WAVE_COLS = 2 * (32 - S);
template <int S>
constexpr int WAVE_X0 = S % 4;  // first strip's x0

// shared memory of one warp: D stages of 19 planes of 64 columns; per level s
// but the last, c_y = 0 populations and F of a row and c_y = +1 populations
// of 2 rows, 2 (32 - s) columns each; a few floats that lanes past a level's
// last pair may read (12 warps of S = 4, D = 1 just fit an SM this way)
constexpr int WAVE_SLOTS = 7 + 2 * 6, WAVE_STAGE = 2 * NPOP + 1;
constexpr int wave_cols(int level) { return 2 * (32 - level); }
constexpr int wave_lag(int level) { return level == 0 ? 0 : wave_lag(level - 1) + WAVE_SLOTS * wave_cols(level); }
template <typename Real, int S, int D>
constexpr size_t wave_smem_bytes() {
  return ((size_t)D * WAVE_STAGE * 64 + wave_lag(S - 1) + 8 + 3) / 4 * 4 * sizeof(Real);
}

template <typename Real>
struct PairOf { using type = float2; };
template <>
struct PairOf<double> { using type = double2; };
template <typename Real>
using Pair = typename PairOf<Real>::type;
__device__ __forceinline__ float2 pair_of(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 pair_of(double a, double b) { return make_double2(a, b); }
// the collision of a pair of nodes
__device__ __forceinline__ void collide_pair(const LBView<float>& V, float2* f, float2* g, float2& F, float2& r,
                                             float2& u, float2& v, float2& t) {
  node_shift2(V, f, g, F, r, u, v, t);
}
__device__ __forceinline__ void collide_pair(const LBView<double>& V, double2* f, double2* g, double2& F, double2& r,
                                             double2& u, double2& v, double2& t) {
  double fa[NPOP], ga[NPOP];
  auto none = [](int, double) {};
#pragma unroll
  for (int k = 0; k < NPOP; k++) fa[k] = f[k].x, ga[k] = g[k].x;
  node_ref<false>(V, 0, fa, ga, F.x, r.x, u.x, v.x, t.x, none, none);
#pragma unroll
  for (int k = 0; k < NPOP; k++) {
    f[k].x = fa[k], g[k].x = ga[k];
    fa[k] = f[k].y, ga[k] = g[k].y;
  }
  node_ref<false>(V, 0, fa, ga, F.y, r.y, u.y, v.y, t.y, none, none);
#pragma unroll
  for (int k = 0; k < NPOP; k++) f[k].y = fa[k], g[k].y = ga[k];
}

template <typename P>
__device__ __forceinline__ void stcs2(char* p, unsigned o, P a) { __stcs(reinterpret_cast<P*>(p + o), a); }
__device__ __forceinline__ void cp16(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// a level's moments at its strip's aligned pairs (ODD: the lane's second
// column with its right neighbour's first)
template <bool ODD, typename Real>
__device__ __forceinline__ void wave_put(Real* p, Pair<Real> a, bool ok) {
  const Pair<Real> b = ODD ? pair_of(a.y, __shfl_down_sync(0xffffffffu, a.x, 1)) : a;
  if (ok) *reinterpret_cast<Pair<Real>*>(p) = b;
}

template <typename Real, int S, int D, bool NUD, typename GetV>
__device__ __forceinline__ void wave_march(GetV&& view, int x0, int ncols, int ya, int Hc, Real* sm) {
  using P2 = Pair<Real>;
  constexpr bool F32 = std::is_same<Real, float>::value;
  constexpr int ES = sizeof(Real), ROW = 64 * ES;  // bytes of a value, of a staged row
  static_assert(S == 2 || S == 4, "x0 - S a multiple of 4 and aligned pairs");
  const LBView<Real>& V1 = view(std::integral_constant<int, 0>{});
  const int nx = V1.nx, ny = V1.ny;
  const unsigned pitch = (unsigned)V1.pitch;
  const size_t plane = V1.plane;
  const bool glo = S == 2 && V1.gh2_lo != nullptr, ghi = S == 2 && V1.gh2_hi != nullptr;
  const int ylo = glo ? -1 : 0, yhi = ghi ? ny : ny - 1;
  const int lane = threadIdx.x & 31;
  const int l1 = min(lane + 1, 31);
  Real* const lag = sm + D * WAVE_STAGE * 64;
  const unsigned sm_addr = (unsigned)__cvta_generic_to_shared(sm);

  // this lane's 16 bytes of a staged row: of f or g by half-warp in FP32, of
  // one plane per instruction in FP64
  constexpr int VEC = 16 / ES;
  const int cq = VEC * (F32 ? (lane & 15) : lane);
  const bool cp_ok = cq < ncols + 2 * S;
  const unsigned cp_col = (unsigned)((x0 - S + cq + nx) % nx);  // (x0 - S >= -4 >= -nx)
  const Real* const cp_base = (!F32 || lane < 16 ? V1.fsrc : V1.gsrc) + cp_col;
  const unsigned cp_dst = sm_addr + (!F32 || lane < 16 ? 0 : NPOP * ROW) + cq * ES;
  const ptrdiff_t g_off = F32 ? 0 : V1.gsrc - V1.fsrc;
  auto issue = [&](int y, int stage) {
    if (y > 0 && y < ny - 1 && cp_ok) {
      const Real* p = cp_base + (size_t)((unsigned)y * pitch);
      const unsigned d = cp_dst + stage * (WAVE_STAGE * ROW);
      static_for<NPOP>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        const Real* q = p + ((ptrdiff_t)(k * plane) - (ptrdiff_t)icy(k) * (ptrdiff_t)pitch);
        cp16(d + k * ROW, q);
        if constexpr (!F32) cp16(d + (NPOP + k) * ROW, q + g_off);
      });
      if (!F32 || lane < 16) cp16(d + 2 * NPOP * ROW, V1.Fin + ((unsigned)y * pitch + cp_col));
    }
    cp_commit();
  };

  const int nit = Hc + 2 * (S - 1);
  int y = ya - (S - 1);
  // A nudged run's increments of g at the lane's level-1 pair (w_k times the
  // node's sum of step n, as the apply pass forms them; none where the sum is
  // 0): a row's mask words are loaded three iterations ahead, its sums (where
  // a bit is set) two, and converted one ahead, both nodes together.  The
  // loads are straight-line code (rows clamped to the domain, as rows outside
  // it do not count; predicated loads of the sums): guarded by branches they
  // cost 15 us of an 88 us launch at 2048x1024, with one observation.
  const bool nudged = NUD && V1.nmask != nullptr;  // (an ensemble's members may have none)
  const int nxa = (x0 - (S - 1) + 2 * lane + nx) % nx, nxb = nxa + 1 == nx ? 0 : nxa + 1;
  const unsigned* const mw_a = V1.nmask + (nxa >> 5);
  const unsigned* const mw_b = V1.nmask + (nxb >> 5);
  unsigned ma = 0, mb = 0;
  long long na = 0, nb = 0;
  auto load_mask = [&](int yy) {
    const size_t o = (size_t)min(max(yy, 0), ny - 1) * (pitch >> 5);
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(ma) : "l"(mw_a + o));
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(mb) : "l"(mw_b + o));
  };
  auto load_sums = [&](int yy) {
    const unsigned long long* row = V1.nacc + (size_t)min(max(yy, 0), ny - 1) * pitch;
    auto one = [](const unsigned long long* p, unsigned bit) -> long long {
      long long v;
      asm volatile(
          "{.reg .pred p; setp.ne.u32 p, %2, 0; mov.s64 %0, 0; @p ld.global.s64 %0, [%1];}"
          : "=l"(v) : "l"(p), "r"(bit));
      return v;
    };
    na = one(row + nxa, (ma >> (nxa & 31)) & 1u);
    nb = one(row + nxb, (mb >> (nxb & 31)) & 1u);
  };
  bool inc_a = false, inc_b = false;
  Real ia[3] = {}, ib[3] = {};  // increments of the weights' three classes
  auto convert = [&]() {
    inc_a = na != 0, inc_b = nb != 0;
    if (__any_sync(0xffffffffu, inc_a || inc_b)) {
      const double sa = (double)na * (1.0 / FIX_SCALE), sb = (double)nb * (1.0 / FIX_SCALE);
      ia[0] = nudge_increment<Real>(0, sa), ib[0] = nudge_increment<Real>(0, sb);
      ia[1] = nudge_increment<Real>(1, sa), ib[1] = nudge_increment<Real>(1, sb);
      ia[2] = nudge_increment<Real>(5, sa), ib[2] = nudge_increment<Real>(5, sb);
    }
  };
  if (nudged) {
    load_mask(y);
    load_sums(y);
    convert();
    load_mask(y + 1);
    load_sums(y + 1);
    load_mask(y + 2);
  }
#pragma unroll
  for (int d = 0; d < D; d++) issue(d < nit ? y + d : -1, d);
  int stage = 0;
  int p0 = 0, p1 = 6;  // c_y = +1 slots of this iteration's row (and of the row two before it), and of the row before
  for (int it = 0; it < nit; it++, y++) {
    P2 f[NPOP], g[NPOP], F, r, u, v, t;
    cp_wait<D - 1>();
    __syncwarp();
    const Real* st = sm + stage * WAVE_STAGE * 64;
    // a staged plane at the lane's pair, its right neighbour's, and one column right of its own
    auto sown = [&](int i) { return reinterpret_cast<const P2*>(st + i * 64)[lane]; };
    auto snxt = [&](int i) { return reinterpret_cast<const P2*>(st + i * 64)[l1]; };
    auto smid = [&](int i) { return pair_of(st[i * 64 + 2 * lane + 1], st[i * 64 + 2 * l1]); };
    if (y > 0 && y < ny - 1) {
      static_for<NPOP>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        f[k] = icx(k) == 1 ? sown(k) : (icx(k) == -1 ? snxt(k) : smid(k));
        g[k] = icx(k) == 1 ? sown(NPOP + k) : (icx(k) == -1 ? snxt(NPOP + k) : smid(NPOP + k));
      });
      F = smid(2 * NPOP);
    } else if (y >= ylo && y <= yhi) {
      Real a[2 * NPOP], b[2 * NPOP];
      auto one = [&](int x, Real* p, Real& Fx) {
        x = (x + nx) % nx;
        if (S == 2 && (y < 0 || y >= ny)) {
          pull_ghost_row<Real, size_t>(V1, y < 0, x, p, p + NPOP, Fx);
        } else {
          pull_node<Real, LBRB_TWALL_DIRICHLET, size_t, false>(V1, y, x, p, p + NPOP);
          dirichlet_walls(V1, y, p + NPOP);
          Fx = V1.Fin[(unsigned)y * pitch + x];
        }
      };
      one(x0 - (S - 1) + 2 * lane, a, F.x);
      one(x0 - (S - 1) + 2 * lane + 1, b, F.y);
#pragma unroll
      for (int k = 0; k < NPOP; k++) {
        f[k] = pair_of(a[k], b[k]);
        g[k] = pair_of(a[NPOP + k], b[NPOP + k]);
      }
    }
    __syncwarp();
    issue(it + D < nit ? y + D : -1, stage);
    stage = stage + 1 == D ? 0 : stage + 1;
    collide_pair(V1, f, g, F, r, u, v, t);
    if (nudged) {
      if (__any_sync(0xffffffffu, inc_a || inc_b)) {
#pragma unroll
        for (int k = 0; k < NPOP; k++) {
          constexpr int cls[NPOP] = {0, 1, 1, 1, 1, 2, 2, 2, 2};
          const Real ga = g[k].x + ia[cls[k]], gb = g[k].y + ib[cls[k]];
          g[k] = pair_of(inc_a ? ga : g[k].x, inc_b ? gb : g[k].y);
        }
      }
      convert();
      load_sums(y + 2);
      load_mask(y + 3);
    }
    static_for<S>([&](auto sc) {
      constexpr int s = decltype(sc)::value + 1;  // level, whose row yr is now in f, g, F and r, u, v, t
      constexpr int off = S - s;
      const LBView<Real>& V = view(std::integral_constant<int, s - 1>{});
      const int yr = y - (s - 1);
      // the level's moments (and the last level's state) in its strip and chunk
      if ((unsigned)(yr - ya) < (unsigned)Hc) {
        const int c = 2 * lane - off + (off & 1);  // column in the strip of the aligned pair
        const bool ok = c >= 0 && c < ncols;
        const int xc = x0 + c;
        const unsigned o = (unsigned)yr * pitch + (unsigned)(xc >= nx ? xc - nx : xc);
        const unsigned ob = o * (unsigned)ES;  // (bytes within a plane: 2^32 of them would be a run of 200 GB)
        constexpr bool ODD = (off & 1) != 0;
        if constexpr (s == S) {
          if (ok) {
#pragma unroll
            for (int k = 0; k < NPOP; k++) {
              stcs2(reinterpret_cast<char*>(V.fdst) + k * plane * ES, ob, f[k]);
              stcs2(reinterpret_cast<char*>(V.gdst) + k * plane * ES, ob, g[k]);
            }
          }
        }
        if (s == S || V.write_F) wave_put<ODD, Real>(V.Fout + o, F, ok);
        if (V.write_uv) {
          wave_put<ODD, Real>(V.u + o, u, ok);
          wave_put<ODD, Real>(V.v + o, v, ok);
        }
        if (V.write_rt & 1) wave_put<ODD, Real>(V.T + o, t, ok);
        if (V.write_rt & 2) wave_put<ODD, Real>(V.rho + o, r, ok);
      }
      if constexpr (s < S) {
        // the next level's inputs at row yn; this level's row takes their place
        const int yn = yr - 1;
        const bool lo = yn == 0 && !glo, hi = yn == ny - 1 && !ghi;
        constexpr int CW = wave_cols(s);
        Real* w0 = lag + wave_lag(s - 1);
        Real* w1 = w0 + (7 + p0) * CW;
        Real* wp = w0 + (7 + p1) * CW;
        auto own = [&](const Real* q, int i) { return reinterpret_cast<const P2*>(q + i * CW)[lane]; };
        auto nxt = [&](const Real* q, int i) { return reinterpret_cast<const P2*>(q + i * CW)[l1]; };
        auto mid = [&](const Real* q, int i) { return pair_of(q[i * CW + 2 * lane + 1], q[i * CW + 2 * l1]); };
        const P2 a0 = mid(w0, 0), a1 = own(w0, 1), a3 = nxt(w0, 2);
        const P2 b0 = mid(w0, 3), b1 = own(w0, 4), b3 = nxt(w0, 5);
        const P2 Fn = mid(w0, 6);
        P2 a2 = mid(w1, 0), a5 = own(w1, 1), a6 = nxt(w1, 2);
        if (lo) a5 = mid(w1, 1), a6 = mid(w1, 2);
        P2 b2 = mid(w1, 3), b5 = own(w1, 4), b6 = nxt(w1, 5);
        __syncwarp();
        if (2 * lane < CW) {
          auto put = [&](Real* q, int i, P2 a) { reinterpret_cast<P2*>(q + i * CW)[lane] = a; };
          put(w0, 0, f[0]), put(w0, 1, f[1]), put(w0, 2, f[3]);
          put(w0, 3, g[0]), put(w0, 4, g[1]), put(w0, 5, g[3]);
          put(w0, 6, F);
          put(w1, 0, f[2]), put(w1, 1, f[5]), put(w1, 2, f[6]);
          put(w1, 3, g[2]), put(w1, 4, g[5]), put(w1, 5, g[6]);
          if (yr == 0 && !glo) put(wp, 0, f[4]), put(wp, 1, f[7]), put(wp, 2, f[8]);
        }
        auto shm = [&](P2 a) { return pair_of(a.y, __shfl_down_sync(0xffffffffu, a.x, 1)); };
        auto shn = [&](P2 a) {
          return pair_of(__shfl_down_sync(0xffffffffu, a.x, 1), __shfl_down_sync(0xffffffffu, a.y, 1));
        };
        f[4] = shm(f[4]), f[7] = shn(f[7]);  // (f[8]: the lane's own)
        g[4] = shm(g[4]), g[7] = shn(g[7]);
        f[0] = a0, f[1] = a1, f[3] = a3, f[2] = a2, f[5] = a5, f[6] = a6;
        g[0] = b0, g[1] = b1, g[3] = b3, g[2] = b2, g[5] = b5, g[6] = b6;
        F = Fn;
        const LBView<Real>& VN = view(std::integral_constant<int, s>{});
        if (lo || hi) {
          if (lo) {
            g[2] = g[5] = g[6] = pair_of(Real(0), Real(0));
          } else {
            f[4] = mid(wp, 0), f[7] = mid(wp, 1), f[8] = mid(wp, 2);
            g[4] = g[7] = g[8] = pair_of(Real(0), Real(0));
          }
          Real ga[NPOP], gb[NPOP];
#pragma unroll
          for (int k = 0; k < NPOP; k++) ga[k] = g[k].x, gb[k] = g[k].y;
          dirichlet_walls(VN, yn, ga);
          dirichlet_walls(VN, yn, gb);
#pragma unroll
          for (int k = 0; k < NPOP; k++) g[k] = pair_of(ga[k], gb[k]);
        }
        __syncwarp();
        if (it >= 2 * s) collide_pair(VN, f, g, F, r, u, v, t);  // (before that its inputs are not there yet)
      }
    });
    const int pt = p0;
    p0 = p1;
    p1 = pt;
  }
  cp_wait<0>();
}

}  // namespace lbrb
