// lb_kernels.cu -- the fused pull stream + walls + buoyancy + moments +
// collision kernel: one launch per time step, both populations f and g.
//
// Reference semantics (temppart_dump.c, Trajectories):
//   stream          :781-854   f_k(x) <- f_k(x - c_k) for k = 1..8, same for g
//   force           :744-755   F_y = -gravity * rho^{n-1} * T^{n-1}, F_x = 0
//   f walls         :763-777, 859-894   half-way bounce-back from the
//                              pre-stream wall row: f2,f5,f6(1) <- f4,f7,f8(1);
//                              f4,f7,f8(NY) <- f2,f5,f6(NY)
//   g walls (T)     :896-921   g_in = -g_opp(post-stream) + 2 w T_wall
//   g walls (N)     tempvel_nudge.c:684-702, 783-962: rows 1 and NY hold
//                              pre-stream copies of rows 2 and NY-1 and are
//                              not streamed into
//   moments         :957-987 (tempvel_nudge.c:1069-1102 adds 1/2 nud_term)
//   collision       :1097-1180, 1314-1341 (tempvel_nudge.c:1917-1945 nudged g)
//
// Two arithmetic forms:
//   Real = double: the reference's operation order exactly (built with
//     --fmad=false), bit-identical to the reference on x86-64.
//   Real = float: populations stored as deviations from their weights
//     (f_k - w_k rho0, g_k - w_k T0), collision in FP32.
//
// Mapping: one node per thread, a block covers BS consecutive nodes of one
// row (wall handling is block-uniform).  Every population is one plain
// coalesced load at its pull address: x-1 and x+1 fall in the same 128-byte
// lines as the neighbouring threads' loads, so L1/L2 absorb the shift and
// DRAM reads each value once.  All 18 loads are independent and issue back to
// back; the small register budget keeps many warps per SM and enough bytes in
// flight for HBM3e.  The buoyancy F of the next step is written to the other
// of two buffers, so a launch is a pure function of its sources: the launch
// shape (block size, blocks per SM) is picked by timing the candidates on the
// run's own grid (tune_lb).
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <type_traits>

#include "lb_pair.cuh"
#include "particle_dev.cuh"

namespace lbrb {

// post-stream populations only (walls applied): dumpfpre/dumpgpre
template <typename Real, int TWALL>
__global__ void __launch_bounds__(128) lb_pull_kernel(const LBView<Real> V, Real* __restrict__ outf,
                                                      Real* __restrict__ outg) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (x >= V.nx) return;
  Real fs[NPOP], gs[NPOP];
  pull_node<Real, TWALL, size_t>(V, j, x, fs, gs);
  if (TWALL == LBRB_TWALL_DIRICHLET) dirichlet_walls(V, j, gs);
  const size_t o = (size_t)j * V.pitch + x;
#pragma unroll
  for (int k = 0; k < NPOP; k++) {
    outf[(size_t)k * V.plane + o] = fs[k];
    outg[(size_t)k * V.plane + o] = gs[k];
  }
}

template <typename Real, int TWALL, bool REFNUDGE, int BS, int MINB, typename Off, bool FAST>
__global__ void __launch_bounds__(BS, MINB) lb_node_kernel(const LBView<Real> V) {
  pdl_wait();
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (x >= V.nx) return;
  lb_update_node<Real, TWALL, REFNUDGE, Off, FAST>(V, j, x);
}

// ------------------------------------------------------- two steps per launch
// Temporal blocking of two steps n, n+1 in TX x TY tiles, one per block
// (lb_pair.cuh: tile_block, the per-block work).
template <typename Real, int TX, int TY, int NT, int MINB, typename Off>
__global__ void __launch_bounds__(NT, MINB) lb_pair_kernel(const LBView<Real> V1, const LBView<Real> V2) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char pair_smem[];
  tile_block<Real, TX, TY, NT, Off>(V1, V2, blockIdx.x * TX, blockIdx.y * TY, pair_smem);
}
// the same tiles after blocks that advance particles (PJob: the first
// J.nblocks; FP32 at 512x256 with 4096 tracers 3.9 us per step, 5.4 with
// particle launches of their own).  A kernel of its own: launches without
// particles keep the smaller parameter block and the plain grid.
template <typename Real, int TX, int TY, int NT, int MINB, typename Off>
__global__ void __launch_bounds__(NT, MINB)
    lb_pair_job_kernel(const LBView<Real> V1, const LBView<Real> V2, const __grid_constant__ PJob<Real> J,
                       int tiles_x) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char pair_smem[];
  const int b = blockIdx.x - J.nblocks;
  if (b < 0) {
    particle_job(J, blockIdx.x);
    return;
  }
  tile_block<Real, TX, TY, NT, Off>(V1, V2, b % tiles_x * TX, b / tiles_x * TY, pair_smem);
}

// marching (lb_pair.cuh: wave_march): item = strip + chunk * nstrips, one per warp
template <typename Real, int NW, int MINB, int D, bool NUD>
__global__ void __launch_bounds__(32 * NW, MINB)
    lb_wave2_kernel(const LBView<Real> V1, const LBView<Real> V2, int H, int nitems) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char wave_smem[];
  const int w = threadIdx.x >> 5, item = blockIdx.x * NW + w;
  if (item >= nitems) return;
  const int nstrips = (V1.nx + WAVE_COLS<2> - 1) / WAVE_COLS<2>;
  const int strip = item % nstrips, ya = item / nstrips * H;
  wave_march<Real, 2, D, NUD>([&](auto s) -> const LBView<Real>& { return decltype(s)::value == 0 ? V1 : V2; },
                              strip * WAVE_COLS<2> + WAVE_X0<2>, min(WAVE_COLS<2>, V1.nx - strip * WAVE_COLS<2>), ya,
                              min(H, V1.ny - ya),
                              reinterpret_cast<Real*>(wave_smem + w * wave_smem_bytes<Real, 2, D>()));
}

// four steps per launch: the populations and F cross HBM once per four steps
template <typename Real, int NW, int MINB, int D>
__global__ void __launch_bounds__(32 * NW, MINB)
    lb_wave4_kernel(const LBView<Real> V1, const LBView<Real> V2, const LBView<Real> V3, const LBView<Real> V4,
                    int H, int nitems) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char wave_smem[];
  const int w = threadIdx.x >> 5, item = blockIdx.x * NW + w;
  if (item >= nitems) return;
  const int nstrips = (V1.nx + WAVE_COLS<4> - 1) / WAVE_COLS<4>;
  const int strip = item % nstrips, ya = item / nstrips * H;
  wave_march<Real, 4, D, false>(
      [&](auto s) -> const LBView<Real>& {
        if constexpr (decltype(s)::value == 0) return V1;
        else if constexpr (decltype(s)::value == 1) return V2;
        else if constexpr (decltype(s)::value == 2) return V3;
        else return V4;
      },
      strip * WAVE_COLS<4> + WAVE_X0<4>, min(WAVE_COLS<4>, V1.nx - strip * WAVE_COLS<4>), ya, min(H, V1.ny - ya),
      reinterpret_cast<Real*>(wave_smem + w * wave_smem_bytes<Real, 4, D>()));
}

// pair launch shapes: (tile columns, tile rows, threads, min blocks per SM)
struct PairShape { int tx, ty, nt, minb; };
constexpr PairShape PAIR_SHAPES[] = {{32, 8, 256, 4}, {32, 4, 128, 6}, {32, 16, 512, 2}, {64, 4, 256, 3},
                                     {32, 8, 352, 2}, {30, 8, 320, 3}, {32, 8, 256, 5}, {32, 6, 192, 5},
                                     {64, 8, 512, 2}};
constexpr int NPAIR = sizeof(PAIR_SHAPES) / sizeof(PAIR_SHAPES[0]);
static_assert(NPAIR <= NUM_PAIR_SHAPES, "pair shape table");

template <auto kernel, size_t smem>
static cudaError_t tile_limit() {
  // the shared-memory limit is a per-device attribute of the kernel: set
  // once per device (one bit per device ordinal, per kernel)
  static std::atomic<unsigned long long> attr_set{0};
  return smem_limit_once((const void*)kernel, smem, attr_set);
}
template <typename Real, int TX, int TY, int NT, int MINB, typename Off>
static cudaError_t launch_tile(const LBView<Real>& V1, const LBView<Real>& V2, cudaStream_t s, bool pdl,
                               const PJob<Real>* job) {
  constexpr size_t smem = tile_smem_bytes<Real, TX, TY>();
  const int tiles_x = (V1.nx + TX - 1) / TX, tiles_y = (V1.ny + TY - 1) / TY;
  if (job && job->nsteps > 0) {
    constexpr auto kernel = lb_pair_job_kernel<Real, TX, TY, NT, MINB, Off>;
    const cudaError_t e = tile_limit<kernel, smem>();
    if (e != cudaSuccess) return e;
    PJob<Real> J = *job;
    J.nblocks = (J.np + NT - 1) / NT;
    return launch_k(kernel, dim3((unsigned)(J.nblocks + (long)tiles_x * tiles_y)), NT, smem, s, pdl, V1, V2, J, tiles_x);
  }
  constexpr auto kernel = lb_pair_kernel<Real, TX, TY, NT, MINB, Off>;
  const cudaError_t e = tile_limit<kernel, smem>();
  if (e != cudaSuccess) return e;
  return launch_k(kernel, dim3(tiles_x, tiles_y), NT, smem, s, pdl, V1, V2);
}
template <typename Real, int TX, int TY, int NT, int MINB>
static cudaError_t launch_pair_t(const LBView<Real>& V1, const LBView<Real>& V2, cudaStream_t s, bool pdl,
                                 const PJob<Real>* job) {
  // (FP64 holds twice the registers per value: half the blocks per SM)
  constexpr int MB = std::is_same<Real, double>::value ? (MINB + 1) / 2 : MINB;
  if (off32_ok(V1.plane)) return launch_tile<Real, TX, TY, NT, MB, uint32_t>(V1, V2, s, pdl, job);
  return launch_tile<Real, TX, TY, NT, MB, size_t>(V1, V2, s, pdl, job);
}

// The marching shapes: wave_march, one warp per strip and chunk, (warps per
// block, min blocks per SM, waves) in FP32; in FP64 8 warps per SM and the
// waves.  The chunk height is chosen so that the items (strips x chunks) fill
// at most `waves` waves of resident warps: few waves recompute fewer rows
// (two per chunk), many keep the warps of a row band together, which the DRAM
// pages reward.  FP32, 4096x2048: 118 us per step with 8 warps per SM (6
// waves) and with 12 (9 waves); with 15 (128 registers) 128 us, their copies
// queueing behind one another.  FP64 (about 240 registers): 231 us with 8
// warps, 345 with 11 (168 registers, spilling); the 32x6 tile takes 282.
struct WaveShape { int nw, minb, waves; };
constexpr int NMARCH = NUM_PAIR_SHAPES - NPAIR;
constexpr WaveShape WAVE_SHAPES[NMARCH] = {{8, 1, 1}, {8, 1, 2}, {8, 1, 3}, {8, 1, 6}, {4, 3, 4}, {4, 3, 9}};
constexpr int WAVE_SHAPES_FP64[NMARCH] = {1, 2, 3, 4, 6, 9};
// rows of inputs in flight per warp
constexpr int WAVE2_STAGES = 2, WAVE2_STAGES_FP64 = 1;

// the chunk height for `waves` waves of resident warps, and the items
template <typename Kernel>
static cudaError_t wave_grid(Kernel kernel, int nw, size_t smem, std::atomic<int>* occ_cache, int waves, int cols,
                             int nx, int ny, int* H, long* nitems) {
  int occ = 0, dev = 0, nsm = 0;
  cudaError_t e = occupancy_once((const void*)kernel, 32 * nw, smem, occ_cache, &occ);
  if (e == cudaSuccess) e = current_device(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const long nstrips = (nx + cols - 1) / cols;
  const long chunks = std::min((long)ny, std::max(1L, (long)waves * occ * nsm * nw / nstrips));
  *H = (int)((ny + chunks - 1) / chunks);
  *nitems = nstrips * ((ny + *H - 1) / *H);
  return cudaSuccess;
}

template <typename Real, int NW, int MINB, int D, bool NUD>
static cudaError_t launch_wave2_t(const LBView<Real>& V1, const LBView<Real>& V2, int waves, cudaStream_t s,
                                  bool pdl) {
  constexpr auto kernel = lb_wave2_kernel<Real, NW, MINB, D, NUD>;
  constexpr size_t smem = NW * wave_smem_bytes<Real, 2, D>();
  static std::atomic<unsigned long long> attr_set{0};
  static std::atomic<int> occ_cache[MAX_DEVICES] = {};
  cudaError_t e = smem_limit_once((const void*)kernel, smem, attr_set);
  int H = 0;
  long nitems = 0;
  if (e == cudaSuccess) e = wave_grid(kernel, NW, smem, occ_cache, waves, WAVE_COLS<2>, V1.nx, V1.ny, &H, &nitems);
  if (e != cudaSuccess) return e;
  return launch_k(kernel, dim3((unsigned)((nitems + NW - 1) / NW)), 32 * NW, smem, s, pdl, V1, V2, H, (int)nitems);
}
static cudaError_t launch_march(const LBView<float>& V1, const LBView<float>& V2, int m, cudaStream_t s, bool pdl) {
  const WaveShape w = WAVE_SHAPES[m];
  if (w.nw == 8)
    return V1.nmask ? launch_wave2_t<float, 8, 1, WAVE2_STAGES, true>(V1, V2, w.waves, s, pdl)
                    : launch_wave2_t<float, 8, 1, WAVE2_STAGES, false>(V1, V2, w.waves, s, pdl);
  return V1.nmask ? launch_wave2_t<float, 4, 3, WAVE2_STAGES, true>(V1, V2, w.waves, s, pdl)
                  : launch_wave2_t<float, 4, 3, WAVE2_STAGES, false>(V1, V2, w.waves, s, pdl);
}
static cudaError_t launch_march(const LBView<double>& V1, const LBView<double>& V2, int m, cudaStream_t s, bool pdl) {
  return V1.nmask ? launch_wave2_t<double, 8, 1, WAVE2_STAGES_FP64, true>(V1, V2, WAVE_SHAPES_FP64[m], s, pdl)
                  : launch_wave2_t<double, 8, 1, WAVE2_STAGES_FP64, false>(V1, V2, WAVE_SHAPES_FP64[m], s, pdl);
}

// four-step launch shapes: waves of resident warps the chunk height aims at
constexpr int QUAD_WAVES[NUM_QUAD_SHAPES] = {1, 2, 4};
template <typename Real>
static cudaError_t launch_quad(const LBView<Real> (&V)[4], int shape, cudaStream_t s, bool pdl) {
  // 12 warps per SM in FP32, 6 in FP64 (shared memory)
  constexpr bool F32 = std::is_same<Real, float>::value;
  constexpr int NW = F32 ? 4 : 6, MINB = F32 ? 3 : 1, D = 1;
  constexpr auto kernel = lb_wave4_kernel<Real, NW, MINB, D>;
  constexpr size_t smem = NW * wave_smem_bytes<Real, 4, D>();
  static std::atomic<unsigned long long> attr_set{0};
  static std::atomic<int> occ_cache[MAX_DEVICES] = {};
  cudaError_t e = smem_limit_once((const void*)kernel, smem, attr_set);
  int H = 0;
  long nitems = 0;
  if (e == cudaSuccess)
    e = wave_grid(kernel, NW, smem, occ_cache, QUAD_WAVES[shape], WAVE_COLS<4>, V[0].nx, V[0].ny, &H, &nitems);
  if (e != cudaSuccess) return e;
  return launch_k(kernel, dim3((unsigned)((nitems + NW - 1) / NW)), 32 * NW, smem, s, pdl, V[0], V[1], V[2], V[3], H,
                  (int)nitems);
}
cudaError_t launch_quad_fp32(const LBView<float> (&V)[4], int shape, cudaStream_t s, bool pdl) {
  return launch_quad<float>(V, shape, s, pdl);
}
cudaError_t launch_quad_fp64(const LBView<double> (&V)[4], int shape, cudaStream_t s, bool pdl) {
  return launch_quad<double>(V, shape, s, pdl);
}

template <typename Real>
static cudaError_t launch_pair(const LBView<Real>& V1, const LBView<Real>& V2, int shape, cudaStream_t s, bool pdl,
                               const PJob<Real>* job = nullptr) {
  // (no particles in the strips' launches: a strip's warps run for the whole
  // launch, and particle blocks in their places cost more than they hide --
  // 1500x701 with 20,000 inertial particles 12.7 against 11.9 ms per 301 steps)
  if (shape >= NPAIR) return launch_march(V1, V2, shape - NPAIR, s, pdl);
  switch (shape) {
    case 1: return launch_pair_t<Real, 32, 4, 128, 6>(V1, V2, s, pdl, job);
    case 2: return launch_pair_t<Real, 32, 16, 512, 2>(V1, V2, s, pdl, job);
    case 3: return launch_pair_t<Real, 64, 4, 256, 3>(V1, V2, s, pdl, job);
    case 4: return launch_pair_t<Real, 32, 8, 352, 2>(V1, V2, s, pdl, job);
    case 5: return launch_pair_t<Real, 30, 8, 320, 3>(V1, V2, s, pdl, job);
    case 6: return launch_pair_t<Real, 32, 8, 256, 5>(V1, V2, s, pdl, job);
    case 7: return launch_pair_t<Real, 32, 6, 192, 5>(V1, V2, s, pdl, job);
    case 8: return launch_pair_t<Real, 64, 8, 512, 2>(V1, V2, s, pdl, job);
    default: return launch_pair_t<Real, 32, 8, 256, 4>(V1, V2, s, pdl, job);
  }
}

// --------------------------------------------------------------- launch
// launch shapes tried by tune_lb: (threads per block, min blocks per SM,
// pull form: 1 = interior rows without wall logic and 32-bit offsets where
// they fit, 0 = the general pull with 64-bit offsets on every row)
struct Shape { int bs, minb, fast; };
constexpr Shape SHAPES[] = {{256, 1, 1}, {256, 2, 1}, {256, 3, 1}, {128, 4, 1}, {128, 6, 1},
                            {512, 1, 1}, {512, 2, 1}, {256, 3, 0}, {128, 4, 0}, {128, 6, 0}};
constexpr int NSHAPES = sizeof(SHAPES) / sizeof(SHAPES[0]);

template <typename Real, int TWALL, bool REFNUDGE, int BS, int MINB, bool FAST>
static cudaError_t launch_shape(const LBView<Real>& V, cudaStream_t s, bool pdl) {
  dim3 grid((V.nx + BS - 1) / BS, V.ny);
  if (FAST && off32_ok(V.plane))
    return launch_k(lb_node_kernel<Real, TWALL, REFNUDGE, BS, MINB, uint32_t, true>, grid, BS, 0, s, pdl, V);
  return launch_k(lb_node_kernel<Real, TWALL, REFNUDGE, BS, MINB, size_t, FAST>, grid, BS, 0, s, pdl, V);
}

template <typename Real, int TWALL, bool REFNUDGE>
static cudaError_t launch_lb(const LBView<Real>& V, int shape, cudaStream_t s, bool pdl) {
  switch (shape) {
    case 1: return launch_shape<Real, TWALL, REFNUDGE, 256, 2, true>(V, s, pdl);
    case 2: return launch_shape<Real, TWALL, REFNUDGE, 256, 3, true>(V, s, pdl);
    case 3: return launch_shape<Real, TWALL, REFNUDGE, 128, 4, true>(V, s, pdl);
    case 4: return launch_shape<Real, TWALL, REFNUDGE, 128, 6, true>(V, s, pdl);
    case 5: return launch_shape<Real, TWALL, REFNUDGE, 512, 1, true>(V, s, pdl);
    case 6: return launch_shape<Real, TWALL, REFNUDGE, 512, 2, true>(V, s, pdl);
    case 7: return launch_shape<Real, TWALL, REFNUDGE, 256, 3, false>(V, s, pdl);
    case 8: return launch_shape<Real, TWALL, REFNUDGE, 128, 4, false>(V, s, pdl);
    case 9: return launch_shape<Real, TWALL, REFNUDGE, 128, 6, false>(V, s, pdl);
    default: return launch_shape<Real, TWALL, REFNUDGE, 256, 1, true>(V, s, pdl);
  }
}

cudaError_t launch_lb_fp64(const LBView<double>& V, int twall, bool refnudge, int shape,
                           cudaStream_t s, bool pdl) {
  if (twall == LBRB_TWALL_DIRICHLET)
    return refnudge ? launch_lb<double, LBRB_TWALL_DIRICHLET, true>(V, shape, s, pdl)
                    : launch_lb<double, LBRB_TWALL_DIRICHLET, false>(V, shape, s, pdl);
  return refnudge ? launch_lb<double, LBRB_TWALL_ADIABATIC, true>(V, shape, s, pdl)
                  : launch_lb<double, LBRB_TWALL_ADIABATIC, false>(V, shape, s, pdl);
}

cudaError_t launch_lb_fp32(const LBView<float>& V, int twall, int shape, cudaStream_t s, bool pdl) {
  if (twall == LBRB_TWALL_DIRICHLET) return launch_lb<float, LBRB_TWALL_DIRICHLET, false>(V, shape, s, pdl);
  return launch_lb<float, LBRB_TWALL_ADIABATIC, false>(V, shape, s, pdl);
}

// Autotuner: time every launch shape on this run's grid (CUDA events, `reps`
// launches after one warm-up launch each, with programmatic dependent launch
// as the steps use) and return the fastest.  A trial
// launch reads the current state and writes only buffers the real step
// overwrites: the other population buffer, the other F buffer and, when the
// caller's view stores u, v (runs with particles), the u, v slot of the next
// step; rho and T are not written.  Box-nudged FP64 steps update nud_term in
// place and are not tuned (lbrb_step gives them a shape).
template <typename Real>
static int tune(const LBView<Real>& Vin, int twall, bool refnudge, cudaStream_t s, int reps,
                float* best_ms) {
  LBView<Real> V = Vin;  // u, v stores as the caller's view has them
  V.write_rt = 0;
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  // two rounds over all shapes, each shape's faster round counts: a shape
  // timed while the clocks settle or beside a transient gets a second look
  float shape_ms[NSHAPES];
  for (float& m : shape_ms) m = 1e30f;
  for (int round = 0; round < 2; round++) {
    for (int sh = 0; sh < NSHAPES; sh++) {
      auto go = [&]() {
        if constexpr (std::is_same<Real, double>::value) return launch_lb_fp64(V, twall, refnudge, sh, s, true);
        else return launch_lb_fp32(V, twall, sh, s, true);
      };
      if (go() != cudaSuccess) { cudaGetLastError(); continue; }
      cudaEventRecord(a, s);
      for (int r = 0; r < reps; r++) go();
      cudaEventRecord(b, s);
      cudaEventSynchronize(b);
      float ms = 0.f;
      cudaEventElapsedTime(&ms, a, b);
      shape_ms[sh] = std::min(shape_ms[sh], ms);
    }
  }
  int best = 0;
  float bt = 1e30f;
  for (int sh = 0; sh < NSHAPES; sh++)
    if (shape_ms[sh] < bt) { bt = shape_ms[sh]; best = sh; }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (best_ms) *best_ms = bt / reps;
  return best;
}

template <typename Real>
static cudaError_t launch_pull_t(const LBView<Real>& V, int twall, void* outf, void* outg,
                                 cudaStream_t s) {
  dim3 grid((V.nx + 127) / 128, V.ny);
  if (twall == LBRB_TWALL_DIRICHLET)
    lb_pull_kernel<Real, LBRB_TWALL_DIRICHLET><<<grid, 128, 0, s>>>(V, (Real*)outf, (Real*)outg);
  else
    lb_pull_kernel<Real, LBRB_TWALL_ADIABATIC><<<grid, 128, 0, s>>>(V, (Real*)outf, (Real*)outg);
  return cudaGetLastError();
}
cudaError_t launch_pull_fp64(const LBView<double>& V, int twall, void* outf, void* outg, cudaStream_t s) {
  return launch_pull_t<double>(V, twall, outf, outg, s);
}
cudaError_t launch_pull_fp32(const LBView<float>& V, int twall, void* outf, void* outg, cudaStream_t s) {
  return launch_pull_t<float>(V, twall, outf, outg, s);
}

// launches timed per shape: enough that each shape's timed span is well above
// the event resolution and launch jitter on small grids
static int tune_reps(const LBView<float>& V) { return (long)V.nx * V.ny >= (1L << 21) ? 6 : 30; }
static int tune_reps(const LBView<double>& V) { return (long)V.nx * V.ny >= (1L << 21) ? 6 : 30; }

int tune_lb_fp64(const LBView<double>& V, int twall, cudaStream_t s, float* best_ms) {
  return tune<double>(V, twall, false, s, tune_reps(V), best_ms);
}
int tune_lb_fp32(const LBView<float>& V, int twall, cudaStream_t s, float* best_ms) {
  return tune<float>(V, twall, false, s, tune_reps(V), best_ms);
}

// ms per launch of one shape, storing what the view stores
template <typename Real>
static float time_lb(const LBView<Real>& V, int twall, int shape, cudaStream_t s) {
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  const int reps = std::max(3, tune_reps(V) / 5);  // (compared with twice its time: a coarse look)
  float best = 1e30f;
  for (int round = 0; round < 2; round++) {
    for (int r = -1; r < reps; r++) {
      if (r == 0) cudaEventRecord(a, s);
      if constexpr (std::is_same<Real, double>::value) launch_lb_fp64(V, twall, false, shape, s, true);
      else launch_lb_fp32(V, twall, shape, s, true);
    }
    cudaEventRecord(b, s);
    cudaEventSynchronize(b);
    float ms = 1e30f;
    cudaEventElapsedTime(&ms, a, b);
    best = std::min(best, ms);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  return best / reps;
}
float time_lb_fp32(const LBView<float>& V, int twall, int shape, cudaStream_t s) {
  return time_lb<float>(V, twall, shape, s);
}
float time_lb_fp64(const LBView<double>& V, int twall, int shape, cudaStream_t s) {
  return time_lb<double>(V, twall, shape, s);
}

// two steps per launch: V1 is step n (its pops and F outputs unused), V2 step
// n+1 (its pop and F inputs unused)
cudaError_t launch_pair_fp32(const LBView<float>& V1, const LBView<float>& V2, int shape, cudaStream_t s, bool pdl,
                             const PJob<float>* job) {
  return launch_pair<float>(V1, V2, shape, s, pdl, job);
}
cudaError_t launch_pair_fp64(const LBView<double>& V1, const LBView<double>& V2, int shape, cudaStream_t s, bool pdl,
                             const PJob<double>* job) {
  return launch_pair<double>(V1, V2, shape, s, pdl, job);
}

// pair shape autotuner: as tune(), the trial launches write only what the
// views store, buffers the real steps overwrite
template <typename Real>
static int tune_pair(const LBView<Real>& A, const LBView<Real>& B, cudaStream_t s, float* best_ms) {
  const LBView<Real>&V1 = A, &V2 = B;
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  const int reps = tune_reps(V1);
  float shape_ms[NUM_PAIR_SHAPES];
  for (float& m : shape_ms) m = 1e30f;
  for (int round = 0; round < 2; round++) {  // (as tune(): each shape's faster round)
    for (int sh = 0; sh < NUM_PAIR_SHAPES; sh++) {
      if (launch_pair<Real>(V1, V2, sh, s, true) != cudaSuccess) {
        cudaGetLastError();
        continue;
      }
      cudaEventRecord(a, s);
      for (int r = 0; r < reps; r++) launch_pair<Real>(V1, V2, sh, s, true);
      cudaEventRecord(b, s);
      cudaEventSynchronize(b);
      float ms = 0.f;
      cudaEventElapsedTime(&ms, a, b);
      shape_ms[sh] = std::min(shape_ms[sh], ms);
    }
  }
  int best = 0;
  float bt = 1e30f;
  for (int sh = 0; sh < NUM_PAIR_SHAPES; sh++)
    if (shape_ms[sh] < bt) { bt = shape_ms[sh]; best = sh; }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (best_ms) *best_ms = bt / reps;
  return best;
}
// the four-step launch shapes, timed as tune_pair's
template <typename Real>
static int tune_quad(const LBView<Real> (&V)[4], cudaStream_t s, float* best_ms) {
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  const int reps = std::max(3, tune_reps(V[0]) / 2);
  int best = 0;
  float bt = 1e30f;
  for (int round = 0; round < 2; round++) {
    for (int sh = 0; sh < NUM_QUAD_SHAPES; sh++) {
      if (launch_quad<Real>(V, sh, s, true) != cudaSuccess) {
        cudaGetLastError();
        continue;
      }
      cudaEventRecord(a, s);
      for (int r = 0; r < reps; r++) launch_quad<Real>(V, sh, s, true);
      cudaEventRecord(b, s);
      cudaEventSynchronize(b);
      float ms = 1e30f;
      cudaEventElapsedTime(&ms, a, b);
      if (ms < bt) bt = ms, best = sh;
    }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (best_ms) *best_ms = bt / reps;
  return best;
}
int tune_quad_fp32(const LBView<float> (&V)[4], cudaStream_t s, float* best_ms) {
  return tune_quad<float>(V, s, best_ms);
}
int tune_quad_fp64(const LBView<double> (&V)[4], cudaStream_t s, float* best_ms) {
  return tune_quad<double>(V, s, best_ms);
}
int tune_pair_fp32(const LBView<float>& V1, const LBView<float>& V2, cudaStream_t s, float* best_ms) {
  return tune_pair<float>(V1, V2, s, best_ms);
}
int tune_pair_fp64(const LBView<double>& V1, const LBView<double>& V2, cudaStream_t s, float* best_ms) {
  return tune_pair<double>(V1, V2, s, best_ms);
}

}  // namespace lbrb
