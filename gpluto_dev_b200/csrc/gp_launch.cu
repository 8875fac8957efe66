// gp_launch.cu -- template dispatch of the stage kernels.
//
// Compiled twice: with GP_MIXED=0 (FP64 everywhere, -fmad=false so that the
// plain form keeps the reference's rounding sequence) and GP_MIXED=1 (FP32
// reconstruction/limiter/Riemann/EMF arithmetic, FP64 accumulation, CT
// update and con2prim).  In the mixed form the per-direction flux
// differences, inverse-dt terms, UCT face data and edge EMFs -- all computed
// from FP32 fluxes -- are stored as float (the StageDesc pointers then point
// at float arrays); the FP64 form stores them as double.
#include "gp_kernels.cuh"
#include "gp_launch.h"

#ifndef GP_MIXED
#define GP_MIXED 0
#endif
// GP_PART selects the schemes this unit instantiates (0 HD, 1 MHD HLLD with
// the upwind EMFs, 2 RMHD HLLD, 3 MHD with Lax-Friedrichs/HLLC, 4 RMHD with
// HLL/Lax-Friedrichs, 5 the other MHD HLLD and HLL schemes), so that the build
// compiles them in parallel; the entry points
// launch_stage_{fp64,mixed}_p<part> are joined by gp_launch_dispatch.cu.
#ifndef GP_PART
#error "compile gp_launch.cu with -DGP_PART=0 .. 5"
#endif
#define GP_CAT2(a, b) a##b
#define GP_CAT(a, b) GP_CAT2(a, b)

namespace gp {

#if GP_MIXED
using RT = float;
using CTT = float;
#define GP_LAUNCH_STAGE GP_CAT(launch_stage_mixed_p, GP_PART)
#else
using RT = double;
using CTT = double;
#define GP_LAUNCH_STAGE GP_CAT(launch_stage_fp64_p, GP_PART)
#endif

static StageArgs<CTT> make_args(const StageDesc& d) {
  StageArgs<CTT> a;
  a.V = d.V;
  for (int q = 0; q < 3; q++) {
    a.Bs[q] = d.Bs[q];
    a.Bs0[q] = d.Bs0[q];
    a.Bsout[q] = d.Bsout[q];
    a.Ee[q] = reinterpret_cast<CTT*>(d.Ee[q]);
    a.dx[q] = d.dx[q];
    a.inv_dx[q] = fixed_inv(d.dx[q]);
    for (int r = 0; r < 6; r++) a.ct[q][r] = static_cast<CTT*>(d.ct[q][r]);
  }
  a.dtdx = d.dtdx;
  a.dU = reinterpret_cast<CTT*>(d.dU);
  a.Cdt = reinterpret_cast<CTT*>(d.Cdt);
  a.U0 = d.U0;
  a.Uc = d.Uc;
  a.Uout = d.Uout;
  a.Vout = d.Vout;
  a.gamma = d.gamma;
  a.inv_gm1 = gamma_inv(d.gamma);
  a.small_rho = d.small_rho;
  a.small_prs = d.small_prs;
  a.stage = d.stage;
  a.w0 = d.w0;
  a.w1 = d.w1;
  a.wr = d.wr;
  a.invdt_bits = d.invdt_bits;
  a.err = d.err;
  return a;
}

// Grids up to this many cells are launched early.  Above it the launches' latency is
// hidden anyway and it depends on the form (four steps, late -> early): MHD FP64 126^3
// 5394 -> 5424 us, 160^3 10156 -> 10250, RMHD 112^3 22265 -> 22448, HD 126^3 1967 ->
// 1933, MHD mixed 126^3 3528 -> 3483; 256^3 MHD one step FP64 +1%, mixed +1.5%.
constexpr long long kEarlyCells = 1LL << 20;

// Forms that sweep all directions in one launch (sweeps_kernel)
constexpr bool one_sweep_launch(int physics, bool mixed) {
  return physics == PHYS_MHD || (physics == PHYS_HD && mixed);
}

// How the kernels of a stage are launched.
struct How {
  bool early;  // blocks placed while the kernel before drains (step_order)
  int split;   // percent of an SM's memory that is shared memory (0: the driver's choice)
};

// Where two kernels in a row want different splits, the second one's blocks wait
// until the SM is empty.  FP32 MP5 and WENO-Z in 3-D do (sweeps 4 blocks of 35 KB, EMF
// tiles 3 of 54 KB, finish none), and on small grids that costs more than an EMF block
// fewer: with the sweeps' split for all, MP5 32^3 190 -> 135 us a step, 48^3 263 -> 229,
// 64^3 370 -> 340, WENO-Z 272 -> 251; from 2^18 cells on it loses (MP5 64x64x80 416 ->
// 426, 80^3 612 -> 631).
template <int PHYS, int NDIM, int LIM>
static How how_to_launch(long long cells) {
  const bool fix = PHYS == PHYS_MHD && NDIM == 3 && sizeof(RT) == 4 && five_point<LIM>();
  return How{cells <= kEarlyCells, fix && cells <= (1LL << 18) ? 64 : 0};
}

// Launch in stream order
template <typename... K, typename... A>
static void launch(How how, void (*k)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                   A... args) {
  cudaLaunchAttribute at[2];
  unsigned n = 0;
  if (how.early) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (how.split) {
    at[n].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at[n++].val.sharedMemCarveout = how.split;
  }
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = at;
  c.numAttrs = n;
  cudaLaunchKernelEx(&c, k, K(args)...);
}

// Parts an x-row is swept in.  A warp solves 32 faces at a time and a part
// one face more than its cells, so k chunks hold 32 k - 1 cells; a whole
// periodic row needs no extra face.  The count with the fewest (waves of
// resident warps) x (chunks, + 1 for the start-up) is taken: one for grids
// that fill the SMs with whole rows.
template <int LIM>
static int x_segments(int nx, long long rows, int blocks_per_sm) {
  if (LIM == LIM_PPM || five_point<LIM>()) return 1;
  const long long resident = 148LL * blocks_per_sm * (SWEEP_THREADS / 32);
  auto cost = [&](int nseg, int chunks) {
    return (rows * nseg + resident - 1) / resident * (chunks + 1);
  };
  int best = 1;
  long long c = cost(1, (nx + 31) / 32);
  for (int k = (nx + 31) / 32; k >= 1; k--) {
    const int nseg = (nx + 32 * k - 2) / (32 * k - 1);
    if (nseg > 1 && cost(nseg, k) < c) {
      c = cost(nseg, k);
      best = nseg;
    }
  }
  return best;
}

// Cells a thread of a y or z sweep marches over, for `cols` blocks of columns
// of nd cells: the length with the fewest (waves of resident blocks) x (cells
// marched, + 2 for the start-up and the face at the end).  A last wave that
// fills few SMs costs a whole wave, and a grid that does not fill them takes
// the shortest march.
static int march_length(long long cols, int nd, int blocks_per_sm) {
  const long long resident = 148LL * blocks_per_sm;
  int best = 1;
  long long c = 0;
  for (int len = 1; len <= nd && len <= 128; len++) {
    const int nseg = (nd + len - 1) / len;
    const long long q = (cols * nseg + resident - 1) / resident * (len + 2);
    if (len == 1 || q <= c) {
      c = q;
      best = len;
    }
  }
  return best;
}

// y or z sweep over nt transverse positions of nd cells: grid (x-blocks,
// transverse index x pencil segments), flat when nx is not a multiple of the
// block (sweep_m_kernel)
template <int PHYS, int NV, int NDIM, int RS, int CT, int LIM, int DIR>
static void launch_m(const StageArgs<CTT>& a, const Grid3& g, int nt, int nd, cudaStream_t s) {
  const How how = how_to_launch<PHYS, NDIM, LIM>(g.n);
  const long long cols = ((long long)g.nx * nt + SWEEP_THREADS - 1) / SWEEP_THREADS;
  const int seg = march_length(cols, nd, sweep_m_minb<PHYS, RT>());
  const int nseg = (nd + seg - 1) / seg;
  const bool flat = g.nx % SWEEP_THREADS != 0 || (long long)nt * nseg > 65535;
  const dim3 grid = flat ? dim3((unsigned)(cols * nseg)) : dim3(g.nx / SWEEP_THREADS, nt * nseg);
  launch(how, sweep_m_kernel<PHYS, NV, NDIM, RS, CT, LIM, DIR, RT, CTT>, grid, SWEEP_THREADS, 0, s,
         a, g, seg, flat);
}

// blocks of an x-sweep whose rows are in nseg parts
static unsigned x_blocks(long long rows, int nseg) {
  const int wpb = SWEEP_THREADS / 32;
  return (unsigned)((rows * nseg + wpb - 1) / wpb);
}

// The sweeps of a stage in one launch; with `each` in one launch a direction of the
// same kernel (x, y, z), so that profiled steps keep the bits.
template <int PHYS, int NV, int NDIM, int RS, int CT, int LIM, typename F1, typename F2>
static void launch_sweeps(const StageArgs<CTT>& a, const Grid3& g, cudaStream_t s, bool each,
                          F1& pre, F2& post) {
  constexpr int per_sm = sweeps_minb<PHYS, RT>();
  const How how = how_to_launch<PHYS, NDIM, LIM>(g.n);
  const long long rows = (long long)g.ny * g.nz;
  SweepSplit sp = {};
  sp.xseg = x_segments<LIM>(g.nx, rows, per_sm);
  const long long cy = ((long long)g.nx * g.nz + SWEEP_THREADS - 1) / SWEEP_THREADS;
  sp.len[0] = march_length(cy, g.ny, per_sm);
  sp.nb[1] = (int)(cy * ((g.ny + sp.len[0] - 1) / sp.len[0]));
  if (NDIM == 3) {
    const long long cz = ((long long)g.nx * g.ny + SWEEP_THREADS - 1) / SWEEP_THREADS;
    sp.len[1] = march_length(cz, g.nz, per_sm);
    sp.nb[0] = (int)(cz * ((g.nz + sp.len[1] - 1) / sp.len[1]));
  }
  const unsigned nbx = x_blocks(rows, sp.xseg);
  sp.total = sp.nb[0] + sp.nb[1] + (int)nbx;
  auto blocks = [&](unsigned first, unsigned count) {
    sp.first = (int)first;
    pre();
    // FP32 rows in one part keep their shuffles and carry (256^3: 546 us against
    // 600 through shared memory, which is what parts of rows need)
    if (whole_row_form<LIM, RT>() && sp.xseg == 1)
      launch(how, sweeps_kernel<PHYS, NV, NDIM, RS, CT, LIM, whole_row_form<LIM, RT>(), RT, CTT>,
             count, SWEEP_THREADS, 0, s, a, g, sp);
    else
      launch(how, sweeps_kernel<PHYS, NV, NDIM, RS, CT, LIM, false, RT, CTT>, count, SWEEP_THREADS,
             0, s, a, g, sp);
    post();
  };
  if (!each) {
    // Blocks run in their order once the SMs are full, so the direction with the
    // longest ones goes first: x where its rows have more chunks than the marches cells
    // (PPM, MP5 and WENO-Z do not cut rows).  700^2, x last -> first: PPM 469 -> 395 us a
    // step, mixed 279 -> 238, MP5 589 -> 527, mixed 330 -> 306; with shorter rows x first
    // loses (64^3 PPM 306 -> 344), and so it does where all blocks fit (300x200 MP5 204 ->
    // 215).
    const int chunks = (g.nx / sp.xseg + 31) / 32;
    const bool x_first = sp.total > 148 * per_sm && chunks > std::max(sp.len[0], sp.len[1]) + 1;
    blocks(x_first ? sp.nb[0] + sp.nb[1] : 0, sp.total);
    return;
  }
  blocks(sp.nb[0] + sp.nb[1], nbx);
  blocks(sp.nb[0], sp.nb[1]);
  if (NDIM == 3) blocks(0, sp.nb[0]);
}

template <int PHYS, int NV, int NDIM, int RS, int CT, int LIM>
static void run_stage(const StageArgs<CTT>& a, const GridDims& gd, cudaStream_t s,
                      cudaEvent_t* ev) {
  Grid3 g{gd.nx, gd.ny, gd.nz, gd.n, gd.outflow};
  for (int d = 0; d < 3; d++) {
    g.ilo[d] = gd.ilo[d];
    g.ihi[d] = gd.ihi[d];
    g.glo[d] = gd.glo[d];
    g.ghi[d] = gd.ghi[d];
  }
  const How how = how_to_launch<PHYS, NDIM, LIM>(gd.n);
  int kidx = 0;
  auto pre = [&]() { if (ev) cudaEventRecord(ev[2 * kidx], s); };
  auto post = [&]() { if (ev) cudaEventRecord(ev[2 * kidx + 1], s); kidx++; };
  if constexpr (one_sweep_launch(PHYS, sizeof(RT) == 4)) {
    static_assert(!sum_directions<PHYS, CTT>(), "the sweeps read one another's sums");
    launch_sweeps<PHYS, NV, NDIM, RS, CT, LIM>(a, g, s, ev != nullptr, pre, post);
  } else {
    const int rows = gd.ny * gd.nz;
    const int nseg = x_segments<LIM>(gd.nx, rows, sweep_x_minb<PHYS, RT>());
    const unsigned grid = x_blocks(rows, nseg);
    pre();
    if (whole_row_form<LIM, RT>() && nseg == 1)
      launch(how, sweep_x_kernel<PHYS, NV, NDIM, RS, CT, LIM, whole_row_form<LIM, RT>(), RT, CTT>,
             grid, SWEEP_THREADS, 0, s, a, g, nseg);
    else
      launch(how, sweep_x_kernel<PHYS, NV, NDIM, RS, CT, LIM, false, RT, CTT>, grid, SWEEP_THREADS,
             0, s, a, g, nseg);
    post();
    pre();
    launch_m<PHYS, NV, NDIM, RS, CT, LIM, 1>(a, g, gd.nz, gd.ny, s);
    post();
    if constexpr (NDIM == 3) {
      pre();
      launch_m<PHYS, NV, NDIM, RS, CT, LIM, 2>(a, g, gd.ny, gd.nz, s);
      post();
    }
  }
  const unsigned nb = (unsigned)((gd.n + 255) / 256);
  if constexpr (PHYS != PHYS_HD) {
    pre();
    if constexpr (CT == CT_ARITH) {
      launch(how, emf_arith_kernel<NDIM, RT, CTT>, nb, 256, 0, s, a, g);
    } else if constexpr (CT == CT_CONTACT) {
      launch(how, emf_contact_kernel<NDIM, RT, CTT>, nb, 256, 0, s, a, g);
    } else if constexpr (NDIM == 3 && (sizeof(RT) == 8 || five_point<LIM>())) {  // plane-staged EMF
      using T = EmfTile<LIM, CTT>;
      cudaFuncSetAttribute(emf_tile_kernel<LIM, RT, CTT>,
                           cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM);
      // the longest segment (<= ET_SEGMENT planes) that still gives about
      // four waves of resident blocks over 148 SMs
      const long long cols = (long long)((gd.nx + ETX - 1) / ETX) * ((gd.ny + ETY - 1) / ETY);
      int sz = ET_SEGMENT;
      while (sz > 4 && cols * ((gd.nz + sz - 1) / sz) < 148LL * emf_tile_minb<RT>() * 4) sz /= 2;
      dim3 grid((gd.nx + ETX - 1) / ETX, (gd.ny + ETY - 1) / ETY, (gd.nz + sz - 1) / sz);
      launch(how, emf_tile_kernel<LIM, RT, CTT>, grid, dim3(ETX, ETY), T::SMEM, s, a, g, sz);
    } else if constexpr (NDIM == 3) {  // mixed PLM/PPM: z-marching EMF, loads through L1
      // the longest segment (<= EMF_SEGMENT planes) that still gives about
      // four waves of blocks over 148 SMs (3 blocks per SM)
      const long long cols = (long long)((gd.nx + EMF_TX - 1) / EMF_TX) *
                             ((gd.ny + EMF_TY - 1) / EMF_TY);
      int sz = EMF_SEGMENT;
      while (sz > 4 && cols * ((gd.nz + sz - 1) / sz) < 148LL * 3 * 4) sz /= 2;
      dim3 grid((gd.nx + EMF_TX - 1) / EMF_TX, (gd.ny + EMF_TY - 1) / EMF_TY,
                (gd.nz + sz - 1) / sz);
      launch(how, emf_march_kernel<LIM, RT, CTT>, grid, dim3(EMF_TX, EMF_TY), 0, s, a, g, sz);
    } else {
      launch(how, emf_kernel<NDIM, LIM, RT, CTT>, nb, 256, 0, s, a, g);
    }
    post();
  }
  pre();
  launch(how, finish_kernel<PHYS, NV, NDIM, CTT>, nb, 256, 0, s, a, g);
  post();
}

template <int PHYS, int NV, int NDIM, int RS, int CT>
static int by_lim(const StageArgs<CTT>& a, const GridDims& g, int lim, cudaStream_t s,
                  cudaEvent_t* ev) {
  switch (lim) {
    case LIM_MC: run_stage<PHYS, NV, NDIM, RS, CT, LIM_MC>(a, g, s, ev); return 0;
    case LIM_VL: run_stage<PHYS, NV, NDIM, RS, CT, LIM_VL>(a, g, s, ev); return 0;
    case LIM_MINMOD: run_stage<PHYS, NV, NDIM, RS, CT, LIM_MINMOD>(a, g, s, ev); return 0;
    case LIM_PPM: run_stage<PHYS, NV, NDIM, RS, CT, LIM_PPM>(a, g, s, ev); return 0;
    case LIM_MP5: run_stage<PHYS, NV, NDIM, RS, CT, LIM_MP5>(a, g, s, ev); return 0;
    case LIM_WENOZ: run_stage<PHYS, NV, NDIM, RS, CT, LIM_WENOZ>(a, g, s, ev); return 0;
    case LIM_LIMO3: run_stage<PHYS, NV, NDIM, RS, CT, LIM_LIMO3>(a, g, s, ev); return 0;
    case LIM_WENO3: run_stage<PHYS, NV, NDIM, RS, CT, LIM_WENO3>(a, g, s, ev); return 0;
    case LIM_FLAT: run_stage<PHYS, NV, NDIM, RS, CT, LIM_FLAT>(a, g, s, ev); return 0;
    case LIM_VANALBADA:
      run_stage<PHYS, NV, NDIM, RS, CT, LIM_VANALBADA>(a, g, s, ev);
      return 0;
    case LIM_OSPRE: run_stage<PHYS, NV, NDIM, RS, CT, LIM_OSPRE>(a, g, s, ev); return 0;
    case LIM_UMIST: run_stage<PHYS, NV, NDIM, RS, CT, LIM_UMIST>(a, g, s, ev); return 0;
    default: return -1;
  }
}

template <int NDIM>
static int by_scheme(const StageArgs<CTT>& a, const GridDims& g, const SchemeKey& k,
                     cudaStream_t s, cudaEvent_t* ev) {
#if GP_PART == 1
  if (k.physics == PHYS_MHD && k.riemann == RS_HLLD) {
    if (k.ct == CT_UCT_HLLD)
      return by_lim<PHYS_MHD, 8, NDIM, RS_HLLD, CT_UCT_HLLD>(a, g, k.limiter, s, ev);
    if (k.ct == CT_UCT_HLL)
      return by_lim<PHYS_MHD, 8, NDIM, RS_HLLD, CT_UCT_HLL>(a, g, k.limiter, s, ev);
  }
#endif
#if GP_PART == 5
  if (k.physics == PHYS_MHD && k.riemann == RS_HLLD) {
    if (k.ct == CT_CONTACT)
      return by_lim<PHYS_MHD, 8, NDIM, RS_HLLD, CT_CONTACT>(a, g, k.limiter, s, ev);
    if (k.ct == CT_ARITH)
      return by_lim<PHYS_MHD, 8, NDIM, RS_HLLD, CT_ARITH>(a, g, k.limiter, s, ev);
  }
  if (k.physics == PHYS_MHD && k.riemann == RS_HLL) {
    if (k.ct == CT_CONTACT)
      return by_lim<PHYS_MHD, 8, NDIM, RS_HLL, CT_CONTACT>(a, g, k.limiter, s, ev);
    if (k.ct == CT_ARITH)
      return by_lim<PHYS_MHD, 8, NDIM, RS_HLL, CT_ARITH>(a, g, k.limiter, s, ev);
    if (k.ct == CT_UCT_HLL)
      return by_lim<PHYS_MHD, 8, NDIM, RS_HLL, CT_UCT_HLL>(a, g, k.limiter, s, ev);
  }
#endif
#if GP_PART == 3
  // MHD with the Lax-Friedrichs and HLLC solvers (UCT_HLL, ARITHMETIC or CT_CONTACT)
  if (k.physics == PHYS_MHD && k.ct == CT_CONTACT) {
    if (k.riemann == RS_TVDLF)
      return by_lim<PHYS_MHD, 8, NDIM, RS_TVDLF, CT_CONTACT>(a, g, k.limiter, s, ev);
    if (k.riemann == RS_HLLC)
      return by_lim<PHYS_MHD, 8, NDIM, RS_HLLC, CT_CONTACT>(a, g, k.limiter, s, ev);
    return -1;
  }
  if (k.physics == PHYS_MHD && k.ct == CT_ARITH) {
    if (k.riemann == RS_TVDLF)
      return by_lim<PHYS_MHD, 8, NDIM, RS_TVDLF, CT_ARITH>(a, g, k.limiter, s, ev);
    if (k.riemann == RS_HLLC)
      return by_lim<PHYS_MHD, 8, NDIM, RS_HLLC, CT_ARITH>(a, g, k.limiter, s, ev);
    return -1;
  }
  if (k.physics == PHYS_MHD) {
    if (k.riemann == RS_TVDLF && k.ct == CT_UCT_HLL)
      return by_lim<PHYS_MHD, 8, NDIM, RS_TVDLF, CT_UCT_HLL>(a, g, k.limiter, s, ev);
    if (k.riemann == RS_HLLC && k.ct == CT_UCT_HLL)
      return by_lim<PHYS_MHD, 8, NDIM, RS_HLLC, CT_UCT_HLL>(a, g, k.limiter, s, ev);
    return -1;
  }
#endif
#if GP_PART == 2
  if (k.physics == PHYS_RMHD && k.riemann == RS_HLLD && k.ct == CT_UCT_HLL)
    return by_lim<PHYS_RMHD, 8, NDIM, RS_HLLD, CT_UCT_HLL>(a, g, k.limiter, s, ev);
#endif
#if GP_PART == 4
  if (k.physics == PHYS_RMHD && k.ct == CT_UCT_HLL) {
    if (k.riemann == RS_HLL)
      return by_lim<PHYS_RMHD, 8, NDIM, RS_HLL, CT_UCT_HLL>(a, g, k.limiter, s, ev);
    if (k.riemann == RS_TVDLF)
      return by_lim<PHYS_RMHD, 8, NDIM, RS_TVDLF, CT_UCT_HLL>(a, g, k.limiter, s, ev);
  }
#endif
#if GP_PART == 0
  if (k.physics == PHYS_HD) {
    if (k.riemann == RS_HLLC) return by_lim<PHYS_HD, 5, NDIM, RS_HLLC, 0>(a, g, k.limiter, s, ev);
    if (k.riemann == RS_HLL) return by_lim<PHYS_HD, 5, NDIM, RS_HLL, 0>(a, g, k.limiter, s, ev);
    if (k.riemann == RS_TVDLF)
      return by_lim<PHYS_HD, 5, NDIM, RS_TVDLF, 0>(a, g, k.limiter, s, ev);
    return -1;
  }
#endif
  return -1;
}

int GP_LAUNCH_STAGE(const StageDesc& d, const GridDims& g, const SchemeKey& k,
                    cudaStream_t s, cudaEvent_t* ev) {
  StageArgs<CTT> a = make_args(d);
  if (k.ndim == 2) return by_scheme<2>(a, g, k, s, ev);
  if (k.ndim == 3) return by_scheme<3>(a, g, k, s, ev);
  return -1;
}

#if !GP_MIXED && GP_PART == 1
int launch_prim2cons(int physics, const double* V, double* U, long long n, double gamma,
                     cudaStream_t s) {
  const unsigned nb = (unsigned)((n + 255) / 256);
  if (physics == PHYS_MHD) prim2cons_kernel<PHYS_MHD, 8><<<nb, 256, 0, s>>>(V, U, n, gamma);
  else if (physics == PHYS_RMHD) prim2cons_kernel<PHYS_RMHD, 8><<<nb, 256, 0, s>>>(V, U, n, gamma);
  else if (physics == PHYS_HD) prim2cons_kernel<PHYS_HD, 5><<<nb, 256, 0, s>>>(V, U, n, gamma);
  else return -1;
  return 0;
}

int stage_launch_count(const SchemeKey& k) {
  int c = 1 + (k.ndim == 3 ? 2 : 1) + 1;  // sweeps + finish
  if (k.physics != PHYS_HD) c += 1;       // emf
  return c;
}

int stage_launches(const SchemeKey& k, bool mixed) {
  return stage_launch_count(k) - (one_sweep_launch(k.physics, mixed) ? k.ndim - 1 : 0);
}

const char* stage_kernel_name(const SchemeKey& k, int idx) {
  static const char* n3m[] = {"sweep_x", "sweep_y", "sweep_z", "emf", "finish"};
  static const char* n2m[] = {"sweep_x", "sweep_y", "emf", "finish"};
  static const char* n3h[] = {"sweep_x", "sweep_y", "sweep_z", "finish"};
  static const char* n2h[] = {"sweep_x", "sweep_y", "finish"};
  if (idx < 0 || idx >= stage_launch_count(k)) return "?";
  if (k.physics != PHYS_HD) return k.ndim == 3 ? n3m[idx] : n2m[idx];
  return k.ndim == 3 ? n3h[idx] : n2h[idx];
}
#endif

}  // namespace gp
