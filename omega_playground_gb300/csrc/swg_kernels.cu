// Tendency, stage-update and diagnostic kernels of the GB300 shallow-water
// path (sm_103a, FP64).
//
// GB300 issues FP64 at 1/64 of its FP32 rate (about 0.6 T DFMA/s), so one
// tendency evaluation is bound by FP64 instructions, not by HBM.  The
// kernels are arranged to issue as few FP64 instructions per cell-level as
// possible:
//  - every intermediate is computed exactly once per stage and kept in
//    HBM/L2 for its consumers (no halo recomputation);
//  - all K-independent factors are folded into per-entity coefficient tables
//    (loaded as warp-broadcasts) and zero TRiSK weights are dropped;
//  - tracer terms are rewritten as weighted sums over neighbour values whose
//    weights are shared by all tracers of a cell;
//  - the wide sums (PV flux, tracers, tracer Laplacians; in large models also
//    the vertex and divergence sums) run on the integer pipes in fixed point
//    (swg_fixed.cuh), which idle beside FP64;
//  - sums and products by themselves are multiply-adds with all operands in
//    registers, which issue faster (mul_reg, swg_device.cuh);
//  - reciprocals are one third-order step from the hardware approximation (3
//    FP64 instructions instead of about 9 for IEEE division);
//  - the RK stage update is fused into the last two kernels.
// One thread handles one (entity, level); k is the fastest index, so a warp
// reads 32 consecutive levels (256 contiguous bytes) of one entity.
//
// Reference functors restated (omega_playground src/model/...):
//   k_vertex    vorticity_aux.hpp:294-325        (rvort, PV at vertices)
//   k_cell1     kinetic_aux.hpp:50-79, tracer_aux.hpp:181-201
//   k_edge1     thickness_aux.hpp:123-142, vorticity_aux.hpp:327-341,
//               vel_hyperdiff_edge.hpp:237-261 / vel_diff_edge.hpp:72-81
//   k_aux2      kinetic_aux.hpp:59-71 (ke), vel_hyperdiff_edge.hpp:263-307,
//               tracer_hyperdiff_cell.hpp:301-336
//   k_edge_final pv_flux_edge.hpp:149-177, ke_grad_edge.hpp:223-237,
//               ssh_grad_edge.hpp:281-294, vel_diff_edge.hpp:61-86,
//               vel_hyperdiff_edge.hpp:309-334, rk4.cpp:94-138, lsrk.cpp:47-86
//   k_cell_final (k_cell_tracers with fixed-point sums) thickness_hadv_cell.hpp:59-83, tracer_hadv_cell.hpp:60-90,
//               tracer_diff_cell.hpp:162-193, tracer_hyperdiff_cell.hpp:338-368
#include "swg_device.cuh"

#include <algorithm>
#include <type_traits>
#include <cstring>

namespace swg {
namespace {

constexpr int TPB = 256;

// Shape of a kernel without or with fixed-point sums (see HTPB)
template <bool FX> struct Shape {
  static constexpr int threads = TPB, aux2_blocks = 0, edge_blocks = 0;
};
template <> struct Shape<true> {
  // edge_blocks: 256x256x64: 500 us with 12, 487 with 14, 513 with 16
  static constexpr int threads = HTPB, aux2_blocks = HEAVY_AUX2_BLOCKS,
                       edge_blocks = 14;
};

// The minimum of resident blocks that bounds the registers of k_vertex and
// k_cell1 with fixed-point sums (RAW): 8 gives 32, 6 gives 40.  256x256 cells,
// 64 levels: k_vertex 184 us in FP64, 133 with 34 registers, 118 with 32;
// 64x64x64, 1 tracer: k_cell1 12.1 us in FP64, 10.1 with 40, 12.3 with 32.

// Single-instance kernels: one launch per pass over (entity, level),
// templated on the value type (double, or Dual for the tangent-linear model).
template <class T, int RAW>
__global__ void __launch_bounds__(TPB, RAW ? 8 : 0)
    k_vertex(MeshView m, ModelView p, AuxViewT<T> a, const T *__restrict__ h,
             const T *__restrict__ vn) {
  const unsigned i = blockIdx.x * TPB + threadIdx.x;
  if (i < unsigned(m.nvertices) * unsigned(m.nlayers))
    pt_vertex<T, RAW>(m, p, a, h, vn, i);
}

template <class T, int RAW>
__global__ void __launch_bounds__(TPB, RAW ? 6 : 0)
    k_cell1(MeshView m, ModelView p, AuxViewT<T> a, const T *__restrict__ h,
            const T *__restrict__ vn, const T *__restrict__ tr) {
  const unsigned i = blockIdx.x * TPB + threadIdx.x;
  if (i < unsigned(m.ncells) * unsigned(m.nlayers))
    pt_cell1<T, RAW>(m, p, a, h, vn, tr, i);
}

template <class T>
__global__ void __launch_bounds__(TPB)
    k_edge1(MeshView m, ModelView p, AuxViewT<T> a, const T *__restrict__ h,
            const T *__restrict__ vn) {
  const unsigned i = blockIdx.x * TPB + threadIdx.x;
  if (i < unsigned(m.nedges) * unsigned(m.nlayers))
    pt_edge1<T>(m, p, a, h, vn, i);
}

// TR4 as in pt_aux2
template <class T, int TR4>
__global__ void __launch_bounds__(Shape<TR4 == 2>::threads,
                                  Shape<TR4 == 2>::aux2_blocks)
    k_aux2(MeshView m, ModelView p, AuxViewT<T> a, unsigned base) {
  const unsigned i = base + blockIdx.x * blockDim.x + threadIdx.x;
  if (i < unsigned(m.nvertices + m.ncells) * unsigned(m.nlayers))
    pt_aux2<T, TR4>(m, p, a, i);
}

template <int NE, class T, bool FX>
__global__ void __launch_bounds__(Shape<FX>::threads, Shape<FX>::edge_blocks)
    k_edge_final(MeshView m, ModelView p, AuxViewT<T> a, StageArgsT<T> s) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < unsigned(m.nedges) * unsigned(m.nlayers))
    pt_edge_final<NE, T, FX>(m, p, a, s, i);
}

template <int NE>
__global__ void __launch_bounds__(HTPB)
    k_pv_sum(MeshView m, AuxView a) {
  const unsigned i = blockIdx.x * HTPB + threadIdx.x;
  if (i < unsigned(m.nedges) * unsigned(m.nlayers))
    pt_pv_sum<NE>(m, a, i);
}

template <class T>
__global__ void __launch_bounds__(TPB)
    k_cell_final(MeshView m, ModelView p, AuxViewT<T> a, StageArgsT<T> s) {
  const unsigned i = blockIdx.x * TPB + threadIdx.x;
  if (i < unsigned(m.ncells) * unsigned(m.nlayers))
    pt_cell_final<T, 0, false, std::is_same<T, double>::value>(m, p, a, s, i);
}

// fixed-point tracer sums; D4 = tracer del4
template <bool D4>
__global__ void __launch_bounds__(HTPB, HEAVY_CELL_BLOCKS)
    k_cell_tracers(MeshView m, ModelView p, AuxView a, StageArgs s) {
  __shared__ fx_t sm[2 * TR_SLOTS * HTPB];
  const unsigned i = blockIdx.x * HTPB + threadIdx.x;
  if (i < unsigned(m.ncells) * unsigned(m.nlayers))
    pt_cell_final<double, D4 ? 2 : 1, true>(m, p, a, s, i, sm + threadIdx.x,
                                            HTPB);
}

template <int NE, class T>
__global__ void __launch_bounds__(TPB)
    k_lin_edge(MeshView m, ModelView p, StageArgsT<T> s) {
  const unsigned i = blockIdx.x * TPB + threadIdx.x;
  if (i < unsigned(m.nedges) * unsigned(m.nlayers))
    pt_lin_edge<NE, T>(m, p, s, i);
}

template <class T>
__global__ void __launch_bounds__(TPB)
    k_lin_cell(MeshView m, ModelView p, StageArgsT<T> s) {
  const unsigned i = blockIdx.x * TPB + threadIdx.x;
  if (i < unsigned(m.ncells) * unsigned(m.nlayers))
    pt_lin_cell<T>(m, p, s, i);
}

// Small models (below SMALL_EDGE_LEVELS): the two independent pairs of passes
// as one launch each, so a stage is a chain of four launches without the
// fork and join of the pairs (four events).  A launch of such a model takes
// its latency, about 3 us, whatever its passes compute (RK4 step of 12x10
// cells, 3 levels, 2 tracers, launched one by one: 114 us forked, 94 joint).
__global__ void __launch_bounds__(HTPB)
    k_vertex_cell1(MeshView m, ModelView p, AuxView a,
                   const double *__restrict__ h, const double *__restrict__ vn,
                   const double *__restrict__ tr) {
  const unsigned VK = unsigned(m.nvertices) * unsigned(m.nlayers);
  const unsigned i = blockIdx.x * HTPB + threadIdx.x;
  if (i < VK)
    pt_vertex<double, 0>(m, p, a, h, vn, i);
  else if (i - VK < unsigned(m.ncells) * unsigned(m.nlayers))
    pt_cell1<double, 0>(m, p, a, h, vn, tr, i - VK);
}
// blocks below `edge_blocks` take edges, the others cells (not for an
// in-place stage, whose edges read the h that the cells rewrite)
template <int NE>
__global__ void __launch_bounds__(HTPB, HEAVY_CELL_BLOCKS)
    k_final(MeshView m, ModelView p, AuxView a, StageArgs s,
            unsigned edge_blocks) {
  __shared__ fx_t sm[2 * TR_SLOTS * HTPB];
  if (blockIdx.x < edge_blocks) {
    const unsigned i = blockIdx.x * HTPB + threadIdx.x;
    if (i < unsigned(m.nedges) * unsigned(m.nlayers))
      pt_edge_final<NE, double, 0>(m, p, a, s, i);
  } else {
    const unsigned i = (blockIdx.x - edge_blocks) * HTPB + threadIdx.x;
    if (i < unsigned(m.ncells) * unsigned(m.nlayers))
      pt_cell_final<double, -1, true, true>(m, p, a, s, i, sm + threadIdx.x,
                                            HTPB);
  }
}

// Thickness flux of a per-field tendency call (compute_h/vn/tr_tendency):
// F = mean_h vn from the last auxiliary state's mean thickness and the
// caller's normal velocity (pv_flux_edge.hpp and thickness_hadv_cell.hpp
// multiply the two per edge), and with G also F Q for the PV flux; the
// same expressions as pt_edge1, so equal inputs give equal fluxes.
template <bool G>
__global__ void __launch_bounds__(TPB)
    k_field_flux(MeshView m, AuxView a, const double *__restrict__ vn) {
  const unsigned i = blockIdx.x * TPB + threadIdx.x;
  if (i >= unsigned(m.nedges) * unsigned(m.nlayers))
    return;
  const double F = a.mh[i] * vn[i];
  a.F[i] = F;
  if (G)
    store_pv(a, i, F, a.Q[i]);
}

// Elementwise helpers for the unfused stepper path (forcing hook set).
__global__ void k_axpby(double *__restrict__ y, const double *__restrict__ x,
                        const double *__restrict__ z, double alpha,
                        double beta, long long n, int kind) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  switch (kind) {
  case 0: y[i] *= alpha; break;                    // tend *= a
  case 1: y[i] = fma(alpha, x[i], y[i]); break;    // state += dtb * tend
  case 2: y[i] = fma(alpha, x[i], z[i]); break;    // provis = old + dta * tend
  default: y[i] = alpha; break;                    // fill
  }
  (void)beta;
}

// Diagnostics: one partial sum per block, summed on the host in block order.
template <int WHICH>
__global__ void __launch_bounds__(TPB)
    k_diag(MeshView m, ModelView p, const double *__restrict__ h,
           const double *__restrict__ vn, double *partials) {
  __shared__ double red[TPB];
  const int K = m.nlayers;
  const long long n = (WHICH == 2 ? (long long)m.nvertices : m.ncells) * K;
  double s = 0.0;
  for (long long i = blockIdx.x * (long long)TPB + threadIdx.x; i < n;
       i += (long long)gridDim.x * TPB) {
    const int ent = int(i / K), k = int(i - (long long)ent * K);
    const int *maxlev = WHICH == 2 ? m.maxlev_v : m.maxlev_c;
    if (maxlev && k >= maxlev[ent])
      continue;
    if (WHICH == 0) { // mass: area_cell h
      s += m.area_cell_d[ent] * h[i];
    } else if (WHICH == 1) { // energy: area (g h^2/2 + h ke)
      double ke = 0.0;
      for (int j = 0; j < MAXE; ++j) {
        const double u = vn[size_t(m.ec[6 * ent + j]) * K + k];
        ke += m.cke[6 * ent + j] * u * u;
      }
      const double hc = h[i];
      // the linear model's kinetic energy is weighted by h0
      // (shallow_water_hierarchical.cpp:743-771)
      s += m.area_cell_d[ent] *
           (p.grav * hc * hc / 2 + (p.linear ? p.h0 : hc) * ke);
    } else { // circulation: sum_j dc s vn + f area_triangle
      double cir = 0.0;
      for (int j = 0; j < 3; ++j)
        cir += m.dcs_v[3 * ent + j] * vn[size_t(m.ev[3 * ent + j]) * K + k];
      s += cir + p.f_vertex[ent] * m.area_tri_d[ent];
    }
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = TPB / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
      red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    partials[blockIdx.x] = red[0];
}

unsigned nblocks(long long n, int tpb = TPB) {
  return unsigned((n + tpb - 1) / tpb);
}

template <class T>
void launch_aux2(const MeshView &m, const ModelView &p, const AuxViewT<T> &a,
                 cudaStream_t st) {
  const long long K = m.nlayers, VK = m.nvertices * K;
  // vertex threads only when the velocity del4 curl is needed
  const unsigned base = (p.do_vn && p.vel_del4) ? 0u : unsigned(VK);
  const long long n = VK + m.ncells * K - base;
  if (!(p.ntracers > 0 && p.tr_del4)) {
    k_aux2<T, 0><<<nblocks(n), TPB, 0, st>>>(m, p, a, base);
    return;
  }
  if constexpr (std::is_same<T, double>::value)
    if (a.lx) {
      k_aux2<T, 2><<<nblocks(n, HTPB), HTPB, 0, st>>>(m, p, a, base);
      return;
    }
  k_aux2<T, 1><<<nblocks(n), TPB, 0, st>>>(m, p, a, base);
}
template <class T>
void launch_edge_final(const MeshView &m, const ModelView &p,
                       const AuxViewT<T> &a, const StageArgsT<T> &s,
                       cudaStream_t st) {
  const long long n = (long long)m.nedges * m.nlayers;
  if constexpr (std::is_same<T, double>::value)
    if (a.FGx) {
      if (m.ne == 8)
        k_edge_final<8, T, true><<<nblocks(n, HTPB), HTPB, 0, st>>>(m, p, a, s);
      else
        k_edge_final<10, T, true>
            <<<nblocks(n, HTPB), HTPB, 0, st>>>(m, p, a, s);
      return;
    }
  if (m.ne == 8)
    k_edge_final<8, T, false><<<nblocks(n), TPB, 0, st>>>(m, p, a, s);
  else
    k_edge_final<10, T, false><<<nblocks(n), TPB, 0, st>>>(m, p, a, s);
}

template <class T>
void launch_cell_final(const MeshView &m, const ModelView &p,
                       const AuxViewT<T> &a, const StageArgsT<T> &s,
                       cudaStream_t st) {
  const long long n = (long long)m.ncells * m.nlayers;
  if constexpr (std::is_same<T, double>::value)
    if (p.ntracers > 0 && a.nx) {
      if (p.tr_del4)
        k_cell_tracers<true><<<nblocks(n, HTPB), HTPB, 0, st>>>(m, p, a, s);
      else
        k_cell_tracers<false><<<nblocks(n, HTPB), HTPB, 0, st>>>(m, p, a, s);
      return;
    }
  k_cell_final<T><<<nblocks(n), TPB, 0, st>>>(m, p, a, s);
}

// ---- opt-in per-kernel timing: an event pair around every tendency kernel
struct Timed {
  const char *name;
  cudaEvent_t start, stop;
};
std::vector<Timed> g_timed;
bool g_profile = false;
// > 0 while a ProfileOff guard is alive on this thread: launches not timed
thread_local int t_profile_off = 0;

struct Scope {
  const char *name;
  cudaStream_t st;
  cudaEvent_t a = nullptr, b = nullptr;
  Scope(const char *n, cudaStream_t s) : name(n), st(s) {
    if (g_profile && !t_profile_off && cudaEventCreate(&a) == cudaSuccess &&
        cudaEventCreate(&b) == cudaSuccess)
      cudaEventRecord(a, st);
  }
  ~Scope() {
    if (a && b) {
      cudaEventRecord(b, st);
      g_timed.push_back({name, a, b});
    }
    ++g_launches;
  }
};

} // namespace

bool profiling_enabled() { return g_profile; }

ProfileOff::ProfileOff() { ++t_profile_off; }
ProfileOff::~ProfileOff() { --t_profile_off; }

int profile_enable(int on) {
  g_profile = on != 0;
  return SWG_OK;
}

int profile_read(int max_kernels, char *names, double *total_ms,
                 long long *launches, int *count) {
  std::vector<std::string> keys;
  std::vector<double> ms;
  std::vector<long long> n;
  for (auto &t : g_timed) {
    float x = 0.f;
    cudaError_t err = cudaEventSynchronize(t.stop);
    if (err == cudaSuccess)
      err = cudaEventElapsedTime(&x, t.start, t.stop);
    cudaEventDestroy(t.start);
    cudaEventDestroy(t.stop);
    if (err != cudaSuccess) {
      g_timed.clear();
      return cuda_fail(err, "swg_profile_read");
    }
    size_t j = 0;
    while (j < keys.size() && keys[j] != t.name)
      ++j;
    if (j == keys.size()) {
      keys.push_back(t.name);
      ms.push_back(0.0);
      n.push_back(0);
    }
    ms[j] += x;
    n[j] += 1;
  }
  g_timed.clear();
  const int m = std::min<int>(max_kernels, int(keys.size()));
  for (int j = 0; j < m; ++j) {
    std::strncpy(names + 32 * j, keys[j].c_str(), 31);
    names[32 * j + 31] = 0;
    total_ms[j] = ms[j];
    launches[j] = n[j];
  }
  *count = m;
  return SWG_OK;
}

namespace {

// Whether the pairs of passes run as one launch (per-kernel timing keeps them
// apart).  Those sum velocities and thicknesses in FP64: a level slice of a
// model with fixed-point sums of them (p.raw, FGx) keeps the passes apart.
template <class T>
bool small_model(const MeshView &m, const ModelView &p, const AuxViewT<T> &a) {
  if (!std::is_same<T, double>::value || g_profile)
    return false;
  return !a.FGx && !p.raw &&
         (long long)m.nedges * m.nlayers < SMALL_EDGE_LEVELS;
}

template <class T>
void launch_aux_t(const MeshView &m, const ModelView &p, const AuxViewT<T> &a,
                  const T *h, const T *vn, const T *tr, cudaStream_t st,
                  const Fork *fk) {
  const long long K = m.nlayers;
  const long long VK = m.nvertices * K, CK = m.ncells * K, EK = m.nedges * K;
  if (p.linear) // the linear model has no intermediates
    return;
  NvtxRange range("auxstate");
  constexpr int FIXED = std::is_same<T, double>::value; // raw sums possible
  // vertex and cell passes read only the state: independent
  const bool vert = p.do_vn;
  const bool cell1 = (p.do_vn && (p.vel_del2 || p.vel_del4)) || p.ntracers > 0;
  auto run_vertex = [&](cudaStream_t s) {
    Scope sc("k_vertex", s);
    if (FIXED && (p.raw & RAW_VERTEX))
      k_vertex<T, FIXED><<<nblocks(VK), TPB, 0, s>>>(m, p, a, h, vn);
    else
      k_vertex<T, 0><<<nblocks(VK), TPB, 0, s>>>(m, p, a, h, vn);
  };
  auto run_cell1 = [&](cudaStream_t s) {
    Scope sc("k_cell1", s);
    if (FIXED && (p.raw & RAW_DIV))
      k_cell1<T, FIXED><<<nblocks(CK), TPB, 0, s>>>(m, p, a, h, vn, tr);
    else
      k_cell1<T, 0><<<nblocks(CK), TPB, 0, s>>>(m, p, a, h, vn, tr);
  };
  // per-kernel timing (profiling on) runs the passes one after another so
  // that each event pair times its own kernel alone
  if (g_profile)
    fk = nullptr;
  if (vert && cell1 && small_model<T>(m, p, a)) {
    if constexpr (std::is_same<T, double>::value) {
      Scope sc("k_vertex_cell1", st);
      k_vertex_cell1<<<nblocks(VK + CK, HTPB), HTPB, 0, st>>>(m, p, a, h, vn,
                                                              tr);
    }
  } else if (vert && cell1)
    fork_join(fk, st, run_vertex, run_cell1);
  else if (vert)
    run_vertex(st);
  else if (cell1)
    run_cell1(st);
  if (p.do_vn || p.do_h || p.ntracers > 0) {
    Scope sc("k_edge1", st);
    k_edge1<T><<<nblocks(EK), TPB, 0, st>>>(m, p, a, h, vn);
  }
  const bool tr4 = p.ntracers > 0 && p.tr_del4;
  if (p.do_vn || tr4) {
    Scope sc("k_aux2", st);
    launch_aux2<T>(m, p, a, st);
  }
}

template <class T>
void launch_tendency_t(const MeshView &m, const ModelView &p,
                       const AuxViewT<T> &a, const StageArgsT<T> &s,
                       cudaStream_t st, const Fork *fk) {
  const long long K = m.nlayers;
  const long long CK = m.ncells * K, EK = m.nedges * K;
  NvtxRange range("tendencies");
  if (p.linear) {
    // The linear passes read neighbouring h and vn of the stage input
    // directly, so an in-place (LSRK) stage first forms the tendency and
    // then updates the state.
    StageArgsT<T> ls = s;
    const bool in_place = s.ep.mode == EPI_LSRK;
    if (in_place)
      ls.ep.mode = EPI_LSRK_TEND;
    if (p.do_vn) {
      Scope sc("k_lin_edge", st);
      if (m.ne == 8)
        k_lin_edge<8, T><<<nblocks(EK), TPB, 0, st>>>(m, p, ls);
      else
        k_lin_edge<10, T><<<nblocks(EK), TPB, 0, st>>>(m, p, ls);
    }
    if (p.do_h) {
      Scope sc("k_lin_cell", st);
      k_lin_cell<T><<<nblocks(CK), TPB, 0, st>>>(m, p, ls);
    }
    if constexpr (std::is_same<T, double>::value) {
      if (in_place && p.do_vn) {
        Scope sc("k_axpby", st);
        k_axpby<<<nblocks(EK), TPB, 0, st>>>(s.fvn.out, s.fvn.tend, nullptr,
                                             s.ep.dtb, 0.0, EK, 1);
      }
      if (in_place && p.do_h) {
        Scope sc("k_axpby", st);
        k_axpby<<<nblocks(CK), TPB, 0, st>>>(s.fh.out, s.fh.tend, nullptr,
                                             s.ep.dtb, 0.0, CK, 1);
      }
    }
    return;
  }
  launch_aux_t<T>(m, p, a, s.h, s.vn, s.tr, st, fk);
  const bool edge = p.do_vn, cell = p.do_h || p.ntracers > 0;
  auto run_edge = [&](cudaStream_t q) {
    NvtxRange r("vn_tendency");
    Scope sc("k_edge_final", q);
    launch_edge_final<T>(m, p, a, s, q);
  };
  auto run_cell = [&](cudaStream_t q) {
    NvtxRange r("h_tendency+tr_tendency");
    Scope sc("k_cell_final", q);
    launch_cell_final<T>(m, p, a, s, q);
  };
  // The final passes are independent unless the stage updates the state in
  // place (LSRK): there the edge pass reads h, which the cell pass rewrites,
  // so the edge pass goes first.
  if (edge && cell && s.ep.mode != EPI_LSRK && small_model<T>(m, p, a)) {
    if constexpr (std::is_same<T, double>::value) {
      NvtxRange r("vn_tendency+h_tendency+tr_tendency");
      Scope sc("k_final", st);
      const unsigned nb = nblocks(EK, HTPB);
      if (m.ne == 8)
        k_final<8><<<nb + nblocks(CK, HTPB), HTPB, 0, st>>>(m, p, a, s, nb);
      else
        k_final<10><<<nb + nblocks(CK, HTPB), HTPB, 0, st>>>(m, p, a, s, nb);
    }
  } else if (edge && cell)
    fork_join(s.ep.mode == EPI_LSRK || g_profile ? nullptr : fk, st, run_edge,
              run_cell);
  else if (edge)
    run_edge(st);
  else if (cell)
    run_cell(st);
}

} // namespace

void launch_tendency(const MeshView &m, const ModelView &p, const AuxView &a,
                     const StageArgs &s, cudaStream_t st, const Fork *fk) {
  launch_tendency_t<double>(m, p, a, s, st, fk);
}

void launch_tendency_dual(const MeshView &m, const ModelView &p,
                          const AuxViewT<Dual> &a, const StageArgsT<Dual> &s,
                          cudaStream_t st) {
  launch_tendency_t<Dual>(m, p, a, s, st, nullptr);
}

void launch_aux(const MeshView &m, const ModelView &p, const AuxView &a,
                const double *h, const double *vn, const double *tr,
                cudaStream_t st, const Fork *fk) {
  launch_aux_t<double>(m, p, a, h, vn, tr, st, fk);
}

void launch_pv_sum(const MeshView &m, const AuxView &a, cudaStream_t st) {
  const long long n = (long long)m.nedges * m.nlayers;
  if (m.ne == 8)
    k_pv_sum<8><<<nblocks(n, HTPB), HTPB, 0, st>>>(m, a);
  else
    k_pv_sum<10><<<nblocks(n, HTPB), HTPB, 0, st>>>(m, a);
  ++g_launches;
}

void launch_field_tendency(const MeshView &m, const ModelView &p,
                           const AuxView &a, int field, const double *h,
                           const double *vn, double *tend, int mode,
                           cudaStream_t st) {
  const long long K = m.nlayers, CK = m.ncells * K, EK = m.nedges * K;
  StageArgs s{};
  s.h = h;
  s.vn = vn;
  s.ep.mode = mode;
  ModelView q = p;
  if (p.linear) { // the linear terms read h and vn themselves
    if (field == 0) {
      s.fh.tend = tend;
      Scope sc("k_lin_cell", st);
      k_lin_cell<double><<<nblocks(CK), TPB, 0, st>>>(m, q, s);
    } else {
      s.fvn.tend = tend;
      Scope sc("k_lin_edge", st);
      if (m.ne == 8)
        k_lin_edge<8, double><<<nblocks(EK), TPB, 0, st>>>(m, q, s);
      else
        k_lin_edge<10, double><<<nblocks(EK), TPB, 0, st>>>(m, q, s);
    }
    return;
  }
  {
    Scope sc("k_field_flux", st);
    if (field == 1)
      k_field_flux<true><<<nblocks(EK), TPB, 0, st>>>(m, a, vn);
    else
      k_field_flux<false><<<nblocks(EK), TPB, 0, st>>>(m, a, vn);
  }
  if (field == 1) {
    s.fvn.tend = tend;
    NvtxRange r("vn_tendency");
    Scope sc("k_edge_final", st);
    launch_edge_final<double>(m, q, a, s, st);
    return;
  }
  // the cell pass writes h when do_h is set and the tracers when ntracers
  // > 0: one of the two per call
  q.do_h = field == 0;
  if (field == 0) {
    q.ntracers = 0;
    s.fh.tend = tend;
  } else {
    s.ftr.tend = tend;
  }
  NvtxRange r(field == 0 ? "h_tendency" : "tr_tendency");
  Scope sc("k_cell_final", st);
  launch_cell_final<double>(m, q, a, s, st);
}

int fork_create(Fork &f) {
  cudaError_t err = cudaStreamCreateWithFlags(&f.side, cudaStreamNonBlocking);
  if (err == cudaSuccess)
    err = cudaEventCreateWithFlags(&f.go, cudaEventDisableTiming);
  if (err == cudaSuccess)
    err = cudaEventCreateWithFlags(&f.done, cudaEventDisableTiming);
  if (err != cudaSuccess) {
    fork_destroy(f);
    return cuda_fail(err, "fork stream");
  }
  return SWG_OK;
}

void fork_destroy(Fork &f) {
  if (f.go)
    cudaEventDestroy(f.go);
  if (f.done)
    cudaEventDestroy(f.done);
  if (f.side)
    cudaStreamDestroy(f.side);
  f = Fork{};
}

void launch_axpby(double *y, const double *x, const double *z, double alpha,
                  double beta, long long n, int kind, cudaStream_t st) {
  if (n <= 0)
    return;
  k_axpby<<<nblocks(n), TPB, 0, st>>>(y, x, z, alpha, beta, n, kind);
  ++g_launches;
}

int reduce_diag(int which, const MeshView &m, const ModelView &p,
                const double *h, const double *vn, double *partials,
                int npart, double *out, cudaStream_t st) {
  if (which == 0)
    k_diag<0><<<npart, TPB, 0, st>>>(m, p, h, vn, partials);
  else if (which == 1)
    k_diag<1><<<npart, TPB, 0, st>>>(m, p, h, vn, partials);
  else
    k_diag<2><<<npart, TPB, 0, st>>>(m, p, h, vn, partials);
  ++g_launches;
  std::vector<double> hp(npart);
  cudaError_t err = cudaMemcpyAsync(hp.data(), partials, npart * sizeof(double),
                                    cudaMemcpyDeviceToHost, st);
  if (err == cudaSuccess)
    err = cudaStreamSynchronize(st);
  if (err != cudaSuccess)
    return cuda_fail(err, "diagnostic reduction");
  double s = 0.0;
  for (double x : hp)
    s += x;
  *out = s;
  return SWG_OK;
}

} // namespace swg
