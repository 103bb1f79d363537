// Launchers for one (lattice, storage) pair; included once per inst_*.cu so
// that the kernel instantiations compile in parallel.
#pragma once

#include "engine_internal.h"
#include "kernels.cuh"

namespace lbmc {

// Shared memory of the pipelined kernel's stages, per block (at least two
// stages of Q rows): with FP32 rows of 256 nodes, two stages, seven blocks
// per SM.
constexpr long long PIPE_STAGE_BUDGET = 32 * 1024;

// The chip this is written for: a slice of it (fewer SMs) only shifts where
// the last wave begins.
constexpr int B200_SMS = 148;
// Dynamic shared memory of a resident block at most: two buffers of 1024
// D2Q9 nodes in FP64.
constexpr int RESIDENT_SMEM = 2 * 9 * RESIDENT_MAX_THREADS * 8;

template <class L, class S>
struct Launchers {
  using C = typename Storage<S>::C;

  static StepArgs<C> make_args(const DeviceState &d, long long t, bool store, int first, int planes, bool keep,
                               int block_planes = 1, bool flat = false) {
    StepArgs<C> a;
    a.f = d.f;
    a.pitch = d.pitch;
    a.cls = d.cls;
    a.B = static_cast<const C *>(d.B);
    for (int k = 0; k < 3; k++) {
      a.force[k] = static_cast<const C *>(d.force[k]);
      a.force_u[k] = (C)d.force_u[k];
      a.u[k] = static_cast<C *>(d.u[k]);
      a.L[k] = d.L[k];
      a.s[k] = d.aa ? (int)((t & 1) % d.L[k]) : (int)(t % d.L[k]);
    }
    a.aa = d.aa;
    a.tiled = d.tiled;
    a.odd = (int)(t & 1);
    a.rho = static_cast<C *>(d.rho);
    a.sf_buf = static_cast<const C *>(d.sf_buf);
    a.sf_index = d.sf_index;
    a.diag_partials = d.partials;
    a.diag_flag = d.flag;
    a.n = (int)d.n;
    a.tau = (C)d.tau;
    a.omega = (C)(1.0 / d.tau);
    // MRT rates pre-divided by the moment norms D_k = sum_i M_ki^2.
    for (int k = 0; k < 15; k++) a.s_mrt[k] = k < L::Q ? (C)(d.s_mrt[k] / (double)L::mnorm(k)) : C(0);
    a.c_smag = (C)d.c_smag;
    a.scale = (C)d.scale;
    a.inv_scale = (C)(1.0 / d.scale);
    a.compat = d.compat;
    a.store = store ? 1 : 0;
    a.error_flag = d.error_flag;
    a.timeout_cycles = d.timeout_cycles;
    a.rows = (long long)d.L[1] * d.L[2];
    a.stages = d.stages;
    a.table = d.table_dev;
    a.closure = static_cast<const MlpStep *>(d.closure);
    a.mlp = d.closure_consts;
    // The last blocks, as many as one wave of the chip holds, let the next
    // step come up.
    const long long plane_nodes = d.n / plane_count(d);
    a.first_node = (int)(first * plane_nodes);
    a.span = (int)(planes * plane_nodes);
    if (flat) {
      a.release_row = (int)(((long long)a.span + DIRECT_BLOCK - 1) / DIRECT_BLOCK - wave(d));
    } else {
      const dim3 g = grid_dim(d, (planes + block_planes - 1) / block_planes);
      a.release_row = (int)((long long)g.y * g.z - (wave(d) + g.x - 1) / g.x);
    }
    a.first_plane = first;
    a.end_plane = (first + planes - 1) % plane_count(d) + 1;
    a.keep = keep ? 1 : 0;
    a.sr_seed = sr_step_seed(t);
    return a;
  }

  // Blocks of the direct kernel that the chip holds at a time.
  static long long wave(const DeviceState &d) {
    return (long long)B200_SMS * (d.col == COL_BGK_MLP1   ? direct_min_blocks<S, COL_BGK_MLP1>()
                                  : d.col == COL_BGK_MLP  ? direct_min_blocks<S, COL_BGK_MLP>()
                                  : d.col == COL_BGK_SMAG ? direct_min_blocks<S, COL_BGK_SMAG>()
                                                          : direct_min_blocks<S, COL_BGK>());
  }

  // Whether a block of the direct kernel may take two planes one after the
  // other: that halves the blocks, whose start-up (dispatch, parameters) costs
  // the steps that HBM does not hold back.  Tiled AA, us a step with one and
  // two planes: BF16 Smagorinsky 256^3 236 and 230, FP16 with stochastic rounding
  // 250 and 247, D2Q9 FP32 4096x2048 102 and 89; FP32 D3Q15 256^3 254 and 258.
  template <int COL>
  static constexpr bool two_planes() {
    return (sizeof(S) == 2 || L::DIM == 2) && !learned_closure(COL);
  }
  // ... and where it does: the coarser last wave costs more than the start-up
  // (64^3 6.5 -> 8.1 us, FP16 192^3 102 -> 105) unless another slab of a sweep
  // fills it, or in D2Q9 from 16 waves on (2048x2048 FP16 48.3 -> 47.1).
  static int planes_per_block(const DeviceState &d, int planes, bool swept, bool diag) {
    const bool can = (sizeof(S) == 2 || L::DIM == 2) && !learned_closure(d.col);
    if (!can || !d.tiled || diag || planes < 2) return 1;
    const dim3 g = grid_dim(d, planes);
    return swept || (L::DIM == 2 && (long long)g.x * g.y * g.z >= 16 * wave(d)) ? 2 : 1;
  }

  // One block row per (y, z); blocks of up to DIRECT_BLOCK threads along x.
  static dim3 block_dim(const DeviceState &d) {
    int bx = (d.L[0] + 31) / 32 * 32;
    return dim3(bx < DIRECT_BLOCK ? bx : DIRECT_BLOCK, 1, 1);
  }
  static dim3 grid_dim(const DeviceState &d, int planes) {
    const int bx = (int)block_dim(d).x;
    const unsigned nx = (unsigned)((d.L[0] + bx - 1) / bx);
    return d.dim == 3 ? dim3(nx, (unsigned)d.L[1], (unsigned)planes) : dim3(nx, (unsigned)planes, 1);
  }
  static dim3 grid_dim(const DeviceState &d) { return grid_dim(d, plane_count(d)); }
  static long long blocks(const DeviceState &d) {
    const dim3 g = grid_dim(d);
    return (long long)g.x * g.y * g.z;
  }

  // Pipelined (bulk-copy) launch geometry: stages of Q rows in shared memory.
  static size_t stage_bytes(const DeviceState &d) { return (size_t)L::Q * d.L[0] * sizeof(S); }
  static bool pipelined_eligible(const DeviceState &d) {
    return d.pipeline && (d.L[0] * sizeof(S)) % 16 == 0 && 2 * stage_bytes(d) <= 200 * 1024;
  }
  static int pipe_stages(const DeviceState &d) {
    long long st = PIPE_STAGE_BUDGET / (long long)stage_bytes(d);
    if (st < 2) st = 2;
    if (st > PIPE_MAX_STAGES) st = PIPE_MAX_STAGES;
    return (int)st;
  }
  // One producer warp plus up to pipe_consumers<S>() / 32 consumer warps.
  static int pipe_threads(const DeviceState &d) {
    int bx = (d.L[0] + 31) / 32 * 32;
    return 32 + (bx < pipe_consumers<S>() ? bx : pipe_consumers<S>());
  }

  template <int COL, bool FORCE, bool BLEND, bool DIAG>
  static cudaError_t launch(const StepArgs<C> &a, const DeviceState &d, int planes, int block_planes, cudaStream_t st) {
    // The learned closure evaluates its network warp-wide, which the direct
    // kernel's converged warps allow: it never runs in the pipelined kernel.
    if constexpr (!learned_closure(COL)) {
      if (d.use_pipeline) {
        auto kern = step_pipelined_kernel<L, S, COL, FORCE, BLEND, DIAG>;
        const size_t smem = (size_t)d.stages * stage_bytes(d);
        static thread_local size_t configured = 0;  // per instantiation
        if (configured < smem) {
          cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
          if (e != cudaSuccess) return e;
          configured = smem;
        }
        kern<<<(unsigned)d.pipe_grid, pipe_threads(d), smem, st>>>(a);
        return cudaSuccess;
      }
    }
    auto run = [&](auto kern) {
      return launch_chained(kern, grid_dim(d, (planes + block_planes - 1) / block_planes), block_dim(d), st, a);
    };
    if (!d.aa) return run(step_kernel<L, S, COL, FORCE, BLEND, DIAG, STREAM_SHIFT>);
    if constexpr (!DIAG && two_planes<COL>())
      if (block_planes == 2)
        return a.odd ? run(step_kernel<L, S, COL, FORCE, BLEND, DIAG, STREAM_AAT_ODD, 2>)
                     : run(step_kernel<L, S, COL, FORCE, BLEND, DIAG, STREAM_AAT_EVEN, 2>);
    if (d.tiled)
      return a.odd ? run(step_kernel<L, S, COL, FORCE, BLEND, DIAG, STREAM_AAT_ODD>)
                   : run(step_kernel<L, S, COL, FORCE, BLEND, DIAG, STREAM_AAT_EVEN>);
    if (a.odd) return run(step_kernel<L, S, COL, FORCE, BLEND, DIAG, STREAM_AA_ODD>);
    auto even = step_kernel<L, S, COL, FORCE, BLEND, DIAG, STREAM_AA_EVEN>;
    if constexpr (flat_step<COL, DIAG, STREAM_AA_EVEN>())
      return launch_chained(even, dim3((unsigned)((a.span + DIRECT_BLOCK - 1) / DIRECT_BLOCK)), dim3(DIRECT_BLOCK), st, a);
    return run(even);
  }

  template <int COL, bool BLEND>
  static cudaError_t launch_fd(const StepArgs<C> &a, const DeviceState &d, bool diag, int planes, int block_planes,
                               cudaStream_t st) {
    if (d.forcing) {
      if (diag) return launch<COL, true, BLEND, true>(a, d, planes, block_planes, st);
      return launch<COL, true, BLEND, false>(a, d, planes, block_planes, st);
    }
    if (diag) return launch<COL, false, BLEND, true>(a, d, planes, block_planes, st);
    return launch<COL, false, BLEND, false>(a, d, planes, block_planes, st);
  }

  template <int COL>
  static cudaError_t launch_col(const StepArgs<C> &a, const DeviceState &d, bool diag, int planes, int block_planes,
                               cudaStream_t st) {
    if (d.blend) return launch_fd<COL, true>(a, d, diag, planes, block_planes, st);
    return launch_fd<COL, false>(a, d, diag, planes, block_planes, st);
  }

  static cudaError_t step(const DeviceState &d, long long t, bool store, bool diag, int first, int planes, bool swept,
                          bool keep, cudaStream_t st) {
    const int block_planes = planes_per_block(d, planes, swept, diag);
    const bool flat = d.aa && !d.tiled && !(t & 1) && !diag && !learned_closure(d.col);  // flat_step()
    const StepArgs<C> a = make_args(d, t, store, first, planes, keep, block_planes, flat);
    if (d.n_sf > 0) {
      const int nb = (d.n_sf + 127) / 128;
      sf_gather_kernel<L, S><<<nb, 128, 0, st>>>(a, d.sf_nodes, d.sf_face, d.n_sf,
                                                  static_cast<C *>(d.sf_buf));
    }
    cudaError_t e;
    switch (d.col) {
      case COL_BGK: e = launch_col<COL_BGK>(a, d, diag, planes, block_planes, st); break;
      case COL_BGK_SMAG: e = launch_col<COL_BGK_SMAG>(a, d, diag, planes, block_planes, st); break;
      case COL_MRT_NC: e = launch_col<COL_MRT_NC>(a, d, diag, planes, block_planes, st); break;
      case COL_BGK_MLP: e = launch_col<COL_BGK_MLP>(a, d, diag, planes, block_planes, st); break;
      case COL_BGK_MLP1: e = launch_col<COL_BGK_MLP1>(a, d, diag, planes, block_planes, st); break;
      default: e = launch_col<COL_MRT>(a, d, diag, planes, block_planes, st); break;
    }
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
  }

  template <int COL, bool FORCE, bool BLEND>
  static auto resident_kernel() {
    return step_resident_kernel<L, S, COL, FORCE, BLEND>;
  }
  template <class F>
  static cudaError_t with_resident_kernel(const DeviceState &d, F &&f) {
    auto fb = [&](auto col) {
      constexpr int COL = decltype(col)::value;
      if (d.forcing) return d.blend ? f(resident_kernel<COL, true, true>()) : f(resident_kernel<COL, true, false>());
      return d.blend ? f(resident_kernel<COL, false, true>()) : f(resident_kernel<COL, false, false>());
    };
    switch (d.col) {
      case COL_BGK: return fb(std::integral_constant<int, COL_BGK>{});
      case COL_BGK_SMAG: return fb(std::integral_constant<int, COL_BGK_SMAG>{});
      case COL_MRT_NC: return fb(std::integral_constant<int, COL_MRT_NC>{});
      default: return fb(std::integral_constant<int, COL_MRT>{});
    }
  }
  static cudaLaunchConfig_t resident_config(const DeviceState &d, cudaLaunchAttribute &attr, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)d.resident_cluster);
    cfg.blockDim = dim3((unsigned)((d.resident_per + 31) / 32 * 32));
    cfg.dynamicSmemBytes = 2 * (size_t)L::Q * d.resident_per * sizeof(S);
    cfg.stream = st;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)d.resident_cluster;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cfg;
  }
  // Shared memory and cluster size beyond the portable limits, allowed per
  // kernel (cheap, and the same value every time for a kernel and a size).
  static cudaError_t allow_resident(const void *kern, const cudaLaunchConfig_t &cfg) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, RESIDENT_SMEM);
    return e;
  }
  static cudaError_t resident(const DeviceState &d, long long t, int steps, cudaStream_t st) {
    if constexpr (L::DIM == 2) {
      const StepArgs<C> a = make_args(d, t, false, 0, plane_count(d), false), end = make_args(d, t + steps, false, 0,
                                                                                             plane_count(d), false);
      ResidentRun run = {d.resident_per, steps, t, {end.s[0], end.s[1], end.s[2]}, end.odd};
      return with_resident_kernel(d, [&](auto kern) {
        cudaLaunchAttribute attr = {};
        const cudaLaunchConfig_t cfg = resident_config(d, attr, st);
        const cudaError_t e = allow_resident((const void *)kern, cfg);
        return e == cudaSuccess ? cudaLaunchKernelEx(&cfg, kern, a, run) : e;
      });
    } else {
      return cudaErrorNotSupported;
    }
  }
  // Whether one cluster can hold the domain: a node per thread, at least 256
  // threads a block (fewer, fuller blocks below 4096 nodes), 16 blocks at most.
  static cudaError_t plan_resident(DeviceState &d) {
    d.resident_cluster = 0;
    if constexpr (L::DIM == 2) {
      if (!d.auto_kernel || d.n > RESIDENT_MAX_CLUSTER * RESIDENT_MAX_THREADS) return cudaSuccess;
      int c = 1;
      while (c < RESIDENT_MAX_CLUSTER && 256LL * c < d.n) c *= 2;
      d.resident_cluster = c;
      d.resident_per = (int)((d.n + c - 1) / c);
      return with_resident_kernel(d, [&](auto kern) {
        cudaLaunchAttribute attr = {};
        const cudaLaunchConfig_t cfg = resident_config(d, attr, nullptr);
        int clusters = 0;
        cudaError_t e = allow_resident((const void *)kern, cfg);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg);
        if (e != cudaSuccess || clusters < 1) {  // no room for it: step by step
          cudaGetLastError();
          d.resident_cluster = 0;
        }
        return cudaSuccess;
      });
    }
    return cudaSuccess;
  }

  // Chooses the kernel and its launch geometry for a handle (called once by
  // lbmc_init after the device state is filled in).
  static cudaError_t plan(DeviceState &d) {
    // The direct-load kernel is the default; the bulk-copy pipeline runs when
    // asked for (lbmc_config.kernel) and the rows allow it.
    d.use_pipeline = (d.pipeline == 2 && !d.aa && pipelined_eligible(d)) ? 1 : 0;
    if (!d.use_pipeline) {
      d.nblocks = blocks(d);
      return cudaSuccess;
    }
    d.stages = pipe_stages(d);
    const size_t smem = (size_t)d.stages * stage_bytes(d);
    // Occupancy of the heaviest instantiation the handle can launch.
    int per_sm = 0;
    cudaError_t e;
    auto probe = [&](auto kern) {
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, pipe_threads(d), smem);
    };
    switch (d.col) {
      case COL_BGK: probe(step_pipelined_kernel<L, S, COL_BGK, true, true, true>); break;
      case COL_BGK_SMAG: probe(step_pipelined_kernel<L, S, COL_BGK_SMAG, true, true, true>); break;
      case COL_MRT_NC: probe(step_pipelined_kernel<L, S, COL_MRT_NC, true, true, true>); break;
      default: probe(step_pipelined_kernel<L, S, COL_MRT, true, true, true>); break;
    }
    if (e != cudaSuccess) return e;
    if (per_sm < 1) {
      d.use_pipeline = 0;
      d.nblocks = blocks(d);
      return cudaSuccess;
    }
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long rows = (long long)d.L[1] * d.L[2];
    long long grid = (long long)sms * per_sm;
    if (grid > rows) grid = rows;
    d.pipe_grid = grid;
    d.nblocks = grid;
    return cudaSuccess;
  }

  static cudaError_t fetch_population(const DeviceState &d, long long t, int i, double *out,
                                      cudaStream_t st) {
    const StepArgs<C> a = make_args(d, t, false, 0, plane_count(d), false);
    fetch_population_kernel<L, S><<<grid_dim(d), block_dim(d), 0, st>>>(a, i, out);
    return cudaGetLastError();
  }

  static cudaError_t upload_population(const DeviceState &d, long long t, int i, const double *in,
                                       cudaStream_t st) {
    const StepArgs<C> a = make_args(d, t, false, 0, plane_count(d), false);
    upload_population_kernel<L, S><<<grid_dim(d), block_dim(d), 0, st>>>(a, i, in);
    return cudaGetLastError();
  }

  static const LatticeStorageOps *ops() {
    static const LatticeStorageOps o = {(int)sizeof(C), (int)sizeof(S), &step, &resident, &fetch_population,
                                        &upload_population, &plan, &plan_resident};
    return &o;
  }
};

}  // namespace lbmc

#define LBMC_DEFINE_OPS(NAME, LAT, STORE) \
  namespace lbmc {                        \
  const LatticeStorageOps *NAME() { return Launchers<LAT, STORE>::ops(); } \
  }
