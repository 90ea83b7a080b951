// hw_kernels.cuh -- the persistent evolve kernel and the single-RHS kernel of one
// slice size M (instantiated once per M in hw_inst_<M>.cu).
#pragma once

#include "hw_breaking.cuh"
#include "hw_rhs_fast.cuh"
#include "hw_rhs_gen.cuh"
#include "hw_kernels.h"
#include "hw_stepper.cuh"
#include "hw_output.cuh"

// resident CTAs per SM the register allocation is sized for (slice M, M / 8 threads)
#ifndef HW_EVOLVE_MIN_BLOCKS
#define HW_EVOLVE_MIN_BLOCKS(M) (4096 / (M))
#endif

namespace hwdev {

// One member's work of a launch: mode 0 advances it through its output samples up to
// its stop index (clipping steps at each sample like the reference), mode 1 takes one
// evolve_apply to sd.t1.  The member's descriptor is in shared memory (sd).
template <int M>
__device__ __forceinline__ void evolve_member(DevMember* mems, int mi, int mode, DevMember& sd, Scratch<M>& sc,
                                              double2* smem_buf, int C, int rank) {
  if (threadIdx.x == 0) {
    sd = mems[mi];
    sc.bufs.y = sd.y;
    sc.bufs.yn = sd.ynew;
    for (int i = 0; i < 7; ++i) sc.bufs.k[i] = sd.kb[i];
    sc.full = 0;
    sc.idle = -1;
  }
  // a cluster barrier, not only the CTA's: the RHS's first phase writes into the
  // partner CTA's shared memory, which must be running
  member_sync(C);
  Ctx<M> X = make_ctx<M>(sd, smem_buf, sc, rank);
  spread_unmoved(X);
  StepState S{sd.t, sd.h, sd.status, sd.k1_valid, 0, 0, 0};
  int iout = sd.i_out;
  if (S.status == kOk) {
    if (mode == 1) {
      evolve_apply<M>(X, S, sd.t1);
    } else {
      while (iout < sd.i_stop && S.status == kOk) {
        const double ti = sd.tt[iout];
        while (S.t < ti && S.status == kOk) {
          evolve_apply<M>(X, S, ti);
          if (S.rhs >= sd.rhs_budget && S.status == kOk) S.status = kBudget;   // bounded launch
        }
        if (S.status == kOk) {
          if (sd.ngauge > 0 || sd.fields) output_stage<M>(X, S, iout);
          ++iout;
        }
      }
    }
  }
  member_sync(C);
  if (rank == 0 && threadIdx.x == 0) {
    DevMember& g = mems[mi];
    g.t = S.t;
    g.h = S.h;
    g.status = S.status;
    g.k1_valid = S.k1_valid;
    g.i_out = iout;
    g.rhs_calls += S.rhs;
    g.accepted += S.acc;
    g.rejected += S.rej;
    g.y = sc.bufs.y;
    g.ynew = sc.bufs.yn;
    for (int i = 0; i < 7; ++i) g.kb[i] = sc.bufs.k[i];
  }
}

// The evolve kernel, persistent over a work queue: a grid of resident clusters (one
// cluster of C CTAs per member at a time) whose leaders take the next entry of the
// class's member list (ordered longest-first) from the queue counter until the list
// is used up, so no cluster waits for a member another cluster is running and the
// number of members in flight -- and their stage vectors in L2 -- is the grid's.
// With queue == nullptr cluster b runs entry b of the list (one cluster per member).
template <int M>
__global__ void __launch_bounds__(M / kPts, HW_EVOLVE_MIN_BLOCKS(M))
    k_evolve(DevMember* mems, const int* list, int mode, int* queue, int nlist) {
  extern __shared__ double2 smem_buf[];
  __shared__ DevMember sd;
  __shared__ Scratch<M> sc;
  __shared__ int s_next;
  cg::cluster_group cl = cg::this_cluster();
  const int C = int(cl.num_blocks());
  const int rank = int(cl.block_rank());
  if (!queue) {
    evolve_member<M>(mems, list[blockIdx.x / C], mode, sd, sc, smem_buf, C, rank);
    return;
  }
  for (;;) {
    if (rank == 0 && threadIdx.x == 0) s_next = atomicAdd(queue, 1);
    member_sync(C);
    // every CTA reads the leader's entry before the leader can take the next one: the
    // member's work below passes through cluster barriers first
    const int w = C > 1 ? *cl.map_shared_rank(&s_next, 0) : s_next;
    if (w >= nlist) break;
    evolve_member<M>(mems, list[w], mode, sd, sc, smem_buf, C, rank);
  }
  // no CTA leaves while a peer may still read its shared memory
  member_sync(C);
}

// Single RHS evaluation of member mi: kout = f(t, zs).  With y_ref the state comes from
// there and the result goes to dy_ref, both in the reference layout (4N doubles); with
// scratch, the member's zs, kout and fields are in that array.
template <int M>
__global__ void __launch_bounds__(M / kPts, (4096 / M)) k_rhs(DevMember* mems, int mi, double t,
                                                              const double* y_ref, double* dy_ref,
                                                              double2* scratch) {
  extern __shared__ double2 smem_buf[];
  __shared__ DevMember sd;
  __shared__ Scratch<M> sc;
  cg::cluster_group cl = cg::this_cluster();
  const int C = int(cl.num_blocks());
  const int rank = int(cl.block_rank());
  if (threadIdx.x == 0) {
    sd = mems[mi];
    const int N = sd.N;
    if (scratch) {
      sd.zs = scratch;
      sd.kb[6] = scratch + 2 * N;
      for (int i = 0; i < kScratch; ++i) sd.sc[i] = scratch + size_t(4 + i) * N;
    }
    sc.stg.s = 0;
    sc.stg.sig = -1;
    sc.full = 1;
    sc.idle = -1;
  }
  __syncthreads();
  Ctx<M> X = make_ctx<M>(sd, smem_buf, sc, rank);
  const int N = sd.N;
  if (y_ref) {
    // reference layout -> this CTA's spectral slice of the stage input
    HW_FOREACH(X) {
      const int kk = X.c + (idx << sd.logC);
      sd.zs[p] = make_double2(y_ref[kk], y_ref[N + kk]);
      sd.zs[N + p] = make_double2(y_ref[2 * N + kk], y_ref[3 * N + kk]);
    }
  }
  rhs_eval<M>(X, t, sd.kb[6]);
  if (dy_ref) {
    HW_FOREACH(X) {
      const int kk = X.c + (idx << sd.logC);
      const double2 e = sd.kb[6][p], u = sd.kb[6][N + p];
      dy_ref[kk] = e.x;
      dy_ref[N + kk] = e.y;
      dy_ref[2 * N + kk] = u.x;
      dy_ref[3 * N + kk] = u.y;
    }
  }
  member_sync(C);
  if (rank == 0 && threadIdx.x == 0) mems[mi].rhs_calls += 1;
}

template <int M>
cudaError_t set_attrs() {
  const int bytes = int(slice_smem_bytes(M));
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(k_evolve<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(k_rhs<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(k_evolve<M>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_rhs<M>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

// resident clusters of C CTAs of the evolve kernel (the persistent grid's size limit)
template <int M>
int max_clusters(int C) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(C));
  cfg.blockDim = dim3(M / kPts);
  cfg.dynamicSmemBytes = slice_smem_bytes(M);
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = unsigned(C);
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, k_evolve<M>, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return n;
}

// a launch of `clusters` clusters of C CTAs
template <int M, typename... P, typename... A>
cudaError_t launch_clusters(void (*kernel)(P...), int clusters, int C, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(clusters * C));
  cfg.blockDim = dim3(M / kPts);
  cfg.dynamicSmemBytes = slice_smem_bytes(M);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = unsigned(C);
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace hwdev

#define HW_INSTANTIATE(MM)                                                                          \
  cudaError_t hw_attr_##MM() { return hwdev::set_attrs<MM>(); }                                    \
  cudaError_t hw_evolve_##MM(int mode, hwdev::DevMember* mems, const int* list, int nmem, int C,   \
                             cudaStream_t s, int* queue, int ngrid) {                               \
    return hwdev::launch_clusters<MM>(hwdev::k_evolve<MM>, queue ? ngrid : nmem, C, s, mems, list,  \
                                      mode, queue, nmem);                                           \
  }                                                                                                 \
  cudaError_t hw_rhs_##MM(hwdev::DevMember* mems, int mi, int C, double t, const double* y,         \
                          double* dy, double2* scratch, cudaStream_t s) {                           \
    return hwdev::launch_clusters<MM>(hwdev::k_rhs<MM>, 1, C, s, mems, mi, t, y, dy, scratch);      \
  }                                                                                                 \
  int hw_max_clusters_##MM(int C) { return hwdev::max_clusters<MM>(C); }
