// neighbors.cu -- neighbor-list build with fused density, and export to the
// reference layout.
#include "build_kernel.cuh"
#include "neighbors.cuh"

namespace alb {

namespace {

inline uint32_t blocks_for(uint32_t n, int block) { return (n + block - 1) / block; }

// Threads per particle of the export: eight 16-byte entries (float) fill a
// 128-byte line of the particle's row.  One thread per particle stored its
// entries 1 KB apart from its neighbors' lanes: 455 us for 306,525 particles
// with 64-entry rows, 240 us with eight (B200, whole update).  Without rows there
// is one count and one density per particle, and one thread (512,000 particles,
// eight threads 19.4 us, one 7.1).
constexpr uint32_t kExportLanes = 8;

template <class TF, uint32_t LANES>
__global__ void k_export_neighbors(Cn<TF> c, uint32_t cap, uint32_t n,
                                   const uint32_t* __restrict__ perm,
                                   const vec4<TF>* __restrict__ xs,
                                   const uint32_t* __restrict__ nbr,
                                   const uint32_t* __restrict__ ncount,
                                   const TF* __restrict__ rho_sorted, TF* __restrict__ out_nbr,
                                   uint32_t* __restrict__ out_num, TF* __restrict__ out_rho) {
  const uint32_t s = blockIdx.x * (blockDim.x / LANES) + threadIdx.x / LANES;
  const uint32_t lane = threadIdx.x % LANES;
  if (s >= n) return;
  const uint32_t i = perm[s];
  const uint32_t cnt = ncount[s];
  if (lane == 0) {
    out_num[i] = cnt;
    if (out_rho) out_rho[i] = rho_sorted[s];
  }
  if (!out_nbr) return;
  const vec3<TF> xi = xyz(xs[s]);
  // the caller's buffer may start anywhere
  const bool aligned = reinterpret_cast<uintptr_t>(out_nbr) % sizeof(vec4<TF>) == 0;
  for (uint32_t k = lane; k < cnt; k += LANES) {
    const uint32_t t = nbr[nbr_index(k, s, n)];
    const uint32_t j = perm[t];
    const vec3<TF> xj = xyz(xs[t]);
    TF* e = out_nbr + (size_t(i) * cap + k) * 4;
    const vec3<TF> d = pdisp(c, xi, xj);  // wrapped in y on a periodic update
    vec4<TF> w{d.x, d.y, d.z, TF(0)};
    if constexpr (sizeof(TF) == 4)
      w.w = __uint_as_float(j);
    else
      w.w = __longlong_as_double((long long)j);
    if (aligned) {
      *reinterpret_cast<vec4<TF>*>(e) = w;
    } else {
      e[0] = w.x;
      e[1] = w.y;
      e[2] = w.z;
      e[3] = w.w;
    }
  }
}

}  // namespace

template <class TF, class BK>
int build_neighbors_density(const Cn<TF>& c, const GridDims& g, const GridState& gs,
                            const vec4<TF>* xs, const ScanSoa<TF>& soa, const BK& bk,
                            uint32_t* nbr, uint32_t* ncount, TF* rho, TF* alpha, TF* rho_rec,
                            cudaStream_t st) {
  if (gs.n == 0) return AL_OK;
  const uint32_t blocks = blocks_for(gs.n, kBlock);
  // compile-time wrap flag: the non-periodic build carries no wrap branches
  if (alpha && c.wrap)
    k_build_neighbors<TF, BK, true, NoExtra<TF>, true><<<blocks, kBlock, 0, st>>>(
        c, g, gs.cell_start, xs, soa, gs.n, gs.n, bk, nbr, ncount, rho, alpha, rho_rec, gs.flags,
        NoExtra<TF>{}, FusedBuild{});
  else if (alpha)
    k_build_neighbors<TF, BK, true, NoExtra<TF>, false><<<blocks, kBlock, 0, st>>>(
        c, g, gs.cell_start, xs, soa, gs.n, gs.n, bk, nbr, ncount, rho, alpha, rho_rec, gs.flags,
        NoExtra<TF>{}, FusedBuild{});
  else if (c.wrap)
    k_build_neighbors<TF, BK, false, NoExtra<TF>, true><<<blocks, kBlock, 0, st>>>(
        c, g, gs.cell_start, xs, soa, gs.n, gs.n, bk, nbr, ncount, rho, alpha, rho_rec, gs.flags,
        NoExtra<TF>{}, FusedBuild{});
  else
    k_build_neighbors<TF, BK, false, NoExtra<TF>, false><<<blocks, kBlock, 0, st>>>(
        c, g, gs.cell_start, xs, soa, gs.n, gs.n, bk, nbr, ncount, rho, alpha, rho_rec, gs.flags,
        NoExtra<TF>{}, FusedBuild{});
  ALB_CUDA(cudaGetLastError());
  return AL_OK;
}

template <class TF>
int export_neighbors(const Cn<TF>& c, const GridDims& g, const GridState& gs,
                     const vec4<TF>* xs,
                     const uint32_t* nbr, const uint32_t* ncount, const TF* rho_sorted,
                     TF* particle_neighbors, uint32_t* particle_num_neighbors,
                     TF* particle_density, cudaStream_t st) {
  if (gs.n == 0) return AL_OK;
  const uint32_t lanes = particle_neighbors ? kExportLanes : 1;
  const auto kernel =
      particle_neighbors ? k_export_neighbors<TF, kExportLanes> : k_export_neighbors<TF, 1>;
  kernel<<<blocks_for(gs.n, int(kBlock / lanes)), kBlock, 0, st>>>(
      c, g.cap_nbr, gs.n, gs.perm, xs, nbr, ncount, rho_sorted, particle_neighbors,
      particle_num_neighbors, particle_density);
  ALB_CUDA(cudaGetLastError());
  return AL_OK;
}

#define ALB_INST(TF, BK)                                                                  \
  template int build_neighbors_density<TF, BK<TF>>(                                       \
      const Cn<TF>&, const GridDims&, const GridState&, const vec4<TF>*,                   \
      const ScanSoa<TF>&, const BK<TF>&, uint32_t*, uint32_t*, TF*, TF*, TF*, cudaStream_t);
ALB_INST(float, RefBoundaryKernel)
ALB_INST(double, RefBoundaryKernel)
ALB_INST(float, SortedBoundaryKernel)
ALB_INST(double, SortedBoundaryKernel)
#undef ALB_INST
template int export_neighbors<float>(const Cn<float>&, const GridDims&, const GridState&,
                                     const vec4<float>*,
                                     const uint32_t*, const uint32_t*, const float*, float*,
                                     uint32_t*, float*, cudaStream_t);
template int export_neighbors<double>(const Cn<double>&, const GridDims&, const GridState&,
                                      const vec4<double>*,
                                      const uint32_t*, const uint32_t*, const double*, double*,
                                      uint32_t*, double*, cudaStream_t);

}  // namespace alb
