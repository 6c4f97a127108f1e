// The mixed form's wall searches beside each other, for test_gpu_wall_search.py:
// the search of one thread (next_wall_ray) and that of a warp (next_wall_warp)
// on the same rays, and the roots that the peel-off walk finds on a cone.
#include <cstdint>

#include "hc3d_transport.cuh"

using namespace hc3d;
using namespace hc3d::dev;

struct RayIn {
  float x, y, z, ux, uy, uz;
  int ir, it, ip, own;
};
struct Found {
  int ok;       // a wall was found
  float dt;
  int iface;    // 1..6
};
struct ConeIn {
  float c2, hemi, p2, cz, uz, t;
};

namespace {

template <bool kFused>
__global__ void k_search(DevModel m, const RayIn* in, int n, Found* lone, Found* warp) {
  const int k = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (k >= n) return;  // a whole warp
  const RayIn q = in[k];
  const PathLen S{0.f, 0.f};
  Ray r;
  ray_init(r, Pos2{q.x, 0.f}, Pos2{q.y, 0.f}, Pos2{q.z, 0.f}, q.ux, q.uy, q.uz);
  float dt = 0.f;
  int win = 0, side = 0;
  const bool ok = next_wall_warp<kFused>(m, r, S, q.ir, q.it, q.ip, q.own, dt, win, side);
  if ((threadIdx.x & 31) == 0) {
    warp[k] = Found{ok, ok ? dt : 0.f, ok ? (win < 4 ? win + 1 : 5 + side) : 0};
    ray_init(r, Pos2{q.x, 0.f}, Pos2{q.y, 0.f}, Pos2{q.z, 0.f}, q.ux, q.uy, q.uz);
    float d1 = 0.f;
    int iface = 0;
    const bool ok1 = next_wall_ray<kFused>(m, r, S, q.ir, q.it, q.ip, q.own, d1, iface);
    lone[k] = Found{ok1, ok1 ? d1 : 0.f, ok1 ? iface : 0};
  }
}

__global__ void k_cone(const ConeIn* in, int n, float2* roots) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  PeelWalk w;
  w.p2 = in[k].p2;
  w.cz = in[k].cz;
  w.uz = in[k].uz;
  w.t = in[k].t;
  float r1, r2;
  w.cone_roots(make_float2(in[k].c2, in[k].hemi), false, r1, r2);
  roots[k] = make_float2(r1, r2);
}

}  // namespace

// walls: r2arr (nrg) FP64, then the FP32 pairs of DevModel::wallw (nr1 spheres, ntg cones, npg planes)
extern "C" int wall_search(int nrg, int ntg, int npg, const double* r2arr, const float2* wallw, const RayIn* in, int n,
                           int fused, Found* lone, Found* warp) {
  DevModel m{};
  m.nrg = nrg; m.ntg = ntg; m.npg = npg;
  m.nr1 = nrg - 1; m.nt1 = ntg - 1; m.np1 = npg - 1; m.nplane = m.nr1 * m.nt1;
  m.r2arr = r2arr;
  m.wallw = wallw;
  m.r2pair = wallw;
  m.conef = wallw + m.nr1;
  m.planef = wallw + m.nr1 + ntg;
  const int blocks = (n + 3) / 4;
  if (fused) k_search<true><<<blocks, 128>>>(m, in, n, lone, warp);
  else k_search<false><<<blocks, 128>>>(m, in, n, lone, warp);
  if (cudaGetLastError() != cudaSuccess) return 1;
  return cudaDeviceSynchronize() != cudaSuccess;
}

extern "C" int cone_search(const ConeIn* in, int n, float2* roots) {
  k_cone<<<(n + 127) / 128, 128>>>(in, n, roots);
  if (cudaGetLastError() != cudaSuccess) return 1;
  return cudaDeviceSynchronize() != cudaSuccess;
}
