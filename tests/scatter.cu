// A scattering of the mixed form by one thread and by a warp, and the draws
// around it, for test_gpu_scatter_rounding.py.
#include <cstdint>

#include "hc3d_transport.cuh"

using namespace hc3d;
using namespace hc3d::dev;

struct Event {
  float cost, sint, phi, cosp, sinp, sip, sqp, sup, svp, g, pl;
  float kapd[4], rho[4], u;  // of the species' selection
  unsigned pid;
};
struct Left {
  float cost, sint, phi, cosp, sinp, sip, sqp, sup, svp;  // the packet after the scattering
  float mu, smu, rprob;
  int species, draws;
};

namespace {

__device__ Pkt<float> packet(const Event& e) {
  Pkt<float> p;
  p.cost = e.cost; p.sint = e.sint; p.phi = e.phi; p.cosp = e.cosp; p.sinp = e.sinp;
  p.sip = e.sip; p.sqp = e.sqp; p.sup = e.sup; p.svp = e.svp;
  for (int k = 0; k < kSlots; ++k) { p.g[k] = e.g; p.pl[k] = e.pl; p.kapd[k] = e.kapd[k]; }
  return p;
}

__device__ void put(Left& o, const Pkt<float>& p, float rprob, int species, int draws) {
  o.cost = p.cost; o.sint = p.sint; o.phi = p.phi; o.cosp = p.cosp; o.sinp = p.sinp;
  o.sip = p.sip; o.sqp = p.sqp; o.sup = p.sup; o.svp = p.svp;
  o.rprob = rprob;
  o.species = species;
  o.draws = draws;
}

__global__ void k_lone(const Event* in, int n, Left* out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  Pkt<float> p = packet(in[k]);
  Rng rng, first;
  rng_init(rng, 1u, 2u, in[k].pid);
  first = rng;
  ScatTry<float> q;
  scat_draw<float>(p, in[k].g, in[k].pl, first, q);
  stokes<float>(p, (int)(in[k].pid & 3u), rng);
  put(out[k], p, q.rprob, select_species<float>(in[k].kapd, in[k].rho, in[k].u), (int)(4u * rng.c0) - rng.left);
  draw_mu<float>(rng, out[k].mu, out[k].smu);
}

__global__ void k_warp(const Event* in, int n, Left* out) {
  __shared__ DrawTable<float> draws[4];
  const int k = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (k >= n) return;  // a whole warp
  Pkt<float> p = packet(in[k]);
  WarpRng<float> rng;
  rng_init(rng, draws + (threadIdx.x >> 5), 1u, 2u, (uint64_t)in[k].pid, 0u, 0);
  ScatTry<float> q;
  scat_draw<float>(p, in[k].g, in[k].pl, rng, q);
  rng_init(rng, draws + (threadIdx.x >> 5), 1u, 2u, (uint64_t)in[k].pid, 0u, 0);
  stokes<float>(p, (int)(in[k].pid & 3u), rng);
  Rho<float> rho;
  for (int s = 0; s < kSlots; ++s) rho.v[s] = in[k].rho[s];
  const int species = select_known(p, rho, in[k].u);
  ensure(rng, 1);
  const float mu = 1.f - 2.f * rng.t->u[rng.at];
  if ((threadIdx.x & 31) == 0) {
    put(out[k], p, q.rprob, species, (int)(4u * rng.block) + rng.at);
    out[k].mu = mu;
    out[k].smu = sin_of(mu);
  }
}

}  // namespace

extern "C" int scatter(const Event* in, int n, Left* lone, Left* warp) {
  k_lone<<<(n + 127) / 128, 128>>>(in, n, lone);
  k_warp<<<(n + 3) / 4, 128>>>(in, n, warp);
  if (cudaGetLastError() != cudaSuccess) return 1;
  return cudaDeviceSynchronize() != cudaSuccess;
}
