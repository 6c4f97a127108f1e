// Mixed-precision instantiation of the transport kernel (FP32 walk, scatter,
// peel and Stokes; FP64 position, radial quadratic, peel escape tau and the
// per-event table lookups).
#include "hc3d_transport.cuh"

namespace hc3d {

cudaError_t launch_transport_mixed(const DevModel& m, const DevTallies& t, const TallyDims& d, const RunArgs& a,
                                   const LaunchCfg& cfg) {
  dev::k_transport<float><<<cfg.blocks, cfg.threads, m.dust_smem, cfg.stream>>>(m, t, d, a);
  return cudaGetLastError();
}

cudaError_t launch_transport_batch_mixed(const BatchItem* items, const int64_t* first, int n, unsigned long long* work,
                                         int64_t total, const LaunchCfg& cfg) {
  dev::k_transport_batch<float><<<cfg.blocks, cfg.threads, 0, cfg.stream>>>(items, first, n, work, total);
  return cudaGetLastError();
}

const void* transport_batch_fn_mixed() { return (const void*)dev::k_transport_batch<float>; }

}  // namespace hc3d

namespace hc3d {

// k_tail's draw tables take static shared memory: dust tables that no longer
// fit beside them (48 KB a block) are read from global memory
static DevModel tail_model_mixed(const DevModel& m) {
  DevModel q = m;
  if (m.dust_smem + 4 * (int)(sizeof(dev::DrawTable<float>) + sizeof(dev::Ahead<float>)) + 256 > 48 * 1024) q.dust_smem = 0;
  return q;
}

cudaError_t launch_wave_transport_mixed(const DevModel& m, const DevTallies& t, const TallyDims& d, const RunArgs& a,
                                        const WaveBufs& w, int q, int E, const LaunchCfg& cfg) {
  dev::k_wave<float, true, true><<<cfg.blocks, cfg.threads, m.dust_smem, cfg.stream>>>(
      m, t, d, a, static_cast<dev::Slot<float>*>(w.pool), static_cast<dev::PeelRec<float>*>(w.queue[q]), w.qcount[q], E,
      w.alive[q], w.live[q]);
  return cudaGetLastError();
}

cudaError_t launch_wave_tail_mixed(const DevModel& m, const DevTallies& t, const TallyDims& d, const RunArgs& a,
                                   const WaveBufs& w, int q, int E, const LaunchCfg& cfg) {
  const DevModel tm = tail_model_mixed(m);
  dev::k_tail<float, true, true><<<cfg.blocks, 128, tm.dust_smem, cfg.stream>>>(
      tm, t, d, a, static_cast<dev::Slot<float>*>(w.pool), w.alive[1 - q], w.live[1 - q], w.next_live,
      static_cast<dev::PeelRec<float>*>(w.queue[q]), w.qcount[q], E, w.alive[q], w.live[q]);
  return cudaGetLastError();
}

template <bool kFused>
static cudaError_t launch_packets_as(const DevModel& m, const DevTallies& t, const TallyDims& d, const RunArgs& a,
                                 const TailBufs& b, const LaunchCfg& cfg, int tail_blocks) {
  auto* pool = static_cast<dev::Slot<float>*>(b.pool);
  dev::k_wave<float, false, kFused><<<cfg.blocks, cfg.threads, m.dust_smem, cfg.stream>>>(m, t, d, a, pool, nullptr, nullptr, 0,
                                                                             b.count, nullptr);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const DevModel tm = tail_model_mixed(m);
  dev::k_tail<float, false, kFused><<<tail_blocks, 128, tm.dust_smem, cfg.stream>>>(tm, t, d, a, pool, b.count, nullptr,
                                                                       b.count + 1, nullptr, nullptr, 0, nullptr,
                                                                       nullptr);
  return cudaGetLastError();
}

cudaError_t launch_packets_mixed(const DevModel& m, const DevTallies& t, const TallyDims& d, const RunArgs& a,
                                 const TailBufs& b, const LaunchCfg& cfg, int tail_blocks, bool fused) {
  return fused ? launch_packets_as<true>(m, t, d, a, b, cfg, tail_blocks)
               : launch_packets_as<false>(m, t, d, a, b, cfg, tail_blocks);
}

const void* packets_fn_mixed() { return (const void*)dev::k_wave<float, false, false>; }
const void* tail_fn_mixed(bool peel) {
  return peel ? (const void*)dev::k_tail<float, true, true> : (const void*)dev::k_tail<float, false, false>;
}
int tail_smem_mixed(const DevModel& m) { return tail_model_mixed(m).dust_smem; }

// the block shapes of k_peel_mixed: (threads, blocks per SM at launch bounds)
constexpr int kPeelShapes[kPeelVariants][2] = {{128, 5}, {192, 3}};

cudaError_t launch_wave_peel_mixed(const DevModel& m, const DevTallies& t, const TallyDims& d, const RunArgs& a,
                                   const WaveBufs& w, int q, const LaunchCfg& cfg) {
  const auto* qu = static_cast<const dev::PeelRec<float>*>(w.queue[q]);
  switch (cfg.variant) {
    case 1:
      dev::k_peel_mixed<float, 192, 3><<<cfg.blocks, 192, a.npeel * sizeof(dev::PeelDir), cfg.stream>>>(m, t, d, a, qu, w.qcount[q], w.next_ray[q]);
      break;
    default:
      dev::k_peel_mixed<float, 128, 5><<<cfg.blocks, 128, a.npeel * sizeof(dev::PeelDir), cfg.stream>>>(m, t, d, a, qu, w.qcount[q], w.next_ray[q]);
  }
  return cudaGetLastError();
}

int peel_threads_mixed(int variant) { return kPeelShapes[variant < 0 || variant >= kPeelVariants ? 0 : variant][0]; }

size_t slot_bytes_mixed() { return sizeof(dev::Slot<float>); }
size_t rec_bytes_mixed() { return sizeof(dev::PeelRec<float>); }
const void* wave_fn_mixed() { return (const void*)dev::k_wave<float, true, true>; }
const void* peel_fn_mixed(int variant) {
  switch (variant) {
    case 1: return (const void*)dev::k_peel_mixed<float, 192, 3>;
    default: return (const void*)dev::k_peel_mixed<float, 128, 5>;
  }
}

}  // namespace hc3d
