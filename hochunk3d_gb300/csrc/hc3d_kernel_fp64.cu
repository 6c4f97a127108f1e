// All-FP64 instantiation of the transport kernel.  This translation unit is
// compiled with --fmad=false: multiplies and adds round separately, as in the
// CPU restatement, so the two can be compared packet by packet.
#include "hc3d_transport.cuh"

namespace hc3d {

cudaError_t launch_transport_fp64(const DevModel& m, const DevTallies& t, const TallyDims& d, const RunArgs& a,
                                  const LaunchCfg& cfg) {
  dev::k_transport<double><<<cfg.blocks, cfg.threads, m.dust_smem, cfg.stream>>>(m, t, d, a);
  return cudaGetLastError();
}

cudaError_t launch_transport_batch_fp64(const BatchItem* items, const int64_t* first, int n, unsigned long long* work,
                                         int64_t total, const LaunchCfg& cfg) {
  dev::k_transport_batch<double><<<cfg.blocks, cfg.threads, 0, cfg.stream>>>(items, first, n, work, total);
  return cudaGetLastError();
}

const void* transport_batch_fn_fp64() { return (const void*)dev::k_transport_batch<double>; }

}  // namespace hc3d

namespace hc3d {

// k_tail's draw tables take static shared memory: dust tables that no longer
// fit beside them (48 KB a block) are read from global memory
static DevModel tail_model_fp64(const DevModel& m) {
  DevModel q = m;
  if (m.dust_smem + 4 * (int)(sizeof(dev::DrawTable<double>) + sizeof(dev::Ahead<double>)) + 256 > 48 * 1024) q.dust_smem = 0;
  return q;
}

cudaError_t launch_wave_transport_fp64(const DevModel& m, const DevTallies& t, const TallyDims& d, const RunArgs& a,
                                        const WaveBufs& w, int q, int E, const LaunchCfg& cfg) {
  dev::k_wave<double, true, true><<<cfg.blocks, cfg.threads, m.dust_smem, cfg.stream>>>(
      m, t, d, a, static_cast<dev::Slot<double>*>(w.pool), static_cast<dev::PeelRec<double>*>(w.queue[q]), w.qcount[q], E,
      w.alive[q], w.live[q]);
  return cudaGetLastError();
}

cudaError_t launch_wave_tail_fp64(const DevModel& m, const DevTallies& t, const TallyDims& d, const RunArgs& a,
                                   const WaveBufs& w, int q, int E, const LaunchCfg& cfg) {
  const DevModel tm = tail_model_fp64(m);
  dev::k_tail<double, true, true><<<cfg.blocks, 128, tm.dust_smem, cfg.stream>>>(
      tm, t, d, a, static_cast<dev::Slot<double>*>(w.pool), w.alive[1 - q], w.live[1 - q], w.next_live,
      static_cast<dev::PeelRec<double>*>(w.queue[q]), w.qcount[q], E, w.alive[q], w.live[q]);
  return cudaGetLastError();
}

cudaError_t launch_packets_fp64(const DevModel& m, const DevTallies& t, const TallyDims& d, const RunArgs& a,
                                 const TailBufs& b, const LaunchCfg& cfg, int tail_blocks, bool) {
  auto* pool = static_cast<dev::Slot<double>*>(b.pool);
  dev::k_wave<double, false, false><<<cfg.blocks, cfg.threads, m.dust_smem, cfg.stream>>>(m, t, d, a, pool, nullptr, nullptr, 0,
                                                                             b.count, nullptr);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const DevModel tm = tail_model_fp64(m);
  dev::k_tail<double, false, false><<<tail_blocks, 128, tm.dust_smem, cfg.stream>>>(tm, t, d, a, pool, b.count, nullptr,
                                                                       b.count + 1, nullptr, nullptr, 0, nullptr,
                                                                       nullptr);
  return cudaGetLastError();
}

const void* packets_fn_fp64() { return (const void*)dev::k_wave<double, false, false>; }
const void* tail_fn_fp64(bool peel) {
  return peel ? (const void*)dev::k_tail<double, true, true> : (const void*)dev::k_tail<double, false, false>;
}
int tail_smem_fp64(const DevModel& m) { return tail_model_fp64(m).dust_smem; }

cudaError_t launch_wave_peel_fp64(const DevModel& m, const DevTallies& t, const TallyDims& d, const RunArgs& a,
                                   const WaveBufs& w, int q, const LaunchCfg& cfg) {
  dev::k_peel<double><<<cfg.blocks, cfg.threads, 0, cfg.stream>>>(
      m, t, d, a, static_cast<const dev::PeelRec<double>*>(w.queue[q]), w.qcount[q], w.next_ray[q]);
  return cudaGetLastError();
}

size_t slot_bytes_fp64() { return sizeof(dev::Slot<double>); }
size_t rec_bytes_fp64() { return sizeof(dev::PeelRec<double>); }
const void* wave_fn_fp64() { return (const void*)dev::k_wave<double, true, true>; }
const void* peel_fn_fp64() { return (const void*)dev::k_peel<double>; }

}  // namespace hc3d
