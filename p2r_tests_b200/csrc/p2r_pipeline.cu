// Host-buffer driver: the track blocks split into chunks whose host->device copy, fused forward and
// device->host copy run on a small pool of streams, so the copies of one chunk overlap the
// kernel of another. This is the transfer pipeline of the reference's multi-stream CUDA
// driver (cuda_v4.cu:912-1010: per-stream cudaMemcpyAsync H2D, kernel, D2H), over the same
// Matriplex arrays. Track blocks and their hit blocks are contiguous in both arrays (track block
// ib + nb*ev, hit block lay + nlayer*(ib + nb*ev)) and independent, so any range of blocks is one
// contiguous byte range of each.
// In restart mode only the last layer reaches the output (the reference's restart loop
// rewrites it at every layer from the same input track), so only that layer's hit block of
// each track block is copied: one strided 2-D copy per chunk, a 1/nlayer share of the hits.
//
// The host link bounds the call (55.5 GB/s host->device); every gap between two copies and the last
// chunk's kernel and copy back come on top. So chunks are equal numbers of blocks, but the last of three
// or more is a quarter of the others; there is at most one for every 4 MiB of input, since smaller copies
// cost more than they hide (a batch below 8 MiB is one chunk; the short last one may have little over
// 1 MiB); and in chained mode the tracks (one byte in seven at 20 layers) go over in one copy before the
// hits.
// Measured on one B200, pinned buffers, 8 chunks asked for, chunks of whole events before -> this:
// 9600 x 10 x 20 1617 -> 1541 us (80 MB in, 1440 us at the link's rate), 9600 x 60 x 20 9.34 -> 8.83 ms,
// 5000 x 7 x 12 470 -> 428 us, 9600 x 1 x 20 203 -> 201 us; restart 9600 x 10 505 -> 440 us. Tracks in
// one copy in restart mode too, where they are most of the bytes: 9600 x 60 2.1 -> 2.5 ms.
#include <cuda_runtime.h>

#include <mutex>

#include "p2r_internal.h"

namespace {

constexpr int kMaxDevices = 64;
constexpr int kPoolStreams = 3;
constexpr size_t kMinChunkBytes = size_t(4) << 20;  // host->device bytes per chunk, on average
constexpr int kLastShare = 4;                       // the last chunk is 1 / kLastShare of another

struct StreamPool {
  std::mutex mu;  // one call at a time enqueues on the pool (the fork / join events are shared)
  bool ready = false;
  cudaStream_t s[kPoolStreams];
  cudaEvent_t fork;
  cudaEvent_t join[kPoolStreams];
};

StreamPool g_pools[kMaxDevices];
std::mutex g_pool_mu;

int get_pool(StreamPool** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return p2r_set_errorf(P2R_ERR_CUDA, "p2r_forward_host: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) return p2r_set_error(P2R_ERR_UNSUPPORTED, "p2r_forward_host: device index");
  std::lock_guard<std::mutex> lk(g_pool_mu);
  StreamPool& p = g_pools[dev];
  if (!p.ready) {
    for (int i = 0; i < kPoolStreams; ++i) p.s[i] = nullptr, p.join[i] = nullptr;
    p.fork = nullptr;
    for (int i = 0; i < kPoolStreams && e == cudaSuccess; ++i) {
      e = cudaStreamCreateWithFlags(&p.s[i], cudaStreamNonBlocking);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&p.join[i], cudaEventDisableTiming);
    }
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&p.fork, cudaEventDisableTiming);
    if (e != cudaSuccess) {  // release what was created, so a later call starts from nothing
      for (int i = 0; i < kPoolStreams; ++i) {
        if (p.join[i]) cudaEventDestroy(p.join[i]);
        if (p.s[i]) cudaStreamDestroy(p.s[i]);
      }
      if (p.fork) cudaEventDestroy(p.fork);
      return p2r_set_errorf(P2R_ERR_CUDA, "p2r_forward_host: %s", cudaGetErrorString(e));
    }
    p.ready = true;
  }
  *out = &p;
  return P2R_OK;
}

}  // namespace

extern "C" int p2r_forward_host(const p2r_config* cfg, const void* host_trk_in, const void* host_hits,
                                void* host_trk_out, void* dev_trk_in, void* dev_hits, void* dev_trk_out,
                                int32_t nchunks, void* stream) {
  P2rRange range("p2r_forward_host");
  int rc = p2r_check_config(cfg, "p2r_forward_host");
  if (rc) return rc;
  if (!host_trk_in || !host_hits || !host_trk_out || !dev_trk_in || !dev_hits || !dev_trk_out)
    return p2r_set_error(P2R_ERR_INVALID, "p2r_forward_host: null pointer");
  if (nchunks < 1) return p2r_set_error(P2R_ERR_INVALID, "p2r_forward_host: nchunks must be >= 1");
  if ((rc = p2r_check_aligned("p2r_forward_host", 4, {dev_trk_in, dev_hits, dev_trk_out}))) return rc;
  if (cfg->nevts == 0 || cfg->nb == 0) return p2r_clear_error();
  {  // the copies write dev_trk_in and dev_hits, the kernels dev_trk_out: all three disjoint
    const size_t tb = (size_t)cfg->nevts * cfg->nb * 28 * cfg->bsize * sizeof(float);
    const size_t hb = (size_t)cfg->nevts * cfg->nb * cfg->nlayer * 9 * cfg->bsize * sizeof(float);
    if ((rc = p2r_check_disjoint("p2r_forward_host", "dev_trk_in and dev_trk_out", dev_trk_in, tb, dev_trk_out, tb)) ||
        (rc = p2r_check_disjoint("p2r_forward_host", "dev_hits and dev_trk_out", dev_hits, hb, dev_trk_out, tb)) ||
        (rc = p2r_check_disjoint("p2r_forward_host", "dev_trk_in and dev_hits", dev_trk_in, tb, dev_hits, hb)))
      return rc;
  }
  StreamPool* pool = nullptr;
  if ((rc = get_pool(&pool))) return rc;
  std::lock_guard<std::mutex> lk(pool->mu);
  const int64_t nblocks = (int64_t)cfg->nevts * cfg->nb;
  const size_t trk_blk = (size_t)28 * cfg->bsize * sizeof(float);
  const size_t hit_blk = (size_t)9 * cfg->bsize * sizeof(float);  // one layer of one track block
  const size_t hit_trk = (size_t)cfg->nlayer * hit_blk;                // all layers of one track block
  const size_t last = (size_t)(cfg->nlayer - 1) * hit_blk;          // offset of the last layer's block
  const bool restart = cfg->mode == P2R_MODE_RESTART;
  const size_t total = (size_t)nblocks * (trk_blk + (restart ? hit_blk : hit_trk));
  int64_t chunks = (int64_t)(total / kMinChunkBytes);
  chunks = chunks < 1 ? 1 : (chunks > nchunks ? nchunks : chunks);
  if (chunks > nblocks) chunks = nblocks;
  cudaStream_t caller = (cudaStream_t)stream;
  cudaError_t e = cudaEventRecord(pool->fork, caller);
  for (int i = 0; i < kPoolStreams && e == cudaSuccess; ++i) e = cudaStreamWaitEvent(pool->s[i], pool->fork, 0);
  if (e != cudaSuccess) return p2r_set_errorf(P2R_ERR_CUDA, "p2r_forward_host: %s", cudaGetErrorString(e));
  // the caller's stream waits for everything queued on the pool, also when a step fails
  auto join = [&]() {
    cudaError_t je = cudaSuccess;
    for (int i = 0; i < kPoolStreams && je == cudaSuccess; ++i) {
      je = cudaEventRecord(pool->join[i], pool->s[i]);
      if (je == cudaSuccess) je = cudaStreamWaitEvent(caller, pool->join[i], 0);
    }
    return je;
  };
  const bool tracks_first = !restart && chunks > 1;
  if (tracks_first) {
    if ((e = cudaMemcpyAsync(dev_trk_in, host_trk_in, nblocks * trk_blk, cudaMemcpyHostToDevice, pool->s[0])) == cudaSuccess &&
        (e = cudaEventRecord(pool->join[0], pool->s[0])) == cudaSuccess)
      for (int i = 1; i < kPoolStreams && e == cudaSuccess; ++i) e = cudaStreamWaitEvent(pool->s[i], pool->join[0], 0);
    if (e != cudaSuccess) {
      join();
      return p2r_set_errorf(P2R_ERR_CUDA, "p2r_forward_host: H2D: %s", cudaGetErrorString(e));
    }
  }
  const int64_t step = chunks > 2 ? kLastShare : 1;
  const int64_t parts = step * (chunks - 1) + 1;
  for (int64_t c = 0; c < chunks; ++c) {
    const int64_t b0 = nblocks * (step * c) / parts, b1 = c + 1 == chunks ? nblocks : nblocks * (step * (c + 1)) / parts;
    if (b1 == b0) continue;
    const int64_t nb = b1 - b0;
    cudaStream_t s = pool->s[c % kPoolStreams];
    char* dti = (char*)dev_trk_in + b0 * trk_blk;
    char* dh = (char*)dev_hits + b0 * hit_trk;
    char* dto = (char*)dev_trk_out + b0 * trk_blk;
    if ((!tracks_first && (e = cudaMemcpyAsync(dti, (const char*)host_trk_in + b0 * trk_blk, nb * trk_blk,
                                               cudaMemcpyHostToDevice, s)) != cudaSuccess) ||
        (e = restart ? cudaMemcpy2DAsync(dh + last, hit_trk, (const char*)host_hits + b0 * hit_trk + last, hit_trk, hit_blk,
                                         (size_t)nb, cudaMemcpyHostToDevice, s)
                     : cudaMemcpyAsync(dh, (const char*)host_hits + b0 * hit_trk, nb * hit_trk, cudaMemcpyHostToDevice,
                                       s)) != cudaSuccess) {
      join();
      return p2r_set_errorf(P2R_ERR_CUDA, "p2r_forward_host: H2D: %s", cudaGetErrorString(e));
    }
    p2r_config sub = *cfg;
    sub.nevts = 1;
    sub.nb = nb;
    if ((rc = p2r_forward(&sub, dti, dh, dto, nullptr, nullptr, s))) {
      join();
      return rc;
    }
    if ((e = cudaMemcpyAsync((char*)host_trk_out + b0 * trk_blk, dto, nb * trk_blk, cudaMemcpyDeviceToHost,
                             s)) != cudaSuccess) {
      join();
      return p2r_set_errorf(P2R_ERR_CUDA, "p2r_forward_host: D2H: %s", cudaGetErrorString(e));
    }
  }
  if ((e = join()) != cudaSuccess)
    return p2r_set_errorf(P2R_ERR_CUDA, "p2r_forward_host: %s", cudaGetErrorString(e));
  return p2r_clear_error();
}
