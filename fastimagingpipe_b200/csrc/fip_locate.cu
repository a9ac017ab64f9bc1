// Trigger post-processing: transient locations from a tLISI matrix.
//
// The reference's command line writes the raw tLISI matrix and names the
// file locations.fits (README.md:41); reducing the matrix to locations is the
// step that name promises.  A location is a tile whose tLISI is below a
// threshold and is the strict minimum of its 3 x 3 neighbourhood (ties go to
// the lower tile index), refined to the centroid of the neighbourhood's
// drops 1 - tLISI and mapped to image pixels and to the reference's SIN
// projection-plane offsets (p2p's x0, y0 at FIPkernels.cu:317-322 for a
// destination pixel: x = -cell (col - N/2 - 1), y = cell (row - N/2 - 1)).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/fip.h"
#include "fip_common.cuh"
#include "fip_kernels.h"

static_assert(sizeof(fip_location) == 28, "fip_location is seven 4-byte fields");

namespace {

constexpr int kThreads = 256;

// The location at tile b of the matrix t, if there is one.
__device__ __forceinline__ bool location_at(const float* __restrict__ t, int b, int u, int tile,
                                            int n, float cell, float threshold,
                                            fip_location& L) {
  const float v = t[b];
  if (!(v < threshold)) return false;  // NaN tiles never qualify
  const int r = b / u, c = b % u;
  float ws = 0.f, wr = 0.f, wc = 0.f;
  for (int dr = -1; dr <= 1; ++dr)
    for (int dc = -1; dc <= 1; ++dc) {
      const int rr = r + dr, cc = c + dc;
      if (rr < 0 || rr >= u || cc < 0 || cc >= u) continue;
      const int nb = rr * u + cc;
      const float w = t[nb];
      if (nb != b && (w < v || (w == v && nb < b))) return false;  // not the minimum
      const float drop = w == w ? fmaxf(0.f, 1.0f - w) : 0.f;
      ws += drop;
      wr += drop * (float)dr;
      wc += drop * (float)dc;
    }
  const float fr = (float)r + (ws > 0.f ? wr / ws : 0.f);
  const float fc = (float)c + (ws > 0.f ? wc / ws : 0.f);
  // Tile k covers pixels k T .. k T + T - 1: its centre is k T + (T - 1) / 2.
  const float row = fr * (float)tile + 0.5f * (float)(tile - 1);
  const float col = fc * (float)tile + 0.5f * (float)(tile - 1);
  const float h1 = (float)(n / 2 + 1);
  L.tile_row = r;
  L.tile_col = c;
  L.tlisi = v;
  L.row = row;
  L.col = col;
  L.x = -cell * (col - h1);
  L.y = cell * (row - h1);
  return true;
}

// One thread per tile.  out holds room for `cap` records; *count receives the
// number of locations found (records past cap are dropped, the count is not).
__global__ void k_locate(const float* __restrict__ t, int u, int tile, int n, float cell,
                         float threshold, fip_location* __restrict__ out, unsigned* count,
                         unsigned cap) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= u * u) return;
  fip_location L;
  if (!location_at(t, b, u, tile, n, cell, threshold, L)) return;
  const unsigned k = atomicAdd(count, 1u);
  if (k < cap) out[k] = L;
}

// Matrices of up to kOneLaunch tiles: one cluster of eight CTAs walks the
// matrix (coalesced), counts in the first CTA's shared memory and writes its
// few records and their number straight to pinned host memory, so a call is
// one launch and one wait, with no device scratch and no copies.  A 128 x 128
// matrix with 169 locations: 46.5 us a call in the scratch-and-copy form (an
// allocation and its release, a memset, a launch and two synchronising
// copies), 25.2 us in this one (3.9 us of it the kernel; the rest is the wait
// and the caller); 512 x 512 195 and 163 us.  Beyond that the eight CTAs would
// become the bound.  Two minima are never neighbours, so ceil(u / 2)^2 records
// always hold them all.
constexpr int kOneLaunch = 1 << 18, kOneThreads = 1024, kOneCluster = 8;
struct HostRecords {
  unsigned count;
  unsigned cap;  // records the block has room for (host only)
  __host__ __device__ fip_location* rec() { return reinterpret_cast<fip_location*>(this + 1); }
};
__global__ void __cluster_dims__(kOneCluster, 1, 1) __launch_bounds__(kOneThreads)
    k_locate_one(const float* __restrict__ t, int u, int tile, int n, float cell,
                 float threshold, HostRecords* out, unsigned cap) {
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  __shared__ unsigned s_count;
  if (threadIdx.x == 0) s_count = 0;
  cluster.sync();
  unsigned* count = cluster.map_shared_rank(&s_count, 0);
  for (int b = blockIdx.x * kOneThreads + threadIdx.x; b < u * u;
       b += kOneCluster * kOneThreads) {
    fip_location L;
    if (!location_at(t, b, u, tile, n, cell, threshold, L)) continue;
    const unsigned k = atomicAdd(count, 1u);
    if (k < cap) out->rec()[k] = L;
  }
  cluster.sync();
  if (blockIdx.x == 0 && threadIdx.x == 0) out->count = s_count;
}

// Pinned record blocks, one per call in flight (any thread, any device), their
// room a power of two from kLeast records up; at most kKeep idle ones are kept
// (14.7 MB if all are of the largest size), the rest are freed.
class RecordPool {
 public:
  static RecordPool& get() {
    // Never destroyed: idle blocks at exit are left to the driver's teardown.
    static RecordPool& pool = *new RecordPool;
    return pool;
  }
  // A block with room for `records`: the smallest idle one, or a new one.
  HostRecords* take(unsigned records) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      auto best = idle_.end();
      for (auto it = idle_.begin(); it != idle_.end(); ++it)
        if ((*it)->cap >= records && (best == idle_.end() || (*it)->cap < (*best)->cap)) best = it;
      if (best != idle_.end()) {
        HostRecords* p = *best;
        idle_.erase(best);
        return p;
      }
    }
    unsigned cap = kLeast;
    while (cap < records) cap *= 2;
    void* p = nullptr;
    if (cudaHostAlloc(&p, sizeof(HostRecords) + cap * sizeof(fip_location),
                      cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    HostRecords* h = static_cast<HostRecords*>(p);
    h->cap = cap;
    return h;
  }
  // Keeps the block; of kKeep + 1 the smallest is freed, so that blocks left by
  // small matrices do not keep a larger one from staying.
  void give(HostRecords* p) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      idle_.push_back(p);
      if (idle_.size() <= kKeep) return;
      auto least = std::min_element(idle_.begin(), idle_.end(),
                                    [](const HostRecords* a, const HostRecords* b) {
                                      return a->cap < b->cap;
                                    });
      p = *least;
      idle_.erase(least);
    }
    cudaFreeHost(p);
  }

 private:
  RecordPool() { idle_.reserve(kKeep + 1); }
  static constexpr size_t kKeep = 8;
  static constexpr unsigned kLeast = 4096;
  std::mutex mu_;
  std::vector<HostRecords*> idle_;
};

// Deepest drop first; equal values in tile order (the kernels' record order
// depends on scheduling, the returned order does not).
void sort_records(fip_location* rec, size_t count, size_t u) {
  std::sort(rec, rec + count, [u](const fip_location& a, const fip_location& b) {
    if (a.tlisi != b.tlisi) return a.tlisi < b.tlisi;
    return (size_t)a.tile_row * u + a.tile_col < (size_t)b.tile_row * u + b.tile_col;
  });
}

// The one-launch form; false when it does not apply (a large matrix, a
// capturing stream, no pinned memory).
bool locate_one(const float* tlisi, size_t u, size_t unit_size, size_t image_size,
                float cell_size, float threshold, fip_location* out, size_t max_out,
                size_t* found, cudaStream_t s, cudaError_t* err) {
  *err = cudaSuccess;
  if (u * u > (size_t)kOneLaunch) return false;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (cap != cudaStreamCaptureStatusNone) return false;
  const unsigned room = (unsigned)((u + 1) / 2 * ((u + 1) / 2));
  HostRecords* h = RecordPool::get().take(room);
  if (!h) return false;
  k_locate_one<<<kOneCluster, kOneThreads, 0, s>>>(tlisi, (int)u, (int)unit_size, (int)image_size,
                                                   cell_size, threshold, h, h->cap);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    *err = e;  // the block is not reused: the kernel may still write it
    return true;
  }
  const unsigned count = std::min(h->count, h->cap);
  fip_location* rec = h->rec();
  sort_records(rec, count, u);
  for (size_t k = 0; k < count && k < max_out; ++k) out[k] = rec[k];
  *found = count;
  RecordPool::get().give(h);
  return true;
}

}  // namespace

extern "C" int fip_locate_transients(const float* tlisi, size_t image_size, size_t unit_size,
                                     float cell_size, float threshold, fip_location* out,
                                     size_t max_out, size_t* found, void* stream) {
  if (!tlisi || !found || (max_out > 0 && !out))
    return fip_set_error(FIP_ERR_ARG, "null argument");
  if (unit_size == 0 || image_size < unit_size)
    return fip_set_error(FIP_ERR_ARG, "unit_size must be in [1, image_size]");
  if (!(cell_size > 0.f)) return fip_set_error(FIP_ERR_ARG, "cell_size must be positive");
  const size_t u = image_size / unit_size;
  if (u * u > (1u << 26)) return fip_set_error(FIP_ERR_ARG, "tLISI matrix too large");
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = cudaSuccess;
  if (locate_one(tlisi, u, unit_size, image_size, cell_size, threshold, out, max_out, found, s,
                 &e))
    return e == cudaSuccess ? FIP_OK : fip_set_error(FIP_ERR_CUDA, cudaGetErrorString(e));
  const size_t cap = u * u;  // every tile could qualify
  // Stream-ordered scratch (post-processing, not the imaging hot path): the
  // records and the count in one block.
  char* scratch = nullptr;
  const size_t rec_bytes = cap * sizeof(fip_location);
  e = cudaMallocAsync((void**)&scratch, rec_bytes + 16, s);
  if (e != cudaSuccess) return fip_set_error(FIP_ERR_NOMEM, cudaGetErrorString(e));
  fip_location* d_rec = reinterpret_cast<fip_location*>(scratch);
  unsigned* d_count = reinterpret_cast<unsigned*>(scratch + rec_bytes);
  unsigned count = 0;
  std::vector<fip_location> rec;
  e = cudaMemsetAsync(d_count, 0, sizeof(unsigned), s);
  if (e == cudaSuccess) {
    k_locate<<<(unsigned)((cap + kThreads - 1) / kThreads), kThreads, 0, s>>>(
        tlisi, (int)u, (int)unit_size, (int)image_size, cell_size, threshold, d_rec, d_count,
        (unsigned)cap);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&count, d_count, sizeof(unsigned),
                                            cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess && count > 0) {
    rec.resize(std::min<size_t>(count, cap));
    e = cudaMemcpyAsync(rec.data(), d_rec, rec.size() * sizeof(fip_location),
                        cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  const cudaError_t ef = cudaFreeAsync(scratch, s);
  if (e == cudaSuccess) e = ef;
  if (e != cudaSuccess) return fip_set_error(FIP_ERR_CUDA, cudaGetErrorString(e));
  sort_records(rec.data(), rec.size(), u);
  for (size_t k = 0; k < rec.size() && k < max_out; ++k) out[k] = rec[k];
  *found = count;
  return FIP_OK;
}
