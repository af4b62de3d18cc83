// Flatten / unflatten of a staged bucket, or of several, in ONE launch.
//
// A bucket whose tensors are not address-contiguous is communicated through a flat staging
// buffer (reference: one cudaMemcpyAsync per tensor into the buffer and one per tensor back,
// bagua-core-internal/src/datatypes/mod.rs:1012-1023 and 1048-1059; for a bucket of 400
// tensors that is 800 copies per bucket per step).  Here a table of {tensor address, offset in
// the flat buffer, bytes}, sorted by offset, lives on the device and one kernel moves every
// tensor: the flat byte range is cut into 16 KiB tiles; the threads of a block look for the first segment of
// its tile in parallel (a binary search over the table was five dependent reads, half of the 5 us that a 7 MB
// bucket took) and copy the overlap of every segment with the tile, 16 bytes per thread.  Where source and
// destination are not aligned to each other the destination still is, and its vectors are put together from the
// words around them.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels_impl.h"
#include "launch.cuh"

namespace bagua {
namespace kernels {
namespace cuda {

namespace {

constexpr int kMcThreads = 256;
constexpr unsigned long long kTileBytes = 16ull << 10;

// Copies n bytes, any alignment; whole blocks take part.
__device__ __forceinline__ void copy_range(char* __restrict__ dst, const char* __restrict__ src, int n) {
  const int tid = (int)threadIdx.x;
  const int head = min(n, (int)((0 - reinterpret_cast<uintptr_t>(dst)) & 15u));
  if (tid < head) dst[tid] = src[tid];
  dst += head;
  src += head;
  const int nv = (n - head) / 16;
  uint4* d = reinterpret_cast<uint4*>(dst);
  if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
    const uint4* s = reinterpret_cast<const uint4*>(src);
    int i = tid;
    for (; i + 3 * kMcThreads < nv; i += 4 * kMcThreads) {
      const uint4 a = s[i], b = s[i + kMcThreads], c = s[i + 2 * kMcThreads], e = s[i + 3 * kMcThreads];
      d[i] = a;
      d[i + kMcThreads] = b;
      d[i + 2 * kMcThreads] = c;
      d[i + 3 * kMcThreads] = e;
    }
    for (; i < nv; i += kMcThreads) d[i] = s[i];
  } else {
    const uint32_t sh = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 3u) * 8;
    const uint32_t* s = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)3);
#pragma unroll 2
    for (int i = tid; i < nv; i += kMcThreads) {
      const uint32_t* w = s + 4 * i;
      const uint32_t a = w[0], b = w[1], c = w[2], e = w[3], f = sh ? w[4] : 0u;  // w[4]: the bytes reach into it
      d[i] = make_uint4(__funnelshift_r(a, b, sh), __funnelshift_r(b, c, sh), __funnelshift_r(c, e, sh),
                        __funnelshift_r(e, f, sh));
    }
  }
  const int done = head + nv * 16;
  if (tid < n - done) dst[nv * 16 + tid] = src[nv * 16 + tid];
}

// Buckets that are copied in one launch; a bucket's tiles follow those of the ones in front of it.  (As few as there are: a launch with
// 650 bytes of parameters reaches the GPU 2-3 us later than one with 50.)
template <int kMost>
struct Joined {
  MultiCopyItem item[kMost];
  unsigned long long end[kMost];  // tiles up to the bucket's last
  int count;
};

// Bytes t0 to t1, a tile, of a bucket's flat range.
__device__ __forceinline__ void copy_tile(const MultiCopySeg* __restrict__ segs, int nseg, char* flat, unsigned long long t0,
                                          unsigned long long t1, int gather) {
  __shared__ MultiCopySeg s_seg[32];
  const int tid = (int)threadIdx.x;
  // segments are sorted by offset and do not overlap: the first of the tile is the number of those that end in front
  int first = 0;
  for (int k0 = 0; k0 < nseg; k0 += kMcThreads) {
    const int k = k0 + tid;
    const int n = __syncthreads_count(k < nseg && segs[k].offset + segs[k].bytes <= t0);
    first += n;
    if (n < kMcThreads) break;
  }
  bool more = true;
  for (int k0 = first; more && k0 < nseg; k0 += 32) {
    if (tid < 32 && k0 + tid < nseg) s_seg[tid] = segs[k0 + tid];
    __syncthreads();
    for (int k = 0; k < 32 && k0 + k < nseg; ++k) {
      const MultiCopySeg& sg = s_seg[k];
      if (sg.offset >= t1) {
        more = false;
        break;
      }
      const unsigned long long a = max(sg.offset, t0), b = min(sg.offset + sg.bytes, t1);
      if (b <= a) continue;
      char* in_flat = flat + a;
      char* in_tensor = reinterpret_cast<char*>(sg.ptr) + (a - sg.offset);
      if (gather)
        copy_range(in_flat, in_tensor, (int)(b - a));
      else
        copy_range(in_tensor, in_flat, (int)(b - a));
    }
    __syncthreads();
  }
}

template <int kMost>
__global__ void __launch_bounds__(kMcThreads)
    multi_copy_kernel(const __grid_constant__ Joined<kMost> joined, int gather) {
  wait_for_predecessor();
  int bucket = 0;
  unsigned long long before = 0;  // tiles in front of the bucket
  const unsigned long long tiles = joined.end[kMost == 1 ? 0 : joined.count - 1];
  for (unsigned long long at = blockIdx.x; at < tiles; at += gridDim.x) {
    if constexpr (kMost > 1)
      while (at >= joined.end[bucket]) before = joined.end[bucket++];
    const MultiCopyItem& item = joined.item[kMost == 1 ? 0 : bucket];
    const unsigned long long t0 = (at - before) * kTileBytes;
    copy_tile(item.segs, item.nseg, (char*)item.flat, t0, min(t0 + kTileBytes, (unsigned long long)item.bytes), gather);
  }
}

}  // namespace

namespace {
template <int kMost>
void launch_joined(const MultiCopyItem* items, int count, bool gather, cudaStream_t s) {
  Joined<kMost> j;
  j.count = 0;
  unsigned long long tiles = 0;
  for (int k = 0; k < count; ++k) {
    if (items[k].nseg <= 0 || items[k].bytes == 0) continue;
    tiles += (items[k].bytes + kTileBytes - 1) / kTileBytes;
    j.item[j.count] = items[k];
    j.end[j.count++] = tiles;
  }
  if (tiles == 0) return;
  const int grid = (int)std::min<unsigned long long>(tiles, 1ull << 30);
  launch_overlapped(multi_copy_kernel<kMost>, dim3(grid), dim3(kMcThreads), s, j, gather ? 1 : 0);
}
}  // namespace

void multi_copy_joined(const MultiCopyItem* items, int count, bool gather, cudaStream_t s) {
  BAGUA_CHECK(count <= kMaxJoined, Tensor, "too many buckets for one launch");
  if (count == 1)
    launch_joined<1>(items, count, gather, s);
  else if (count <= 4)
    launch_joined<4>(items, count, gather, s);
  else
    launch_joined<kMaxJoined>(items, count, gather, s);
}

void multi_copy(const MultiCopySeg* segs_dev, int nseg, void* flat, size_t total_bytes, bool gather, cudaStream_t s) {
  const MultiCopyItem one{segs_dev, nseg, flat, total_bytes};
  multi_copy_joined(&one, 1, gather, s);
}

}  // namespace cuda
}  // namespace kernels
}  // namespace bagua
