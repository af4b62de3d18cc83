// How the chunks of a MinMaxUInt8 compress call are dealt to blocks: the rules behind minmax_uint8.cu, host only.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace bagua {
namespace kernels {
namespace cuda {
namespace minmax_split {

constexpr int kBlocksPerSM = 2;  // 64 registers per thread
constexpr int64_t kTileBytes = 64 << 10;  // of a tile
// Smallest slice of a block: more blocks read a chunk faster but wait longer for each other (10 MB of fp32 in
// 8 chunks: 8.1 us with 16 KiB, 6.9 with 64; unaligned elements, which take more instructions to load, 1 M of
// fp16 in 3 chunks: 9.4 us with 64 KiB, 7.5 with 32).
constexpr int64_t kSliceBytes = 64 << 10, kSliceBytesUnaligned = 32 << 10;
constexpr int64_t kGroupBytes = 32ll << 20;    // two groups and their output are in L2 (126 MB) at a time

// How the chunks of a call are dealt to blocks.  Calls of several groups have two sets of blocks, one of each
// set on every SM, which take the groups in turn: while one set quantises its group, which is bound by
// instructions (8 per element), the other reads the next from memory.
struct Split {
  int sets;
  int per_group;  // chunks in flight together in a set
  int per_chunk;  // blocks of one chunk
  int grid() const { return sets * per_group * per_chunk; }
};
inline Split split_chunks(int count, int64_t chunk_bytes, bool aligned, int sms) {
  Split s;
  const int64_t all = (int64_t)sms * kBlocksPerSM;
  s.per_group = (int)std::max<int64_t>(1, std::min({kGroupBytes / chunk_bytes, (int64_t)count, all}));
  s.sets = s.per_group < count && chunk_bytes > kTileBytes ? 2 : 1;
  if (s.sets == 2) s.per_group = std::min(s.per_group, sms);
  // a chunk of one tile stays with one block, which then waits for nobody
  s.per_chunk = chunk_bytes <= kTileBytes
                    ? 1
                    : (int)std::max<int64_t>(1, std::min<int64_t>(all / s.sets / s.per_group,
                                                                  chunk_bytes / (aligned ? kSliceBytes : kSliceBytesUnaligned)));
  return s;
}

// A chunk's slots, through which its blocks agree: one per block and one more.
constexpr int kSlotBytes = 16;
inline size_t slot_bytes(int count, int per_chunk) { return (size_t)count * (per_chunk + 1) * kSlotBytes; }

// Smaller chunks belong to a cluster instead, whose blocks agree through each other's shared memory: nothing of the launch has
// to be resident as a whole, it may start while its predecessor ends, and it needs no slots.  (Cooperative launches follow each
// other in steps of 2 us.)  Up to 8 chunks have up to 16 blocks each; more chunks have 8, as clusters of 16 do not find room on all
// SMs at once.  The last slice sizes are those beyond which the launch of all SMs is as fast or faster.  us, cooperative / cluster:
// fp32, one chunk of 128 KB 6.2/4.3, 1 MB 6.2/4.4, 1.6 MB 8.2/6.1, 2.1 MB 8.2/6.8, 3.2 MB 8.2/9.0; 8 chunks of 0.4 MB 8.2/5.2, of 1.3 MB
// 8.2/7.5, of 2 MB 10.3/9.0; 16 chunks of 0.4 MB 8.2/8.5 by 16 and 5.8 by 8 blocks, of 1.3 MB 10.3/10.7 by 8; unaligned fp16,
// 3 chunks of 0.7 MB 9.4/7.8, of 1.4 MB 9.5/10.2.
constexpr int64_t kClusterSlice = 32 << 10;  // aimed at
// Blocks of the cluster that handles a chunk of this size; 1: a block alone, 0: no cluster.  `largest`: of the clusters that the stream's
// context can run.
inline int cluster_blocks(int64_t chunk_bytes, int count, bool aligned, int largest) {
  const int most = std::min(count <= 8 ? 16 : 8, largest);
  if (chunk_bytes <= kTileBytes) return 1;
  if (most < 2) return 0;
  if (chunk_bytes > most * (!aligned ? kTileBytes : count <= 8 ? 2 * kTileBytes : kTileBytes + kTileBytes / 2)) return 0;
  int n = 2;
  while (n < most && n * kClusterSlice < chunk_bytes) n *= 2;
  return n;
}

// What a call for all chunks of a buffer, or for one of them, needs in slots; a call for one may give that chunk more blocks.
inline size_t scratch_bytes(int n_chunks, int64_t chunk_bytes, int sms, int largest) {
  size_t most = 0;
  for (int count : {n_chunks, 1})
    if (!cluster_blocks(chunk_bytes, count, false, largest))
      most = std::max(most, slot_bytes(count, split_chunks(count, chunk_bytes, false, sms).per_chunk));
  return most;
}

}  // namespace minmax_split
}  // namespace cuda
}  // namespace kernels
}  // namespace bagua
