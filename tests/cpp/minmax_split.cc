// The rules by which a compress call is dealt to blocks (csrc/kernels/minmax_split.h): over sizes, counts and alignments, in contexts
// that can run clusters of any size or none, a call gets no larger cluster than there is, and the slots that it needs otherwise.
#include <cstdio>

#include "kernels/minmax_split.h"

using namespace bagua::kernels::cuda::minmax_split;

int main() {
  long cases = 0, clusters = 0, failures = 0;
  for (int largest : {1, 2, 4, 8, 16})
    for (int n_chunks : {1, 2, 3, 8, 9, 16, 64, 1000})
      for (int64_t bytes = 2; bytes < (1ll << 31); bytes = bytes * 5 / 4 + 1)
        for (bool aligned : {false, true})
          for (int count : {n_chunks, 1}) {  // all chunks, or one of them
            ++cases;
            const int blocks = cluster_blocks(bytes, count, aligned, largest);
            clusters += blocks > 1;
            bool ok = blocks <= 1 || blocks <= largest;
            if (blocks == 0) {
              const Split d = split_chunks(count, bytes, aligned, 148);
              ok = ok && d.grid() <= 148 * kBlocksPerSM && scratch_bytes(n_chunks, bytes, 148, largest) >= slot_bytes(count, d.per_chunk);
            }
            // a block alone keeps a tile; the slices of a cluster are two tiles at most
            ok = ok && (blocks == 1) == (bytes <= kTileBytes) && (blocks < 2 || bytes <= blocks * 2 * kTileBytes);
            if (!ok && ++failures < 10)
              std::fprintf(stderr, "largest %d, %d of %d chunks of %lld bytes, aligned %d: %d blocks\n", largest, count, n_chunks, (long long)bytes,
                           aligned, blocks);
          }
  // the whole GPU, as before
  const bool full = cluster_blocks(1 << 20, 1, true, 16) == 16 && cluster_blocks(1 << 20, 16, true, 16) == 0 && cluster_blocks(2 << 20, 1, true, 16) == 16 &&
                    cluster_blocks((2 << 20) + 1, 1, true, 16) == 0 && cluster_blocks((1 << 20) + 1, 1, false, 16) == 0 && scratch_bytes(8, 1 << 20, 148, 16) == 0;
  std::printf("%ld cases, %ld of them by clusters, %ld failures\n", cases, clusters, failures + !full);
  return failures || !full || clusters == 0;
}
