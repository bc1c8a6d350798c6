// batch_max.h -- the work items of the batched max|f| pass (batch.cu
// k_batch_absmax): host arithmetic, no CUDA.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <vector>

namespace fdb {
namespace bt {

// Equal chunks of every instance's cells, a thread block each: first[i] is the
// first chunk of instance i, first[count] their number.  Chunks of a block's 256
// threads x 4 loads in flight up to 8 times that, as the batch has cells for a
// wave of blocks; small instances get one, however large the largest is.
struct MaxChunks {
  uint64_t cells = 0;
  std::vector<uint64_t> first;
};

inline MaxChunks max_chunks(const std::vector<uint64_t>& sizes) {
  constexpr uint64_t kWave = 152 * 8, kMin = 256 * 4, kMax = 8 * kMin;
  MaxChunks m;
  uint64_t total = 0;
  for (uint64_t s : sizes) total += s;
  m.cells = std::min(kMax, std::max(kMin, total / kWave));
  m.first.assign(1, 0);
  for (uint64_t s : sizes) m.first.push_back(m.first.back() + (s + m.cells - 1) / m.cells);
  return m;
}

}  // namespace bt
}  // namespace fdb
