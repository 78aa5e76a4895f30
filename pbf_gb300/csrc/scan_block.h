// scan_block.h — threads per block of the scanning sweeps (lambda and the first
// vorticity pass).  Host code only, so that a CPU test covers the rule.
#pragma once

#include <cstdint>

namespace pbf {

// The blocks that share an SM come from all over the particle order, so a larger
// block means fewer places whose records and lists have to fit in the SM's L1;
// it also waits longer for its slowest warp.  Where the caller chose no block
// (pbf_tuning.block_size 0) and the sweep records pair lists (`pairs`), the lines
// lie where whole runs gain.  Measured at 256 /
// 512 / 1,024 threads (the vorticity pass at most 512: registers), ms:
//   one scene, collapsing: 1.6 million particles, 20 substeps 67.2 / 67.2 / 68.0,
//     2.1 million 83.0 / 81.5 / 81.8, 3.2 million 133.5 / 126.1 / 129.2, 4.5 million
//     205.5 / 191.8 / 177.7, 7.2 million, 16 substeps 247.8 / 228.5 / 209.9;
//   one scene, calm: 2.1 million 60.6 / 61.3 / 63.1, 4.5 million, 12 substeps 77.5 /
//     75.4 / 76.1;
//   batches, 4 substeps, collapsing / calm: 2.35 million 16.5 / 16.3 / 16.6 and 14.2 /
//     14.4 / 14.9, 4.7 million 31.0 / 29.1 / 27.9 and 23.7 / 23.5 / 24.0, 9.3 million
//     66.2 / 62.0 / 59.1 and 50.6 / 50.1 / 51.5.
// The other forms have no lists to keep in L1 and only wait longer: us per
// launch at 256 threads and under the lines above, 7.2 million particles at rest,
// lambda direct 1,703 / 1,742, replaying skin lists 1,429 / 1,536, masked without
// lists 1,187 / 1,229; vorticity 2,152 / 2,174, 1,675 / 1,766, 1,393 / 1,420.  They
// stay at 256.
constexpr uint32_t kMidScene = 1572864, kLargeScene = 4194304;
constexpr unsigned kScanBlock = 256;

inline unsigned scan_block(uint32_t asked, uint32_t n, bool pairs, unsigned largest) {
    if (asked) return asked;
    if (!pairs) return kScanBlock;
    const unsigned block = n < kMidScene ? kScanBlock : n < kLargeScene ? 512u : 1024u;
    return block < largest ? block : largest;
}

}  // namespace pbf
