// Bit spread of Morton codes, on the host and the device.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define TCLOTH_HD __host__ __device__
#else
#define TCLOTH_HD
#endif

namespace tcloth {

// bit k of the 10-bit v to bit 3k
TCLOTH_HD inline uint32_t morton_spread10(uint32_t v) {
  v = (v * 0x00010001u) & 0xFF0000FFu;
  v = (v * 0x00000101u) & 0x0F00F00Fu;
  v = (v * 0x00000011u) & 0xC30C30C3u;
  v = (v * 0x00000005u) & 0x49249249u;
  return v;
}

}  // namespace tcloth
