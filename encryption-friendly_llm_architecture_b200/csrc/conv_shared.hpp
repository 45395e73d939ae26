// Shared memory of the conversions between column passes (convcols.cuh): strips of 256 rows, then the constants of all targets.
#pragma once
#include <cstddef>

#ifdef __CUDACC__
#define HB_EVERYWHERE __host__ __device__
#else
#define HB_EVERYWHERE
#endif

namespace hb {

constexpr int kFpSources = 4; // conversions of up to so many sources may run on the FP64 pipe, whose constants are twice as long
// 16-byte words that there is room for per target, half of the rows and source
HB_EVERYWHERE constexpr int conv_const_words(int sources) { return sources > kFpSources ? 1 : 2; }
constexpr std::size_t conv_const_bytes(int sources, int targets) { return (std::size_t)2 * sources * targets * conv_const_words(sources) * 16; }
HB_EVERYWHERE constexpr int strip_words(int cols) { return 256 * cols + 16 * cols; } // `cols` pad words per 16 rows
constexpr std::size_t strip_bytes(int cols, int strips) { return (std::size_t)strips * strip_words(cols) * 8; }

} // namespace hb
