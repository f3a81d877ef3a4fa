// Lattice coordinates of the FP32 core's fast samplers (wg_unit.cuh, wg_lists.cuh), on the device and, for the
// tests, on the host: 8.56 fixed point, mod 256 (the tables' period).
//
// A coordinate is its unit's base per table and axis plus the hut's chunk offset times the table's step, exact
// to 2^-40 of a cell over a unit.  The top byte is the lattice cell, the 32 bits below it the fraction, which
// one conversion rounds to FP32, within 2^-25 as after an FP64 reduction.  Against the exact sample, 8 million
// samples of random tables (u = 2^-24; largest, root mean square): after an FP64 reduction 3.96 and 0.47 u, so
// 3.96 and 0.47 u, from lattice columns 3.52 and 0.44 u.  A 23-bit fraction shifted into the mantissa gave 4.10
// and 0.70, 4.65 and 0.68 u and was no faster (one seed over the whole world took 1.1 % longer with it).
#pragma once

#include <cmath>
#include <cstdint>

#ifdef __CUDACC__
#define WG_FIXED_FN __host__ __device__ __forceinline__
#else
#define WG_FIXED_FN inline
#endif

namespace wg {

WG_FIXED_FN uint64_t to_fixed(double v) { return (uint64_t)((v - 256.0 * floor(v * (1.0 / 256.0))) * 72057594037927936.0); }
WG_FIXED_FN uint64_t fixed_at(uint64_t base, uint64_t step, uint32_t d) { return base + d * step; }
WG_FIXED_FN uint32_t fixed_cell(uint64_t v) { return (uint32_t)(v >> 56); }
// The fraction in [0, 1] (1 only by rounding: the sample is continuous there).
WG_FIXED_FN float fixed_frac(uint64_t v) { return (float)(uint32_t)(v >> 24) * 2.3283064365386963e-10f; }

}  // namespace wg
