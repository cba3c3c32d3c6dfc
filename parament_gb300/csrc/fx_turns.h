// Which `finished` barrier and phase a product of an fx launch (fx.cuh) completes,
// and what its cutters wait for.  Plain integer functions, so that the CPU tests can
// walk every order of events.
//
// A wait names a phase by its parity alone, so a barrier must not complete two phases
// while a cutter still waits for the first.  The finishers may be done with every
// product that the cutter has handed over, n - 1 included, when it comes to wait for
// product n - 2.  On one barrier that is the phase after, and the wait would be for
// good; with the products on two barriers in turn, a barrier's next phase is product
// n itself, which this cutter has not begun.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define PGB_TURNS __host__ __device__ constexpr
#else
#define PGB_TURNS constexpr
#endif

namespace pgb {
namespace fx {

constexpr uint32_t kFinishedBars = 2;

PGB_TURNS uint32_t finished_bar(uint32_t n) { return n % kFinishedBars; }
PGB_TURNS uint32_t finished_parity(uint32_t n) { return (n / kFinishedBars) & 1; }
// Products that are finished before a cutter touches product n: up to n - 2, and n - 1
// where n takes its operands from it.
PGB_TURNS uint32_t finished_before(uint32_t n, bool needs) { return n == 0 ? 0 : n - (needs ? 0 : 1); }

}  // namespace fx
}  // namespace pgb
