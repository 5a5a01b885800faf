// Included ahead of fixed_check.cpp: an operation of csrc/fixed_geodesic.cuh
// that loses bits of its value ends the program, and so does a sum of products
// whose cross terms (a 32-bit half of one factor times the other's) could come
// to more than 64 bits with other low halves.
#include <cmath>
#include <cstdlib>
#define FX_KEPT(ok) ((ok) ? (void)0 : std::abort())
#define FX_TRACK(code) code
static inline double fx_most(int ah, int bh) { return 0x1p31 * (std::fabs((double)ah) + std::fabs((double)bh)); }
