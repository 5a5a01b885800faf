// Included ahead of fixed_check.cpp: an operation of csrc/fixed_geodesic.cuh
// that loses bits of its value ends the program.
#include <cstdlib>
#define FX_KEPT(ok) ((ok) ? (void)0 : std::abort())
