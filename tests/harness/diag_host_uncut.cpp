// The emulation of diag_host.cpp with rows that do not cut columns at m, the
// form of launches none of whose read lengths crosses (columns_cross).
#include "../../saruman_b200/csrc/diag_tile.cuh"

#define MismatchRows MismatchRowsUncut
#include "diag_host.cpp"

extern "C" int diag_columns_cross(int max_m, int k) { return columns_cross(max_m, k); }
