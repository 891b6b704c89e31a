// Host build of row_magic and row_of (dmsc_b200/csrc/common.cuh) for the CPU
// test: rows of the indices l[0 .. n) of an image of nx indices a row.
#include "../../dmsc_b200/csrc/common.cuh"

extern "C" void row_of_host(int nx, const int* l, int* row, int n, unsigned* magic, int* shift) {
  dmsc::row_magic(nx, magic, shift);
  dmsc::Imgs I{};
  I.magic = magic;
  I.shift = shift;
  for (int i = 0; i < n; ++i) row[i] = dmsc::row_of(I, 0, l[i]);
}
