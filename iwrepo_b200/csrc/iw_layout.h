// Shared-memory layout of the z operators on the FP64 tensor cores, as plain constants: kernels, launch
// code and the tests on the host use the same ones.
#pragma once
#include <cstddef>

#ifdef __CUDACC__
#define IW_HD __host__ __device__
#else
#define IW_HD
#endif

constexpr int kTcMaxN = 40;
// Operator columns in shared memory are AP = 4 (mod 8) doubles apart: the 4
// columns x 8 rows of a B fragment then fall in two shared-memory wavefronts.
// They are padded to a multiple of 4 columns with zeros, so that no fragment
// needs a bounds check.
IW_HD constexpr int tc_nt(int N) { return N <= 16 ? 2 : (N + 7) / 8; }
IW_HD constexpr int tc_ap(int N) { return ((N + 3) & ~7) + 4; }
IW_HD constexpr int tc_nc(int N) { return (N + 3) & ~3; }
// Doubles of an operator that nothing follows in shared memory.  The fragments of its last column
// read rows up to 8 NT - 1, which is past the AP doubles of that column by up to 12 (N = 3, 4; the values
// go to rows past N, which no one uses).
IW_HD constexpr int tc_op_doubles(int N) { return tc_nc(N) * tc_ap(N) + 16; }
