// Summed G tables of a periodic cluster (lattice.cu).
#pragma once

#include <cuda_runtime.h>

namespace gb {

// Tables per ordered pair that launch_lattice_sums writes: table c of pair (i, j) at entries
// c (2 lmax + 2)^2 + p^2 + p + mu of block (i, j) of the dense output (row-major entries of
// the B x B block); their sum is the pair's G.
int lattice_chunks(int N, int lmax, int ncell);

int launch_lattice_sums(int N, int lmax, const double* pos, double k, const double* cells, int ncell, double kx, double ky,
                        double kz, const double* neg_ratio, double2* out, long long ld, cudaStream_t stream);

}   // namespace gb
