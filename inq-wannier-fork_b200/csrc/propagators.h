// Launchers of the Crank-Nicolson solver kernels (propagators.cu).
#pragma once

#include <cstddef>

namespace inqb {

// partial [blocks][4][M] (at most sd_partial_doubles(M) values): per block of points the sums
// over p of (|hsd|^2, Re conj(r) hsd, Im conj(r) hsd, |r|^2), FP64, without dV
size_t sd_partial_doubles(int M);
int launch_sd_sums(int precision, const void* r, const void* hsd, long ld, int M, long N, double* partial,
                   void* stream);
// phi += lambda_m r with the steepest-descent step length from the partials (dV applied
// here); normres[m] = dV sum_p |r|^2
int launch_sd_update(int precision, void* phi, long ldp, const void* r, long ldr, int M, long N, const double* partial,
                     double dV, double* normres, void* stream);

}  // namespace inqb
