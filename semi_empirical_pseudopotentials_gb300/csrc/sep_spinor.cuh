// sep_spinor.cuh -- the spin-orbit operator's launches (sep_spinor.cu) that the
// spinor path (sep_spinor_path.cu) uses.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "../../include/sep_gb300.h"

namespace sep {

// Digit planes of a kept operator's K, and the workspace of an apply on the
// tensor cores
struct VsoTensor {
  long natom = 0, nmax = 0;
  long mb = 0, nkc = 0, nb = 0;  // K's row blocks per atom, chunks, row blocks of products
  uint16_t* ka = nullptr;        // K's planes
  uint16_t* xb = nullptr;        // the products' planes
  int *ea = nullptr, *eb = nullptr;
  int4* top = nullptr;       // per row of K: its four largest values' columns
  ushort4* top_exp = nullptr;  // and their exponent fields
  uint16_t* xe = nullptr;    // exponent field of every product: [atom][spinor][point][8]
  double* sums = nullptr;    // natom mb 128 x (nb 128)
  int* err = nullptr;      // the contraction's status word, and one more
  static bool fits(long natom, long nmax);  // within the launches' limits
  // whether an apply takes less time so than by FP64 FMAs (pairs: sum of nl^2)
  static bool pays(long natom, long nmax, double pairs);
  long spinors() const;  // that one contraction takes: nb 128 / 12
  // sets the sizes and the parts of base; returns the bytes
  size_t carve(void* base, long natom, long nmax);
};

// K of every atom for spinor_vso_kept: natom x nmax x ld doubles, nmax the
// largest list, ld >= nmax
cudaError_t spinor_vso_kernel(long natom, long nnlc, const sep_nlc* nlc, const long* nl,
                              double sigma, long nmax, long ld, double* km, cudaStream_t st);
// the digit planes of that K; *bad (host): some value is not finite, and the
// planes mean nothing.  Waits for st.
cudaError_t spinor_vso_planes(const VsoTensor& v, const long* nl, const double* km, long ld,
                              int* bad, cudaStream_t st);
// The Gaussian form on nsp spinors (4 ngrid doubles apart) into psinl with the
// operator's K, on st: by FP64 FMAs (tensor null) or on the tensor cores.  off,
// idx: the list points of each grid point (k_vso_gather); contrib: 4 natom nmax
// doubles per spinor.  1 <= nsp <= 65535, natom, nmax >= 1.
cudaError_t spinor_vso_kept(const double* psi, long ngrid, long nsp, long natom, long nnlc,
                            const sep_nlc* nlc, const long* nl, double sigma, double dv,
                            const double* km, long nmax, long ld, const VsoTensor* tensor,
                            const int* off, const int* idx, double* contrib, double* psinl,
                            cudaStream_t st);
// Vso on nsp spinors (4 ngrid doubles apart) into psinl (zeroed first), on st,
// K formed in place; the arguments are already checked.  nsp <= 65535.
cudaError_t spinor_vso_launch(const double* psi, long ngrid, long nsp, long natom, long nnlc,
                              const sep_nlc* nlc, const long* nl, double sigma, double dv,
                              int flagkb, const double* elkb, double* psinl, cudaStream_t st);

}  // namespace sep
