// Batched FP64 generalized eigensolver of the submatrix method (sm_eig.cu).
#pragma once

#include <memory>
#include <vector>

#include "common.cuh"

namespace ptb {

// Largest order whose tridiagonalisation may run on one CTA (its vectors fill the
// shared memory); larger ones take a thread-block cluster.  Problems above it go up and
// start before the rest of a batch does.
constexpr int kEigBatchMax = 800;
// Largest submatrix the library's eigensolver takes at all: the tridiagonalisation of
// the largest orders keeps two vectors of this length in shared memory.
constexpr int kEigLargeMax = 12032;
// Batches that may be on their way beside the context's stream at a time.
constexpr int kEigSlots = 4;

// One submatrix as the host plan describes it.
struct EigProbHost {
    int k;          // submatrix index
    int m;          // dimension
    int nown;       // owned columns
    int64_t moff;   // offset of its row map in the maps array
    int64_t eoff;   // offset of its eigenpairs in the flat e / fe arrays
    int64_t o0;     // offset of its owned columns in the owned-column list
    int64_t gbase = 0;   // its H / S element (i, j) at gbase + map(i) + map(j) gld
    int64_t gld = -1;    // -1: the system's ndim
    int mode = 0;        // 0: eigenvalues, fe and owned rows (submatrix method); 2: density P = 2 U_occ U_occ^T
    int nocc = 0;        // mode 2: occupied (lowest) eigenvectors
};

struct EigBatch;

// Launches (on the context's stream, no host synchronisation) the gather,
// Cholesky, reduction, tridiagonalisation, divide and conquer, and the owned
// rows of U and S U with the (e, fe) pairs into d_e / d_fe at each problem's
// eoff.  Returns null for an empty list.  eig_batch_check waits for the stream
// and raises ENOTSPD (an overlap block not positive definite) or EITER (a
// leaf's QL iteration did not converge).
std::shared_ptr<EigBatch> eig_batch_launch(ptbgpu_ctx* c, int64_t n, const double* H, const double* S,
                                           const std::vector<EigProbHost>& probs, const int* d_maps,
                                           const int* d_own_cols, const int* d_ipos, double* d_e, double* d_fe,
                                           int prl, double* flops, int slot = -1);
// With a slot (0 .. kEigSlots - 1) the batch runs on a stream beside the context's, after
// the earlier ones there; the context's stream waits for it here.
void eig_batch_join(ptbgpu_ctx* c, EigBatch& eb);
void eig_batch_check(ptbgpu_ctx* c, EigBatch& eb);

// The owned columns of P_k = U occ U^T at mu for every prepared problem,
// written into the packed result (rows map(i) <= c of column c), or with
// dPdense non-null as m x nown column-major blocks, one after another.
void eig_batch_final(ptbgpu_ctx* c, EigBatch& eb, double mu, const int* d_maps,
                     const int* d_own_cols, double* dP, double* dPdense = nullptr);

// All eigenpairs of a dense problem on the device with the same solver on the
// whole GPU, in the same stages: H U = S U diag(w) (S null: the standard
// problem), H and S full symmetric (n x n, ld n; only the lower triangles are
// read), w ascending, U column-major with U^T S U = I.  Orders up to
// kEigLargeMax.
void eig_full(ptbgpu_ctx* c, int64_t n, const double* H, const double* S, double* w, double* U);
// The same with LAPACK's dsyevd / dsygvd argument convention ('V', upper
// triangles read): A (and B) n x n, ld n; A is overwritten by the eigenvectors.
void eig_full_upper(ptbgpu_ctx* c, int64_t n, double* A, double* B, double* w);

// In-place inverse of the lower triangle of A (n x n, column-major, leading dimension
// ld); of the strict upper triangle only the 64 x 64 diagonal blocks' parts are touched
// (zeroed).  W: n^2 / 4 doubles of scratch at most.
void tri_inverse(ptbgpu_ctx* c, int64_t n, int64_t ld, double* A, double* W);
// With Li from it (ld n) and T as n x n scratch: H <- Li H Li^T (both triangles), and
// X <- Li^T X Li (X symmetric; the upper triangle of the result).
void tri_congruence(ptbgpu_ctx* c, int64_t n, const double* Li, double* H, double* T);
void tri_back(ptbgpu_ctx* c, int64_t n, const double* Li, double* X, double* T);

// The density step of many independent systems as one batch of the
// eigensolver (ptbgpu_eig_density_batch): Hpk / Spk / Ppk host packed arrays
// per system, P_k = 2 sum_{i < nel_k/2} u_i u_i^T of H_k U = S_k U e after the
// filter; stats per system (may be null).
void eig_density_batch(ptbgpu_ctx* c, int64_t ninst, const int64_t* ndim, const int64_t* nel,
                       const double* const* Hpk, const double* const* Spk, double* const* Ppk, double filter,
                       int prl, ptbgpu_stats* st);

// Kernel-level entry of ptbgpu_sygv_batched (dense host problems).
void sygv_batched_entry(ptbgpu_ctx* c, int64_t np, const int64_t* dims, const double* H, const double* S,
                        const int64_t* nown, const int64_t* owned, double mu, double* e, double* fe, double* Pcols);

}  // namespace ptb
