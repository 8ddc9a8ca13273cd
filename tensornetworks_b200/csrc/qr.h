// qr.h -- Householder QR and one-sided Jacobi SVD on the device.
#pragma once
#include "tn_internal.h"

namespace tnb {

// In-place blocked Householder QR of the dense column-major W (m x n, ld m).
// Writes Q (m x k, ld ldq) and R (k x n, ld ldr) when the pointers are non-null.
int qr_dense(Ctx& c, int m, int n, double* W, double* Qout, int ldq, double* Rout, int ldr);

// The QR of A (element (i, c) at A[i ars + c acs], left as it is) by thread-block clusters in one
// launch: Q (m x k) and R (k x n, zeros written below the diagonal), each with
// its own strides, when the pointers are non-null.  The same reflectors as qr_dense (dlarfg's signs),
// sums in another order.  colmap (device, may be null): column c of the matrix is column colmap[c] of A.  QR_UNAVAILABLE (nothing enqueued) for m > 1536, for more column
// blocks of 32 than clusters fit on the device, and when the context's settings
// ask for another path.
constexpr int QR_UNAVAILABLE = -1;
int qr_cluster(Ctx& c, int m, int n, const double* A, long long ars, long long acs, double* Q, long long qrs,
               long long qcs, double* R, long long rrs, long long rcs, const int* colmap = nullptr);
// Waits for the stream after qr_cluster: TN_OK, the error of an expired wait, or QR_UNAVAILABLE when a column's
// remainder had a norm outside 2^-500 .. 2^500 (zero is inside), whose reflector the kernel does not form; the
// factors are then void, A is as it was.
int qr_cluster_status(Ctx& c);

// Reads (and clears) the context's sticky device error word, raised when a
// bounded wait between CTAs expired; waits for the device.
int check_device_error(Ctx& c);
// The same by a copy on the context stream, which it then waits for.
int check_device_error_on_stream(Ctx& c);
// The error word, and the QR's range word after it, allocated and zero (before the first kernel that may raise them).
int ensure_device_error_word(Ctx& c);

// One job of the batched one-sided Jacobi SVD (one cluster or CTA per job).  W is the
// tall (m >= n) working copy, overwritten.  With vectors: U (m x n, ldu),
// Vt (n x n, ldvt) and a scratch V (n x n, ld n).  s (n) is always written.
struct SvdJob {
    double* W;
    int m, n;
    double* V;
    double* U;
    int ldu;
    double* Vt;
    int ldvt;
    double* s;
    int* sweeps;  // may be null
    const int* perm = nullptr;  // set by svd_batched: W is R^T and V is Q of the permuted matrix
};

int svd_batched(Ctx& c, const std::vector<SvdJob>& jobs, bool vectors);

}  // namespace tnb
