// lzsite.h -- the whole Lanczos solve of one site in one launch (FP64 operator).
#pragma once
#include "contract.h"
#include "lanczos.h"

namespace tnb {

constexpr int LZ_SITE_UNAVAILABLE = -1;

// Lowest eigenpair of Heff (terms: build_terms(W, left to right) on the device)
// from the start vector x, which the Ritz vector replaces: the solve of
// lanczos_solve with this operator, as one launch on the context stream.  The
// summary is copied to host_out (pinned) on the stream; nothing waits.
// Returns LZ_SITE_UNAVAILABLE (nothing enqueued) for shapes outside the
// kernel's range, which lanczos_solve / lanczos_solve_async then take.
int lanczos_site(Ctx& c, const ContractShape& s, const WTermDev* terms, int nterms, const double* F, const double* G,
                 double* x, int m, int maxRestarts, double tol, double tol_rel, LzSummary* host_out);

}  // namespace tnb
