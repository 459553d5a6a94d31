// The autotuner's choice of candidates (test infrastructure, never part of the
// library).
#include "../../cadise_gb300/csrc/internal.h"

extern "C" {

int tn_kernels(int traversal, int persistent) { return cg::traversal_kernels(traversal, persistent != 0); }

int tn_skips(int pass, const cgpu_tuning* t, const cgpu_tuning* best, int closest, int any) {
    return cg::autotune_skips(pass, *t, *best, closest, any);
}

}  // extern "C"
