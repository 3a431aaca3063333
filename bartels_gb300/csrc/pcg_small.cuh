// Block-Jacobi PCG of a small system as one thread-block cluster launch per
// inner solve (pcg_small.cu).
#pragma once

#include "internal.cuh"
#include "pcg_common.cuh"

namespace bartels {

constexpr int kSmallMaxN = 24576;  // unknowns: the direction (4 B each) fits shared memory beside the rest

// A scalar-CSR system on the host's side of the decision: row pointers on the
// host, everything else on the device.
struct PcgSmall {
  int n = 0, groups = 0, rows = 0, jcap = 0, smem = 0;  // groups of 32 rows; rows per CTA; staged entries per row
  int64_t entries = 0;                       // padded entries of all groups
  int *off = nullptr;                        // groups + 1, in entries / 32
  float *val = nullptr;                      // entries, [group][j][lane]
  unsigned short *col = nullptr;
};

// Whether the context's device can host the cluster (asked once per context, which
// also sets the kernel's attributes there; BARTELS_PCG_SMALL=0: no). Before pcg_small_run.
bool pcg_small_hosted(bartels_ctx ctx);
// Whether the system (row lengths len(i), i < n) runs as a cluster launch; fills
// the sizes and the group offsets (host).
bool pcg_small_plan(int n, const int *row_ptr, PcgSmall &s, std::vector<int> &off);
size_t pcg_small_bytes(const PcgSmall &s);
// Lay out the buffers in `base` (pcg_small_bytes long) and copy the matrix into
// them. rp / ci / val: device; rows of pinned vertices (3 rows each) become empty.
int pcg_small_fill(bartels_ctx ctx, PcgSmall &s, char *base, const std::vector<int> &off, const int *rp, const int *ci,
                   const float *val, const unsigned char *pinned);
// One inner solve: as k_pcg_init followed by the PCG loop until the state is done
// (done = 1), or until one of its sums leaves the range of float pairs (done =
// kSmallRange): the iterate is then of no use and the general loop has to take over.
enum { kSmallRange = 2 };
int pcg_small_run(bartels_ctx ctx, const PcgSmall &s, const float *rres, const float *minv, float *x, float *p,
                  PcgState *st, double inner_rel2, double abs_tol2, int max_it, int cont);

}  // namespace bartels
