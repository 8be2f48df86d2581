// Internal interface of the MSM pipeline (msm.cu) and the curve helpers kernels (curve.cu).
#pragma once
#include "ctx.hpp"
#include "ec.cuh"

namespace zk {

typedef MsmStatsPod MsmStats;

// scan.cu
uint64_t scan_scratch_elems(uint64_t n);
int exclusive_scan_u32(uint32_t* data, uint64_t n, uint32_t* scratch, bool write_total, cudaStream_t s);

// What the first pass over the scalars of an MSM finds.  A caller that runs several MSMs over the
// same scalars (C and the d_x rows of a KZH commit) passes one of these to each call: the first
// fills it, the others skip the pass.  `compact` lives in the context's compact scratch and stays
// valid until another MSM on the context analyses different scalars.
struct MsmPrep {
  bool valid = false;
  const Fr* scalars = nullptr;
  uint64_t total = 0;
  unsigned max_bits = 0;
  uint32_t max_mag = 0;            // exact largest magnitude when max_bits <= 32
  uint32_t max_span = 0;           // then also the largest of v and -v - 1
  uint64_t nonzero = 0;            // scalars that are not zero
  const int32_t* compact = nullptr;  // signed 32-bit form of every scalar, or NULL when some do not fit
};

// out_dev[row] = sum_i scalars[row * n + i] * bases[gather ? gather[i] : i] for row < rows.
// All pointers are device pointers; scalars are Montgomery-form Fr.  Uses the context's aux
// scratch; returns 0 or a negative status.
int msm_run(zk_ctx* ctx, const Affine* bases, const uint32_t* gather, const Fr* scalars, uint64_t n, uint32_t rows,
            Jacobian* out_dev, MsmStats* stats, MsmPrep* prep = nullptr);

// The same for one row, C of a commitment, and beside it the commitment's rows over the same scalars where that is of use (done).
struct MsmRowsBeside {
  const Affine* bases;
  uint64_t n;     // a row
  uint32_t rows;
  Jacobian* out_dev;
  bool done = false;
};
int msm_run_commit(zk_ctx* ctx, const Affine* bases, const Fr* scalars, uint64_t n, Jacobian* out_dev, MsmStats* stats, MsmPrep* prep,
                   MsmRowsBeside* rows);

int msm_run_rows(zk_ctx* ctx, const Affine* bases, const uint32_t* gather, const uint32_t* row_ids, const Fr* scalars,
                 uint64_t n, uint32_t rows, Jacobian* out_dev, MsmStats* stats, MsmPrep* prep = nullptr);

// Commitment of a selection polynomial (all listed entries one) without the digit / sort / bucket passes: msm.cu.
int msm_select_sums(zk_ctx* ctx, const Affine* full, const Affine* mid, const uint32_t* idx_dev, const uint32_t* bad, uint32_t n,
                    uint32_t low_bits, uint32_t rows, Jacobian* out_dev, void* scratch);

// ---- Host-side inversion (0 maps to 0): the division steps of inverse(), 1.6 us of a CPU core.
template <class P>
inline Fp<P> inverse_host(const Fp<P>& a) {
  return inverse(a);
}

// CurveGroup::into_affine of one point on the host: the point is read back anyway, and a launch for one thread's inversion
// (some 20 us) costs more than the 2 us it takes here.
inline Affine jacobian_to_affine_host(const Jacobian& j) {
  Affine a;
  if (j.z.is_zero()) {
    a.x = Fq::zero();
    a.y = Fq::zero();
  } else {
    const Fq zi = inverse_host(j.z), zi2 = sqr(zi);
    a.x = mul(j.x, zi2);
    a.y = mul(j.y, mul(zi2, zi));
  }
  return a;
}

}  // namespace zk
