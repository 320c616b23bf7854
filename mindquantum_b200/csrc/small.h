// Registers small enough for one block's shared memory: a whole evaluation in one launch (small.cu).
#ifndef MQB_SMALL_H_
#define MQB_SMALL_H_

#include "kernels.cuh"

namespace mqb {

constexpr int kSmallMaxHams = 4;

// One gate of the small-register kernel, in execution order.
struct SmallOp {
    int16_t kind, m, sub;        // OpKind, targets, DenseSub
    int16_t save;                // gradient: 1 + the place of the state before the gate, kept because its conjugate transpose
                                 // does not undo it (0: it does)
    int32_t t0, t1;              // target qubits (matrix bits 0 and 1)
    uint32_t ctrl;               // control mask
    int32_t moff;                // M in the block's matrix table: the per-sample block, then the constant pool
    int32_t doff;                // dM_a at doff + a * mat_size
    int32_t mat_size;
    int32_t grad_mask, slot0;    // gradient angles (0: none) and the slot of the first one
    int32_t check;               // bit 0: norm check after the gate; bits 1..: pass q whose start the gate is,
                                 // for the check of the state before it in the backward sweep (0: none)
};

struct SmallHam {
    const HamClass *classes;
    const HamTerm *terms;
    int n_classes;
};

// R: the arithmetic; S: the caller's states.
template <typename R, typename S = R>
struct SmallArgs {
    int n, n_ops;
    const SmallOp *ops;
    const cplx<R> *mats;         // per-sample matrices
    int64_t mats_stride;
    const cplx<R> *cpool;
    int n_pool;
    const cplx<S> *src;          // nullptr: |0...0>
    int64_t src_stride;
    cplx<S> *dst;                // apply: the final state; gradient: nullptr
    int64_t batch;
    // gradient
    int n_hams;
    SmallHam ham[kSmallMaxHams];
    const cplx<S> *lam_in;       // lambda from the caller instead of the Hamiltonians (n_hams = 1)
    int64_t lam_stride;
    double *f;                   // [batch][n_hams][2]
    double *grad;                // [batch][n_hams][n_params]
    int n_params, n_slots;
    const int32_t *csr_ptr, *csr_slot;
    const double *csr_coeff;
    double scale;
    double *norms;               // [check][batch][2], or nullptr (no checks)
    cplx<R> *saved;              // [SmallOp::save - 1][batch][2^n]
    int ckpt_stride;             // the states the caller's layout counts as stored have no backward check
};

// Shared memory of a block; 0 when the evaluation does not fit the kernel.
size_t small_smem(int n, int elem_bytes, int n_hams, int n_ops, int64_t table_entries, int n_slots);
template <typename R, typename S>
cudaError_t launch_small(const SmallArgs<R, S> &a, size_t smem, cudaStream_t s);

}  // namespace mqb

#endif
