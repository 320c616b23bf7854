// Registers that fit one block's shared memory: one launch evaluates a sample's whole circuit.
//
// A block owns one sample.  It copies the gate records and the sample's matrices into shared memory,
// runs the gates on the state there (a thread per amplitude pair, one barrier per gate), and for a
// gradient applies the Hamiltonians and runs the adjoint sweep on psi and every lambda in the same
// launch, down to the parameters.  Nothing but the results is written (and the states before gates that are not known to be
// unitary, which the sweep reads back).
//
// Why a kernel of its own: the tile kernels hold 2^RB amplitudes in each thread of at least one warp, so
// the smallest registers ran one kernel per gate (a 6-qubit classifier's training step on 32 samples: 310
// launches), and those of a single tile ran one block's serial chain of 16 to 32 amplitudes
// per thread in several launches.  Here a gate costs a shared-memory round trip of one pair per thread
// and a barrier, which is what bounds it: latency, not throughput.  So a complex64 gradient runs in FP64 here
// (10 qubits, 4 Hamiltonians, one sample: 298 us against 277), its caller's states converted on the way in.
#include <cuda_runtime.h>

#include <algorithm>

#include "regmath.cuh"
#include "small.h"

namespace mqb {

namespace {

using reg::cconj;
using reg::cmadd;
using reg::cmul;
using reg::redot;
using reg::warp_sum;

constexpr int kSmallThreads = 512;

size_t up16(size_t x) { return (x + 15) & ~size_t(15); }
__device__ __forceinline__ size_t dup16(size_t x) { return (x + 15) & ~size_t(15); }

__device__ __forceinline__ unsigned ins0(unsigned x, int b) {
    const unsigned lo = x & ((1u << b) - 1u);
    return ((x >> b) << (b + 1)) | lo;
}

// Index of group g's first amplitude (target bits 0) of a gate on one or two targets.
__device__ __forceinline__ unsigned group_base(const SmallOp &op, unsigned g) {
    if (op.m == 1) return ins0(g, op.t0);
    const int lo = min(op.t0, op.t1), hi = max(op.t0, op.t1);
    return ins0(ins0(g, lo), hi);
}

// One gate on the amplitudes x[0 .. 2^m) of a group (adjoint: its conjugate transpose).
template <typename V, bool ADJ>
__device__ __forceinline__ void gate1(const SmallOp &op, const V *M, V &a, V &b) {
    if (op.kind == KIND_DIAG) {
        a = cmul(a, ADJ ? cconj(M[0]) : M[0]);
        b = cmul(b, ADJ ? cconj(M[1]) : M[1]);
    } else if (op.sub == SUB_SWAP) {
        const V t = a;
        a = b;
        b = t;
    } else {
        const V m00 = ADJ ? cconj(M[0]) : M[0], m01 = ADJ ? cconj(M[2]) : M[1];
        const V m10 = ADJ ? cconj(M[1]) : M[2], m11 = ADJ ? cconj(M[3]) : M[3];
        const V na = cmadd(m00, a, cmul(m01, b));
        b = cmadd(m10, a, cmul(m11, b));
        a = na;
    }
}

template <typename V, bool ADJ>
__device__ __forceinline__ void gate2(const SmallOp &op, const V *M, V (&x)[4]) {
    if (op.kind == KIND_DIAG) {
#pragma unroll
        for (int r = 0; r < 4; ++r) x[r] = cmul(x[r], ADJ ? cconj(M[r]) : M[r]);
        return;
    }
    V y[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        V s = cmul(ADJ ? cconj(M[r]) : M[r * 4], x[0]);
#pragma unroll
        for (int c = 1; c < 4; ++c) s = cmadd(ADJ ? cconj(M[c * 4 + r]) : M[r * 4 + c], x[c], s);
        y[r] = s;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) x[r] = y[r];
}

template <typename V, typename W>
__device__ __forceinline__ V as(W a) {
    V r;
    r.x = a.x;
    r.y = a.y;
    return r;
}

template <typename R, typename S>
__global__ void __launch_bounds__(kSmallThreads) small_kernel(const SmallArgs<R, S> a) {
    using V = cplx<R>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int n = a.n, T = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = T >> 5;
    const unsigned dim = 1u << n;
    const int NH = a.n_hams;
    const int64_t b = blockIdx.x;
    V *psi = reinterpret_cast<V *>(smem);
    V *lam = psi + dim;
    V *mt = lam + size_t(NH) * dim;
    size_t o = dup16((size_t(1 + NH) * dim + a.mats_stride + a.n_pool) * sizeof(V));
    SmallOp *sops = reinterpret_cast<SmallOp *>(smem + o);
    o = dup16(o + size_t(a.n_ops) * sizeof(SmallOp));
    double *slots = reinterpret_cast<double *>(smem + o);   // [n_slots][NH]
    double *red = slots + size_t(a.n_slots) * NH;           // [2][12][warps]: partials of one gate, in turn
    {
        const int words = int(sizeof(SmallOp) / 4) * a.n_ops;
        const int32_t *src = reinterpret_cast<const int32_t *>(a.ops);
        int32_t *dst = reinterpret_cast<int32_t *>(sops);
        for (int i = tid; i < words; i += T) dst[i] = src[i];
        const V *m = a.mats + b * a.mats_stride;
        for (int i = tid; i < int(a.mats_stride); i += T) mt[i] = m[i];
        for (int i = tid; i < a.n_pool; i += T) mt[a.mats_stride + i] = a.cpool[i];
        for (int i = tid; i < a.n_slots * NH; i += T) slots[i] = 0;
        for (unsigned i = tid; i < dim; i += T) {
            V v;
            v.x = i == 0;
            v.y = 0;
            psi[i] = a.src ? as<V>(a.src[b * a.src_stride + i]) : v;
        }
    }
    __syncthreads();
    // sum of a value over the block, valid in thread 0; uses red[] (barriers inside)
    auto block_sum = [&](double x) {
        x = warp_sum(x);
        __syncthreads();
        if (lane == 0) red[warp] = x;
        __syncthreads();
        double s = 0;
        if (tid == 0)
            for (int w = 0; w < nw; ++w) s += red[w];
        return s;
    };
    int check = 0;
    auto norm_check = [&] {
        double x = 0;
        for (unsigned i = tid; i < dim; i += T) x += double(psi[i].x) * double(psi[i].x) + double(psi[i].y) * double(psi[i].y);
        x = block_sum(x);
        if (tid == 0) a.norms[2 * (check * a.batch + b)] = x;
        ++check;
        __syncthreads();
    };
    for (int k = 0; k < a.n_ops; ++k) {
        const SmallOp &op = sops[k];
        const V *M = mt + op.moff;
        if (op.save) {
            V *keep = a.saved + ((op.save - 1) * a.batch + b) * dim;
            for (unsigned i = tid; i < dim; i += T) keep[i] = psi[i];
            __syncthreads();
        }
        if (op.m == 1) {
            const unsigned bit = 1u << op.t0;
            for (unsigned g = tid; g < dim / 2; g += T) {
                const unsigned i = group_base(op, g);
                if ((i & op.ctrl) != op.ctrl) continue;
                V x0 = psi[i], x1 = psi[i | bit];
                gate1<V, false>(op, M, x0, x1);
                psi[i] = x0;
                psi[i | bit] = x1;
            }
        } else {
            for (unsigned g = tid; g < dim / 4; g += T) {
                const unsigned i = group_base(op, g);
                if ((i & op.ctrl) != op.ctrl) continue;
                const unsigned id[4] = {i, i | (1u << op.t0), i | (1u << op.t1), i | (1u << op.t0) | (1u << op.t1)};
                V x[4] = {psi[id[0]], psi[id[1]], psi[id[2]], psi[id[3]]};
                gate2<V, false>(op, M, x);
#pragma unroll
                for (int r = 0; r < 4; ++r) psi[id[r]] = x[r];
            }
        }
        __syncthreads();
        if (a.norms && (op.check & 1)) norm_check();
    }
    if (a.dst)
        for (unsigned i = tid; i < dim; i += T) a.dst[b * dim + i] = as<cplx<S>>(psi[i]);
    if (NH == 0) return;
    // lambda_h = H_h psi and f_h = <psi|lambda_h>, sums in FP64
    for (int h = 0; h < NH; ++h) {
        V *lh = lam + size_t(h) * dim;
        if (a.lam_in) {
            for (unsigned i = tid; i < dim; i += T) lh[i] = as<V>(a.lam_in[b * a.lam_stride + i]);
            continue;
        }
        const SmallHam &H = a.ham[h];
        double fr = 0, fi = 0;
        for (unsigned i = tid; i < dim; i += T) {
            double ar = 0, ai = 0;
            for (int c = 0; c < H.n_classes; ++c) {
                const HamClass &hc = H.classes[c];
                double wr = 0, wi = 0;
                for (int q = hc.term_begin; q < hc.term_begin + hc.term_count; ++q) {
                    const HamTerm &ht = H.terms[q];
                    const bool neg = __popc(i & unsigned(ht.my_mz)) & 1;
                    wr += neg ? -ht.cb_re : ht.cb_re;
                    wi += neg ? -ht.cb_im : ht.cb_im;
                }
                const V kv = psi[i ^ unsigned(hc.flip)];
                ar += wr * double(kv.x) - wi * double(kv.y);
                ai += wr * double(kv.y) + wi * double(kv.x);
            }
            const V bv = psi[i];
            fr += double(bv.x) * ar + double(bv.y) * ai;
            fi += double(bv.x) * ai - double(bv.y) * ar;
            V r;
            r.x = ar;
            r.y = ai;
            lh[i] = r;
        }
        fr = block_sum(fr);
        fi = block_sum(fi);
        if (tid == 0) {
            a.f[2 * (b * NH + h)] = fr;
            a.f[2 * (b * NH + h) + 1] = fi;
        }
    }
    __syncthreads();
    // adjoint sweep: psi <- U^dag psi (or the kept state), slot += Re <lambda| dU |psi>, lambda <- U^dag lambda
    int par = 0;
    for (int k = a.n_ops - 1; k >= 0; --k) {
        const SmallOp &op = sops[k];
        const V *M = mt + op.moff;
        const int G = op.grad_mask;
        if (op.save) {
            const V *keep = a.saved + ((op.save - 1) * a.batch + b) * dim;
            for (unsigned i = tid; i < dim; i += T) psi[i] = keep[i];
            __syncthreads();
        }
        double acc[3][kSmallMaxHams];
#pragma unroll
        for (int an = 0; an < 3; ++an)
#pragma unroll
            for (int h = 0; h < kSmallMaxHams; ++h) acc[an][h] = 0;
        if (op.m == 1) {
            const unsigned bit = 1u << op.t0;
            for (unsigned g = tid; g < dim / 2; g += T) {
                const unsigned i = group_base(op, g);
                if ((i & op.ctrl) != op.ctrl) continue;
                V x0 = psi[i], x1 = psi[i | bit];
                if (!op.save) gate1<V, true>(op, M, x0, x1);
                psi[i] = x0;
                psi[i | bit] = x1;
#pragma unroll
                for (int h = 0; h < kSmallMaxHams; ++h) {
                    if (h >= NH) break;
                    V *lh = lam + size_t(h) * dim;
                    V l0 = lh[i], l1 = lh[i | bit];
#pragma unroll
                    for (int an = 0; an < 3; ++an) {
                        if (!((G >> an) & 1)) continue;
                        const V *D = mt + op.doff + an * op.mat_size;
                        V y0, y1;
                        if (op.kind == KIND_DIAG) {
                            y0 = cmul(D[0], x0);
                            y1 = cmul(D[1], x1);
                        } else {
                            y0 = cmadd(D[0], x0, cmul(D[1], x1));
                            y1 = cmadd(D[2], x0, cmul(D[3], x1));
                        }
                        acc[an][h] += double(redot(l0, y0)) + double(redot(l1, y1));
                    }
                    gate1<V, true>(op, M, l0, l1);
                    lh[i] = l0;
                    lh[i | bit] = l1;
                }
            }
        } else {
            for (unsigned g = tid; g < dim / 4; g += T) {
                const unsigned i = group_base(op, g);
                if ((i & op.ctrl) != op.ctrl) continue;
                const unsigned id[4] = {i, i | (1u << op.t0), i | (1u << op.t1), i | (1u << op.t0) | (1u << op.t1)};
                V x[4] = {psi[id[0]], psi[id[1]], psi[id[2]], psi[id[3]]};
                if (!op.save) gate2<V, true>(op, M, x);
#pragma unroll
                for (int r = 0; r < 4; ++r) psi[id[r]] = x[r];
#pragma unroll
                for (int h = 0; h < kSmallMaxHams; ++h) {
                    if (h >= NH) break;
                    V *lh = lam + size_t(h) * dim;
                    V l[4] = {lh[id[0]], lh[id[1]], lh[id[2]], lh[id[3]]};
#pragma unroll
                    for (int an = 0; an < 3; ++an) {
                        if (!((G >> an) & 1)) continue;
                        const V *D = mt + op.doff + an * op.mat_size;
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            V y;
                            if (op.kind == KIND_DIAG) {
                                y = cmul(D[r], x[r]);
                            } else {
                                y = cmul(D[r * 4], x[0]);
#pragma unroll
                                for (int c = 1; c < 4; ++c) y = cmadd(D[r * 4 + c], x[c], y);
                            }
                            acc[an][h] += double(redot(l[r], y));
                        }
                    }
                    gate2<V, true>(op, M, l);
#pragma unroll
                    for (int r = 0; r < 4; ++r) lh[id[r]] = l[r];
                }
            }
        }
        if (G) {
            double *rp = red + size_t(par) * 12 * nw;
#pragma unroll
            for (int an = 0; an < 3; ++an) {
                if (!((G >> an) & 1)) continue;
#pragma unroll
                for (int h = 0; h < kSmallMaxHams; ++h) {
                    if (h >= NH) break;
                    const double x = warp_sum(acc[an][h]);
                    if (lane == 0) rp[(an * kSmallMaxHams + h) * nw + warp] = x;
                }
            }
        }
        __syncthreads();
        // the next gate writes the other half of red, and the one after it follows two barriers later
        if (G && tid < 3 * kSmallMaxHams) {
            const int an = tid / kSmallMaxHams, h = tid % kSmallMaxHams;
            if (((G >> an) & 1) && h < NH) {
                const double *rp = red + (size_t(par) * 12 + tid) * nw;
                double s = 0;
                for (int w = 0; w < nw; ++w) s += rp[w];
                slots[(op.slot0 + __popc(G & ((1 << an) - 1))) * NH + h] = s;
            }
        }
        if (G) par ^= 1;
        const int q = op.check >> 1;
        if (a.norms && q && !(a.ckpt_stride > 0 && q % a.ckpt_stride == 0)) {
            __syncthreads();
            norm_check();
        }
    }
    __syncthreads();
    for (int w = tid; w < a.n_params * NH; w += T) {
        const int h = w / a.n_params, p = w % a.n_params;
        double s = 0;
        for (int e = a.csr_ptr[p]; e < a.csr_ptr[p + 1]; ++e) s += a.csr_coeff[e] * slots[a.csr_slot[e] * NH + h];
        a.grad[b * int64_t(NH) * a.n_params + w] = a.scale * s;
    }
}

int small_threads(int n) { return std::min(kSmallThreads, std::max(32, 1 << (n - 1))); }

}  // namespace

size_t small_smem(int n, int elem_bytes, int n_hams, int n_ops, int64_t table_entries, int n_slots) {
    if (n_hams > kSmallMaxHams) return 0;
    size_t s = up16(((size_t(1 + n_hams) << n) + size_t(table_entries)) * size_t(elem_bytes));
    s = up16(s + size_t(n_ops) * sizeof(SmallOp));
    s += size_t(n_slots) * n_hams * sizeof(double);
    s += size_t(2 * 12) * (kSmallThreads / 32) * sizeof(double);
    return s <= (size_t(200) << 10) ? s : 0;
}

template <typename R, typename S>
cudaError_t launch_small(const SmallArgs<R, S> &a, size_t smem, cudaStream_t s) {
    cudaError_t e = allow_smem<small_kernel<R, S>>();
    if (e != cudaSuccess) return e;
    small_kernel<R, S><<<unsigned(a.batch), small_threads(a.n), smem, s>>>(a);
    return cudaGetLastError();
}

template cudaError_t launch_small<float, float>(const SmallArgs<float, float> &, size_t, cudaStream_t);
template cudaError_t launch_small<double, float>(const SmallArgs<double, float> &, size_t, cudaStream_t);
template cudaError_t launch_small<double, double>(const SmallArgs<double, double> &, size_t, cudaStream_t);

}  // namespace mqb
