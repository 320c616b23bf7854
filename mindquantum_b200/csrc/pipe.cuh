// Asynchronous tile movement of the generated pass kernels (sm_100a): TMA tensor copies between
// global memory and shared-memory tile buffers, completed on mbarriers, and the bounded waits
// around them.  Compiled by NVRTC together with the generated kernels, so only built-in types
// and inline PTX are used.
//
// No copy here uses cluster multicast: every tensor map covers this GPU's own memory and every
// copy lands in the issuing CTA's own shared memory.
#ifndef MQB_PIPE_CUH_
#define MQB_PIPE_CUH_

#include "jit_abi.h"
#include "regmath.cuh"

namespace mqb {
namespace pipe {

typedef unsigned long long u64;

// A CUtensorMap (128 opaque bytes, 64-byte aligned), passed to the kernels as a __grid_constant__.
struct __align__(64) TMap {
    u64 w[16];
};

__device__ __forceinline__ unsigned saddr(const void *p) {
    u64 a;
    asm("cvta.to.shared.u64 %0, %1;" : "=l"(a) : "l"(p));
    return static_cast<unsigned>(a);
}

__device__ __forceinline__ u64 now_ns() {
    u64 t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Limit of every wait on an mbarrier: far above any tile's load or compute time (microseconds),
// so only a broken pipeline reaches it; the kernel then reports MQB_DEV_ERR_TIMEOUT and returns.
constexpr u64 kWaitLimitNs = 2000000000ull;

__device__ __forceinline__ void mbar_init(u64 *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(u64 *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(u64 *bar) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(saddr(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_test(u64 *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(saddr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Wait for the phase of `parity` to complete; false when kWaitLimitNs passed first.
__device__ __forceinline__ bool mbar_wait(u64 *bar, unsigned parity) {
    if (mbar_test(bar, parity)) return true;
    const u64 t0 = now_ns();
    while (!mbar_test(bar, parity))
        if (now_ns() - t0 > kWaitLimitNs) return false;
    return true;
}

// Wait until a buffer's ticket names tile k (the tile whose copies were last started into it);
// false when kWaitLimitNs passed first.  A buffer's mbarrier tells phases apart by parity only, so
// a consumer may test it only once the buffer's previous tile has been handed over: the issuer
// writes the ticket after it has finished with that previous tile.
__device__ __forceinline__ bool wait_ticket(const volatile long long *slot, long long k) {
    if (*slot == k) return true;
    const u64 t0 = now_ns();
    while (*slot != k)
        if (now_ns() - t0 > kWaitLimitNs) return false;
    return true;
}

// Named barrier `id` (1 + consumer group; 0 is __syncthreads) among the n threads of a group.
__device__ __forceinline__ void consumers_sync(int id, int n) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// Named barrier `id` among the n threads of a consumer group, returning whether q holds on every
// one of them: a group takes every wait's outcome together, so no thread leaves the tile loop
// alone and none is left waiting at a later barrier.
__device__ __forceinline__ bool consumers_and(int id, int n, bool q) {
    unsigned r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n bar.red.and.pred p, %2, %3, q;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(r)
        : "r"(static_cast<unsigned>(q)), "r"(id), "r"(n)
        : "memory");
    return r != 0;
}

// The matrices of a pass's ops into shared memory, by the nt consumer threads (one warp per op).
template <typename V>
__device__ __forceinline__ void load_mtab(V *mtab, const JitMtab *mt, int n, const V *mb, const V *cpool, unsigned tid,
                                          unsigned nt) {
    const unsigned lane = tid & 31u, nw = nt >> 5;
    for (int k = static_cast<int>(tid >> 5); k < n; k += static_cast<int>(nw)) {
        const JitMtab e = mt[k];
        const V *src = (e.msrc_ps ? mb : cpool) + e.msrc;
        for (int i = static_cast<int>(lane); i < e.mcount; i += 32) mtab[e.moff + i] = src[i];
    }
}

__device__ __forceinline__ double2 wide(float2 a) { return make_double2(a.x, a.y); }
__device__ __forceinline__ double2 wide(double2 a) { return a; }

// The factor of a value of a run's register bits: in a forward pass as the sum of two complex64 numbers, so that the run
// loses nothing by its table; in the adjoint, whose result is less sensitive, rounded once.
struct alignas(16) Split {
    float2 hi, lo;
};
__device__ __forceinline__ float2 times(float2 a, const Split &t) {
    float2 r;
    r.x = fma(-a.y, t.hi.y, fma(a.x, t.hi.x, fma(-a.y, t.lo.y, a.x * t.lo.x)));
    r.y = fma(a.y, t.hi.x, fma(a.x, t.hi.y, fma(a.y, t.lo.x, a.x * t.lo.y)));
    return r;
}
__device__ __forceinline__ float2 times(float2 a, float2 t) { return reg::cmul(a, t); }
__device__ __forceinline__ void put_factor(Split &t, double2 p) {
    t.hi = make_float2(float(p.x), float(p.y));
    t.lo = make_float2(float(p.x - double(t.hi.x)), float(p.y - double(t.hi.y)));
}
__device__ __forceinline__ void put_factor(float2 &t, double2 p) { t = make_float2(float(p.x), float(-p.y)); }   // of U^dag

// A gate of a run: M at moff, its targets' places among the run's bits (-1: no such target), its controls.
struct RunGate {
    unsigned short moff;
    signed char p0, p1;
    unsigned char ctrl;
};
// An entry of a run's table: the product of n gates' entries for the bits idx.
struct RunEntry {
    unsigned short first;
    unsigned char n, idx;
};

// The tables of a pass's runs from its matrix table, by the nt threads of a group, the products in FP64.
template <typename T, typename V>
__device__ __forceinline__ void load_runs(T *runs, const V *mtab, const RunGate *gates, const RunEntry *entries, int n,
                                          unsigned tid, unsigned nt) {
    for (unsigned e = tid; e < unsigned(n); e += nt) {
        const RunEntry en = entries[e];
        double2 p = make_double2(1, 0);
        for (int k = 0; k < en.n; ++k) {
            const RunGate g = gates[en.first + k];
            if ((en.idx & g.ctrl) != g.ctrl) continue;
            const int r = (g.p0 < 0 ? 0 : en.idx >> g.p0 & 1) | (g.p1 < 0 ? 0 : (en.idx >> g.p1 & 1) << 1);
            p = reg::cmul(p, wide(mtab[g.moff + r]));
        }
        put_factor(runs[e], p);
    }
}

// Matrix entries (`src`: their places in the matrix table) as FP64, for the factors that each thread makes: reading them
// so costs a thread a load, where converting them takes two conversions per factor (MaxCut gradient on 26 vertices, p = 10: 26.9 ms
// with conversions, 26.2 so; on 30 vertices 500 and 489).
template <typename V>
__device__ __forceinline__ void load_wide(double2 *wt, const V *mtab, const unsigned short *src, int n, unsigned tid, unsigned nt) {
    for (unsigned e = tid; e < unsigned(n); e += nt) wt[e] = wide(mtab[src[e]]);
}

// One over the norm that rounding gave the uncontrolled gates of a pass, by the group's first warp after the matrix table
// is complete.  A complex64 rotation's c and s leave c^2 + s^2 off one by some 1e-8, the same for every
// amplitude, so over hundreds of gates the state's norm drifts by 1e-6 and takes the expectation and the
// gradients along; one factor per pass takes it out.
template <typename V>
__device__ __forceinline__ void pass_norm(double *ph, const V *mtab, const JitMtab *mt, int n, unsigned tid) {
    if (tid >= 32u) return;
    double p = 1;
    for (int k = static_cast<int>(tid); k < n; k += 32) {
        const JitMtab e = mt[k];
        if (e.norm == 0) continue;
        const int rows = e.norm < 0 ? -e.norm : e.norm, cnt = e.norm < 0 ? rows : rows * rows;
        const V *M = mtab + e.moff;
        double q = 0;   // mean square of what the gate multiplies amplitudes by
        for (int i = 0; i < cnt; ++i) q += double(M[i].x) * double(M[i].x) + double(M[i].y) * double(M[i].y);
        p *= 1.5 - 0.5 * (q / rows);   // 1 / sqrt(q) for q this close to one
    }
    for (int o = 16; o > 0; o >>= 1) p *= __shfl_xor_sync(0xffffffffu, p, o);
    if (tid == 0u) *ph = p;
}

// Gradient rows of a warp: shared scratch at `scr` holds N = 4 or 8 rows of 32 float partials, or 2 of double.
// row_put stores this lane's partial of row k; rows_flush_as adds the n rows over the lanes (in
// the partials' precision) and the sums to acc[0..n) in FP64.  The accesses are volatile asm without a
// memory clobber: they keep their order among themselves, and the compiler may move the gates' own
// shared-memory reads across them.
__device__ __forceinline__ void row_put(unsigned scr, int k, int lane, float x) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(scr + unsigned(k * 32 + lane) * 4u), "f"(x));
}
__device__ __forceinline__ void row_put(unsigned scr, int k, int lane, double x) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(scr + unsigned(k * 32 + lane) * 8u), "d"(x));
}
__device__ __forceinline__ float four(unsigned at) {
    float x, y, z, w;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x), "=f"(y), "=f"(z), "=f"(w) : "r"(at));
    return (x + y) + (z + w);
}
template <int N>
__device__ __forceinline__ void rows_sum(unsigned scr, int lane, float &s, int &row, bool &first) {
    constexpr int LR = 32 / N;   // lanes per row
    row = lane / LR;
    if (N == 8) {   // two 16-byte chunks per lane, in turned order on odd rows (distinct banks in a quarter-warp)
        const unsigned at = scr + unsigned(row * 128 + (lane & 3) * 16), turn = (row & 1) ? 64u : 0u;
        s = four(at + turn) + four(at + (64u ^ turn));
    } else {
        s = four(scr + unsigned(lane) * 16u);
    }
#pragma unroll
    for (int o = LR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    first = lane % LR == 0;
}
template <int N>
__device__ __forceinline__ void rows_sum(unsigned scr, int lane, double &s, int &row, bool &first) {
    double x, y;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "r"(scr + unsigned(lane) * 16u));
    s = x + y;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    row = lane >> 4;
    first = (lane & 15) == 0;
}
__device__ __forceinline__ void warp_order() { asm volatile("bar.warp.sync 0xffffffff;"); }
template <typename R, int N>
__device__ __forceinline__ void rows_flush_as(unsigned scr, double *acc, int n, int lane) {
    R s;
    int row;
    bool first;
    warp_order();
    rows_sum<N>(scr, lane, s, row, first);
    warp_order();
    if (first && row < n) acc[row] += double(s);
}

// Make this thread's generic-proxy writes to shared memory visible to the TMA (async proxy).
__device__ __forceinline__ void fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Tensor copy global -> shared of one box at coordinates c[0..nd), completing on `bar`.
__device__ __forceinline__ void tma_load(void *dst, const TMap *m, int nd, const int *c, u64 *bar) {
    const unsigned d = saddr(dst), b = saddr(bar);
    const u64 mp = reinterpret_cast<u64>(m);
    switch (nd) {
        case 1:
            asm volatile(
                "cp.async.bulk.tensor.1d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2}], [%3];" ::"r"(d),
                "l"(mp), "r"(c[0]), "r"(b)
                : "memory");
            break;
        case 2:
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(d),
                "l"(mp), "r"(c[0]), "r"(c[1]), "r"(b)
                : "memory");
            break;
        case 3:
            asm volatile(
                "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(d),
                "l"(mp), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(b)
                : "memory");
            break;
        case 4:
            asm volatile(
                "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(d),
                "l"(mp), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(b)
                : "memory");
            break;
        default:
            asm volatile(
                "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(d),
                "l"(mp), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(c[4]), "r"(b)
                : "memory");
            break;
    }
}

// Tensor copy shared -> global of one box (bulk-group completion).
__device__ __forceinline__ void tma_store(const TMap *m, int nd, const int *c, const void *src) {
    const unsigned s = saddr(src);
    const u64 mp = reinterpret_cast<u64>(m);
    switch (nd) {
        case 1:
            asm volatile("cp.async.bulk.tensor.1d.global.shared::cta.bulk_group [%0, {%1}], [%2];" ::"l"(mp), "r"(c[0]), "r"(s)
                         : "memory");
            break;
        case 2:
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(mp), "r"(c[0]),
                         "r"(c[1]), "r"(s)
                         : "memory");
            break;
        case 3:
            asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(mp), "r"(c[0]),
                         "r"(c[1]), "r"(c[2]), "r"(s)
                         : "memory");
            break;
        case 4:
            asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(mp),
                         "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(s)
                         : "memory");
            break;
        default:
            asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4, %5}], [%6];" ::"l"(mp),
                         "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(c[4]), "r"(s)
                         : "memory");
            break;
    }
}

__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// The shared-memory sources of every committed store have been read.
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// Every committed store is complete.
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Coordinates of the box with loop value v of the tile whose first global element index is `base`
// (batch index included above the state's qubits).
__device__ __forceinline__ void box_coords(const TmaGeom &t, u64 base, int v, int *c) {
    for (int k = 0; k < t.n_loop; ++k)
        if (v >> k & 1) base |= u64(1) << t.loop_q[k];
    for (int j = 0; j < t.nd; ++j) {
        u64 x = base >> t.shift[j];
        if (j + 1 < t.nd) x &= (u64(1) << (t.shift[j + 1] - t.shift[j])) - 1;
        if (j == 0) x *= u64(t.epa);
        c[j] = static_cast<int>(x);
    }
}

// Issue the loads of one tile of `map` into `dst` (2^n_loop boxes of box_bytes each).
__device__ __forceinline__ void load_tile(const TMap *m, const TmaGeom &t, u64 base, unsigned char *dst, u64 *bar) {
    int c[5];
    for (int v = 0; v < (1 << t.n_loop); ++v) {
        box_coords(t, base, v, c);
        tma_load(dst + static_cast<u64>(v) * t.box_bytes, m, t.nd, c, bar);
    }
}

__device__ __forceinline__ void store_tile(const TMap *m, const TmaGeom &t, u64 base, const unsigned char *src) {
    int c[5];
    for (int v = 0; v < (1 << t.n_loop); ++v) {
        box_coords(t, base, v, c);
        tma_store(m, t.nd, c, src + static_cast<u64>(v) * t.box_bytes);
    }
}

__device__ __forceinline__ void report(int *err, int code) {
    if (err) atomicCAS(err, 0, code);
}

}  // namespace pipe
}  // namespace mqb

#endif
