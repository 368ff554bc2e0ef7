// Adjoint sweep of the in-place cut-rank DP (complex128): gradients of log Pr(b) with respect to the step matrices.
//
// The forward sweep of a string b is linear in every table and in every step's M row:
//   T_{k+1} = L_k(M_k[b_k]) T_k,   Z(b) = T_ns[0],   Pr(b) = 2^-n |Z(b)|^2,
// with the step map of the executor (gsamp2.cpp:32-38, 59-66): for every coset c of step k, base = XOR of Tkeep
// over the bits of c, the inputs v_t = T_k[base ^ tq_t] and
//   out[tau] = sum_{t: tau0_t = tau} m0 v_t + sum_{t: tau1_t = tau} m1 s_t v_t,   s_t = (-1)^(parity(c & rhoc) ^ par_t),
// m_x = M_k[b_k][x].  The reverse sweep carries lambda_k = dZ/dT_k backwards through the transposed step map:
//   lambda_k[base ^ tq_t] = m0 lambda_{k+1}[tau0_t] + m1 s_t lambda_{k+1}[tau1_t],
//   dZ/dm0 = sum_t lambda_{k+1}[tau0_t] v_t,       dZ/dm1 = sum_t s_t lambda_{k+1}[tau1_t] v_t,
// with lambda_ns = 1 at the final entry.
//
// Both sweeps run in passes of two steps (one where two do not fuse), out of place: the table before a pass is kept for
// the reverse sweep, which computes the table between the pass's two steps again as it goes.  A pass of two steps then
// reads and writes a table once forward, and reads T, reads lambda and writes lambda once in reverse: five table
// transfers for two steps.  One step per pass with a checkpoint every four steps moved sixteen (forward, restore, the
// segment's tables again, the reverse reads and writes), and both forms are bound by HBM.
//
// Tables are compact: the entry at address base(c) ^ tq_t of the table before step k has index c | t << nk, which is
// XOR-linear in the address, so a pass walks its classes (gsb_fuse.h) with one running index per table.  A thread takes a
// whole class; its values of every stage sit in shared-memory slots of its own ([value][thread]: no bank conflicts and
// no barriers), filled by 16-byte asynchronous copies, all of a class at once.
//
// Up to 32 strings are swept together (grid dimension y: each string owns its tables and reduction slots), and the
// whole sequence of such a launch is one CUDA graph; the first string's index lives in device memory and advances at its
// end.  Where the tables of all passes do not fit, only every q-th is kept and the ones between are computed again,
// segment by segment.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "gsb.h"
#include "gsb_common.h"
#include "gsb_fuse.h"
#include "gsb_plan.h"
#include "gsb_step.h"

namespace gsb {

// A launch sweeps `bs` strings at once: string y = blockIdx.y is item *item + y and owns slot y of every buffer.
struct GradCtx {
    const double *M;         // [ns][2][2] (re, im): the caller's matrices
    const int8_t *bits;      // [cap][ns]
    const int *item;         // first string of the launch
    int ns;
};

// Shape of a step's dataflow: with m = 2 and every x = 1 term in the other output than its offset's x = 0 term, the host
// orders the offsets so that the x = 0 terms of the first NTQ - H go to output 0 and those of the last H to output 1
// (relabelling the outputs where that makes H <= NTQ / 2).  RK_ANY: everything else, with runtime tables.
enum { RK_ANY = 0, RK_1_0, RK_2_0, RK_2_1, RK_4_0, RK_4_1, RK_4_2 };

// One step inside a pass.  Every stage's values are numbered so that member j reads values ntq j + t; out[j][tau]: the
// number of its outputs in the next stage (m j + tau in the last one).  Class sign: parity(class & lam) ^ bit j of mpar.
struct GradStep {
    int k, kind, nmem, ntq, m;
    int tau0, tau1;          // bit t: offset t's x = 0 / x = 1 output
    uint32_t mpar;
    double sg[4];            // sign of offset t's x = 1 term
    uint64_t lam;
    unsigned char out[16][2];
};

// A pass: 2^nb classes; class p has index XOR of cin[j] (cout[j]) over the bits of p in the table read (written), and
// its value i of the first (last) stage sits at that index ^ zin[i] (zout[i]).
struct GradPass {
    int d, nb, ssz[3];
    uint32_t cin[34], cout[34], zin[32], zout[32];
    GradStep st[2];
};
static_assert(sizeof(GradPass) <= 3500, "a pass goes by value as a kernel parameter");

constexpr int GRAD_THREADS = 128;
constexpr int GRAD_MAX_VALUES = 64;   // stage values of a class: 64 x 16 B x 128 threads = 128 KB of slots

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 c) {
    return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
__device__ __forceinline__ double2 csign(double2 a, int neg) {
    const int f = neg << 31;
    return make_double2(__hiloint2double(__double2hiint(a.x) ^ f, __double2loint(a.x)),
                        __hiloint2double(__double2hiint(a.y) ^ f, __double2loint(a.y)));
}

__device__ __forceinline__ void copy16(double2 *dst, const double2 *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copies_landed() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The classes a thread visits (grid x times block: a power of two, 2^ls threads): p = t | (g << ls) for the Gray codes g
// of the high bits, so both indices are running values (one XOR each per class).
struct ClassWalk {
    uint64_t p, n, count;
    uint32_t in, out;
    int ls;
    __device__ ClassWalk(const GradPass &g) {
        ls = __ffs((int)(gridDim.x * blockDim.x)) - 1;
        p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
        n = 0;
        in = out = 0;
        count = g.nb > ls ? 1ULL << (g.nb - ls) : p < (1ULL << g.nb) ? 1 : 0;
        for (int j = 0; j < min(g.nb, ls); j++)
            if ((p >> j) & 1) { in ^= g.cin[j]; out ^= g.cout[j]; }
    }
    __device__ bool more() const { return n < count; }
    __device__ void next(const GradPass &g) {
        if (++n >= count) return;
        const int j = ls + __ffsll((long long)n) - 1;
        p ^= 1ULL << j;
        in ^= g.cin[j];
        out ^= g.cout[j];
    }
};

struct MRow {
    double2 m0, m1;
};
__device__ __forceinline__ MRow step_row(const GradStep &s, const GradCtx &g) {
    const int b = g.bits[(size_t)(*g.item + (int)blockIdx.y) * (size_t)g.ns + (size_t)s.k];
    const double *Mk = g.M + (size_t)s.k * 8 + 4 * b;
    return MRow{make_double2(Mk[0], Mk[1]), make_double2(Mk[2], Mk[3])};
}

// This thread's slot i.
__device__ __forceinline__ double2 &slot(double2 *sh, int i) { return sh[i * GRAD_THREADS + (int)threadIdx.x]; }

// Member j's values, inputs in slots a..
template <int NTQ>
__device__ __forceinline__ void member_values(double2 *sh, int a, int j, double2 (&v)[NTQ]) {
#pragma unroll
    for (int t = 0; t < NTQ; t++) v[t] = slot(sh, a + NTQ * j + t);
}

// Coset sums of a shaped member: X[tau] of the x = 0 terms, Z[tau] of the signed x = 1 terms (H = 0: X[0] and Z[1] only).
template <int NTQ, int H>
__device__ __forceinline__ void member_sums(const GradStep &s, const double2 (&v)[NTQ], double2 (&X)[2], double2 (&Z)[2]) {
#pragma unroll
    for (int t = 0; t < NTQ; t++) {
        const int o = t < NTQ - H ? 0 : 1;
        const bool first = t == 0 || (H > 0 && t == NTQ - H);
        X[o] = first ? v[t] : cadd(X[o], v[t]);
        Z[1 - o] = first ? make_double2(s.sg[t] * v[t].x, s.sg[t] * v[t].y)
                         : make_double2(fma(s.sg[t], v[t].x, Z[1 - o].x), fma(s.sg[t], v[t].y, Z[1 - o].y));
    }
}

// A shaped step forward on one class: values in slots a.., output tau of member j to f(j, tau, value).  NM: members, 0
// for a runtime count; known counts leave every index a constant.
template <int NTQ, int H, int NM, typename F>
__device__ __forceinline__ void class_fwd(const GradStep &s, const MRow &m, double2 *sh, int a, int cpar, F f) {
    auto member = [&](int j) {
        double2 v[NTQ], X[2], Z[2];
        member_values<NTQ>(sh, a, j, v);
        member_sums<NTQ, H>(s, v, X, Z);
        const double2 m1 = csign(m.m1, (cpar ^ (int)(s.mpar >> j)) & 1);
        f(j, 0, H == 0 ? cmul(m.m0, X[0]) : cfma(m.m0, X[0], cmul(m1, Z[0])));
        f(j, 1, H == 0 ? cmul(m1, Z[1]) : cfma(m.m0, X[1], cmul(m1, Z[1])));
    };
    if constexpr (NM > 0) {
#pragma unroll
        for (int j = 0; j < NM; j++) member(j);
    } else {
        for (int j = 0; j < s.nmem; j++) member(j);
    }
}

// A shaped step in reverse on one class: inputs in slots a.., lambda of output tau of member j in slot lam(j, tau);
// lambda of its offset t to f(j, t, value), the sums for dZ/dM to acc.
template <int NTQ, int H, int NM, typename L, typename F>
__device__ __forceinline__ void class_bwd(const GradStep &s, const MRow &m, double2 *sh, int a, int cpar, double2 (&acc)[2],
                                          L lam, F f) {
    auto member = [&](int j) {
        double2 v[NTQ], X[2], Z[2];
        member_values<NTQ>(sh, a, j, v);
        const double2 l0 = slot(sh, lam(j, 0)), l1 = slot(sh, lam(j, 1));
        member_sums<NTQ, H>(s, v, X, Z);
        const int cs = (cpar ^ (int)(s.mpar >> j)) & 1;
        const double2 m1 = csign(m.m1, cs);
        double2 p[2], q[2];   // m0 lambda and m1 lambda of the outputs that x = 0 / x = 1 terms reach
        if (H == 0) {
            acc[0] = cfma(l0, X[0], acc[0]);
            acc[1] = cfma(csign(l1, cs), Z[1], acc[1]);
            p[0] = cmul(m.m0, l0);
            q[1] = cmul(m1, l1);
        } else {
            acc[0] = cfma(l0, X[0], cfma(l1, X[1], acc[0]));
            acc[1] = cfma(csign(l0, cs), Z[0], cfma(csign(l1, cs), Z[1], acc[1]));
            p[0] = cmul(m.m0, l0);
            p[1] = cmul(m.m0, l1);
            q[0] = cmul(m1, l0);
            q[1] = cmul(m1, l1);
        }
#pragma unroll
        for (int t = 0; t < NTQ; t++) {
            const int o = t < NTQ - H ? 0 : 1;
            f(j, t, make_double2(fma(s.sg[t], q[1 - o].x, p[o].x), fma(s.sg[t], q[1 - o].y, p[o].y)));
        }
    };
    if constexpr (NM > 0) {
#pragma unroll
        for (int j = 0; j < NM; j++) member(j);
    } else {
        for (int j = 0; j < s.nmem; j++) member(j);
    }
}

// Any step: runtime offsets and outputs (one or two).
template <typename F>
__device__ __forceinline__ void class_fwd_any(const GradStep &s, const MRow &m, double2 *sh, int a, int cpar, F f) {
    for (int j = 0; j < s.nmem; j++) {
        double2 X[2], Z[2];
        X[0] = X[1] = Z[0] = Z[1] = make_double2(0, 0);
        for (int t = 0; t < s.ntq; t++) {
            const double2 v = slot(sh, a + s.ntq * j + t), w = make_double2(s.sg[t] * v.x, s.sg[t] * v.y);
            if ((s.tau0 >> t) & 1) X[1] = cadd(X[1], v);
            else X[0] = cadd(X[0], v);
            if ((s.tau1 >> t) & 1) Z[1] = cadd(Z[1], w);
            else Z[0] = cadd(Z[0], w);
        }
        const double2 m1 = csign(m.m1, (cpar ^ (int)(s.mpar >> j)) & 1);
        f(j, 0, cfma(m.m0, X[0], cmul(m1, Z[0])));
        if (s.m == 2) f(j, 1, cfma(m.m0, X[1], cmul(m1, Z[1])));
    }
}
template <typename L, typename F>
__device__ __forceinline__ void class_bwd_any(const GradStep &s, const MRow &m, double2 *sh, int a, int cpar, double2 (&acc)[2],
                                              L lam, F f) {
    for (int j = 0; j < s.nmem; j++) {
        const double2 l0 = slot(sh, lam(j, 0)), l1 = s.m == 2 ? slot(sh, lam(j, 1)) : make_double2(0, 0);
        const int cs = (cpar ^ (int)(s.mpar >> j)) & 1;
        const double2 m1 = csign(m.m1, cs), s0 = csign(l0, cs), s1 = csign(l1, cs);
        const double2 p0 = cmul(m.m0, l0), p1 = cmul(m.m0, l1), q0 = cmul(m1, l0), q1 = cmul(m1, l1);
        for (int t = 0; t < s.ntq; t++) {
            const double2 v = slot(sh, a + s.ntq * j + t), w = make_double2(s.sg[t] * v.x, s.sg[t] * v.y);
            const bool u0 = (s.tau0 >> t) & 1, u1 = (s.tau1 >> t) & 1;
            acc[0] = cfma(u0 ? l1 : l0, v, acc[0]);
            acc[1] = cfma(u1 ? s1 : s0, w, acc[1]);
            const double2 p = u0 ? p1 : p0, q = u1 ? q1 : q0;
            f(j, t, make_double2(fma(s.sg[t], q.x, p.x), fma(s.sg[t], q.y, p.y)));
        }
    }
}

#define GSB_RK(KIND, CALL, NTQ, H)                  \
    case KIND:                                      \
        switch (s.nmem) {                           \
            case 1: CALL(NTQ, H, 1); break;         \
            case 2: CALL(NTQ, H, 2); break;         \
            case 4: CALL(NTQ, H, 4); break;         \
            default: CALL(NTQ, H, 0); break;        \
        }                                           \
        break;
#define GSB_RKS(CALL, ANY)                          \
    switch (s.kind) {                               \
        GSB_RK(RK_1_0, CALL, 1, 0)                  \
        GSB_RK(RK_2_0, CALL, 2, 0)                  \
        GSB_RK(RK_2_1, CALL, 2, 1)                  \
        GSB_RK(RK_4_0, CALL, 4, 0)                  \
        GSB_RK(RK_4_1, CALL, 4, 1)                  \
        GSB_RK(RK_4_2, CALL, 4, 2)                  \
        default: ANY;                               \
    }
template <typename F>
__device__ __forceinline__ void step_fwd(const GradStep &s, const MRow &m, double2 *sh, int a, int cpar, F f) {
#define GSB_CALL(NTQ, H, NM) class_fwd<NTQ, H, NM>(s, m, sh, a, cpar, f)
    GSB_RKS(GSB_CALL, class_fwd_any(s, m, sh, a, cpar, f))
#undef GSB_CALL
}
template <typename L, typename F>
__device__ __forceinline__ void step_bwd(const GradStep &s, const MRow &m, double2 *sh, int a, int cpar, double2 (&acc)[2],
                                         L lam, F f) {
#define GSB_CALL(NTQ, H, NM) class_bwd<NTQ, H, NM>(s, m, sh, a, cpar, acc, lam, f)
    GSB_RKS(GSB_CALL, class_bwd_any(s, m, sh, a, cpar, acc, lam, f))
#undef GSB_CALL
}
#undef GSB_RKS
#undef GSB_RK

__global__ void k_gr_begin(double2 *T, size_t stride) { T[blockIdx.y * stride] = make_double2(1.0, 0.0); }

// Forward pass: the table `in` to the table `out` (strides: entries between two strings' tables).
template <int D>
__global__ void __launch_bounds__(GRAD_THREADS) k_gr_fwd(const GradPass g, const double2 *__restrict__ in, size_t in_stride,
                                                         double2 *__restrict__ out, size_t out_stride, const GradCtx c) {
    extern __shared__ __align__(16) double2 sh[];
    const MRow ma = step_row(g.st[0], c), mb = step_row(g.st[D - 1], c);
    in += blockIdx.y * in_stride;
    out += blockIdx.y * out_stride;
    ClassWalk w(g);
    if (w.more())
        for (int i = 0; i < g.ssz[0]; i++) copy16(&slot(sh, i), in + (w.in ^ g.zin[i]));
    while (w.more()) {
        copies_landed();
        const uint64_t p = w.p;
        const uint32_t o = w.out;
        const int s1 = g.ssz[0], om = g.st[D - 1].m;
        auto store = [&](int j, int tau, double2 v) { out[o ^ g.zout[om * j + tau]] = v; };
        if (D == 1) {
            step_fwd(g.st[0], ma, sh, 0, __popcll(p & g.st[0].lam), store);
        } else {
            step_fwd(g.st[0], ma, sh, 0, __popcll(p & g.st[0].lam),
                     [&](int j, int tau, double2 v) { slot(sh, s1 + g.st[0].out[j][tau]) = v; });
        }
        w.next(g);   // the first stage is done: the next class's values arrive while the second step runs
        if (w.more())
            for (int i = 0; i < g.ssz[0]; i++) copy16(&slot(sh, i), in + (w.in ^ g.zin[i]));
        if (D == 2) step_fwd(g.st[D - 1], mb, sh, s1, __popcll(p & g.st[D - 1].lam), store);
    }
}

// End of the forward sweep: Z = T_ns[0]; lambda_ns = 1.
__global__ void k_gr_final(const double2 *T, size_t t_stride, double2 *Lam, size_t l_stride, double2 *z_out,
                           const GradCtx g) {
    z_out[*g.item + (int)blockIdx.y] = T[blockIdx.y * t_stride];
    Lam[blockIdx.y * l_stride] = make_double2(1.0, 0.0);
}

__global__ void k_gr_next(int *item, int bs) { *item += bs; }
__global__ void k_gr_set_item(int *item, int v) { *item = v; }

// Measured on the width-20 workload (128 strings, loss and gradient): 23.1 -> 9.4 ms a call with both sweeps in two-step
// passes and runtime tables (the widest reverse pass bound by issue: 900 instructions per class of four values, 0.34 ms for
// 1.3 GB), 8.4 ms with each step's code compiled for its shape and member count (470 instructions, 0.24 ms, 5.4 TB/s: the
// reads of T and lambda).  Five blocks per SM (96 registers) took 4 % off against four; six and eight spill.
//
// Reverse pass: lambda after the pass (`lo`) and the table before it (T) to lambda before it (`li`), and
// dZ/dM_k[b_k][x] of its steps.  Deterministic reduction: per-block partials, the last block sums them in block order
// and writes grad[item][k] = (dZ/dm0, dZ/dm1).
template <int D>
__global__ void __launch_bounds__(GRAD_THREADS, 5) k_gr_bwd(const GradPass g, const double2 *__restrict__ T, size_t t_stride,
                                                         const double2 *__restrict__ lo, double2 *__restrict__ li,
                                                         size_t l_stride, const GradCtx c, double *partials,
                                                         unsigned int *counter, double *grad) {
    extern __shared__ __align__(16) double2 sh[];
    const MRow ma = step_row(g.st[0], c), mb = step_row(g.st[D - 1], c);
    T += blockIdx.y * t_stride;
    lo += blockIdx.y * l_stride;
    li += blockIdx.y * l_stride;
    counter += blockIdx.y;
    const int s1 = g.ssz[0], s2 = D == 2 ? s1 + g.ssz[1] : s1, nl = g.ssz[D];   // slots of stage 1, and of lambda after
    const double2 z = make_double2(0, 0);
    double2 acc[D][2];
#pragma unroll
    for (int s = 0; s < D; s++) acc[s][0] = acc[s][1] = z;
    for (ClassWalk w(g); w.more(); w.next(g)) {
        for (int i = 0; i < g.ssz[0]; i++) copy16(&slot(sh, i), T + (w.in ^ g.zin[i]));
        for (int i = 0; i < nl; i++) copy16(&slot(sh, s2 + i), lo + (w.out ^ g.zout[i]));
        copies_landed();
        const int pa = __popcll(w.p & g.st[0].lam);
        const uint32_t in = w.in;
        const int na = g.st[0].ntq, nb = g.st[D - 1].ntq, om = g.st[D - 1].m;
        auto store = [&](int j, int t, double2 v) { li[in ^ g.zin[na * j + t]] = v; };
        auto after = [&](int j, int tau) { return s2 + om * j + tau; };
        if (D == 1) {
            step_bwd(g.st[0], ma, sh, 0, pa, acc[0], after, store);
        } else {
            // a stage-1 slot holds the second step's input until the member that reads it, then its lambda
            auto mid = [&](int j, int tau) { return s1 + g.st[0].out[j][tau]; };
            step_fwd(g.st[0], ma, sh, 0, pa, [&](int j, int tau, double2 v) { slot(sh, mid(j, tau)) = v; });
            step_bwd(g.st[D - 1], mb, sh, s1, __popcll(w.p & g.st[D - 1].lam), acc[D - 1], after,
                     [&](int j, int t, double2 v) { slot(sh, s1 + nb * j + t) = v; });
            step_bwd(g.st[0], ma, sh, 0, pa, acc[0], mid, store);
        }
    }
    __shared__ double red[4 * D][GRAD_THREADS / 32];
    __shared__ int last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    partials += (size_t)blockIdx.y * gridDim.x * (4 * D);
#pragma unroll
    for (int s = 0; s < D; s++)
#pragma unroll
        for (int x = 0; x < 2; x++) {
            const double r = warp_sum(acc[s][x].x), i = warp_sum(acc[s][x].y);
            if (lane == 0) { red[4 * s + 2 * x][warp] = r; red[4 * s + 2 * x + 1][warp] = i; }
        }
    __syncthreads();
    if (threadIdx.x < 4 * D) {
        double t = 0;
        for (int v = 0; v < GRAD_THREADS / 32; v++) t += red[threadIdx.x][v];
        partials[4 * D * blockIdx.x + threadIdx.x] = t;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || threadIdx.x >= 4 * D) return;
    __threadfence();
    double t = 0;
    for (unsigned int b = 0; b < gridDim.x; b++) t += __ldcg(partials + 4 * D * b + threadIdx.x);
    const GradStep &s = g.st[threadIdx.x >> 2 & (D - 1)];
    grad[((size_t)(*c.item + (int)blockIdx.y) * (size_t)c.ns + (size_t)s.k) * 4 + (threadIdx.x & 3)] = t;
    if (threadIdx.x == 0) *counter = 0;
}

// Index of an address in the compact table before step k (HStep columns): XOR-linear, c | t << nk with the offsets in
// ascending order (their index is linear too: the three nonzero ones XOR to 0).
class TableIndex {
    struct Row {
        uint64_t v;
        uint32_t i;
    };
    std::vector<Row> rows;   // each reduced by the ones before it

public:
    explicit TableIndex(const HStep *s) {
        if (!s) return;      // the table after the last step: one entry
        for (int j = 0; j < s->nk; j++) add(s->tk[(size_t)j], 1u << j);
        if (s->tqs.size() > 1) add(s->tqs[1], 1u << s->nk);
        if (s->tqs.size() > 2) add(s->tqs[2], 2u << s->nk);
    }
    void add(uint64_t v, uint32_t i) {
        reduce(v, i);
        if (v) rows.push_back({v, i});
    }
    void reduce(uint64_t &v, uint32_t &i) const {
        for (const Row &r : rows)
            if (v >> (63 - __builtin_clzll(r.v)) & 1) { v ^= r.v; i ^= r.i; }
    }
    uint32_t operator()(uint64_t v) const {
        uint32_t i = 0;
        reduce(v, i);
        return i;
    }
};

// The pass of steps gp.k0 .. gp.k0 + gp.d - 1; false when it is too large for the kernels.
static bool make_pass(const HPlan &p, const GroupPlan &gp, GradPass &g) {
    memset(&g, 0, sizeof g);
    int values = 0;
    for (int s = 0; s <= gp.d; s++) values += g.ssz[s] = gp.stage_size[s];
    if (values > GRAD_MAX_VALUES || gp.nb > 32) return false;
    g.d = gp.d;
    g.nb = gp.nb;
    const int k1 = gp.k0 + gp.d;
    const TableIndex before(&p.st[(size_t)gp.k0]), after(k1 < p.ns ? &p.st[(size_t)k1] : nullptr);
    std::vector<uint64_t> cols;
    for (int j = 0; j < gp.L; j++) cols.push_back(1ULL << j);
    cols.insert(cols.end(), gp.bhi.begin(), gp.bhi.end());
    for (int j = 0; j < gp.nb; j++) {
        g.cin[j] = before(cols[(size_t)j]);
        g.cout[j] = after(cols[(size_t)j]);
    }
    std::vector<int> number[3];   // of the plan's stage values: member-major in the step that reads them
    int perm[2][4], swp[2];
    for (int s = 0; s < gp.d; s++) {
        const HStep &hs = p.st[(size_t)(gp.k0 + s)];
        const GroupPlan::Step &q = gp.step[s];
        GradStep &a = g.st[s];
        bool shaped = q.m == 2;
        int h = 0;
        for (int t = 0; t < q.ntq; t++) {
            shaped = shaped && hs.tau1[t] == 1 - hs.tau0[t];
            h += hs.tau0[t];
        }
        swp[s] = shaped && 2 * h > q.ntq;
        if (swp[s]) h = q.ntq - h;
        int n = 0;
        for (int out = 0; out < 2; out++)
            for (int t = 0; t < q.ntq; t++)
                if (!shaped ? out == 0 : (hs.tau0[t] ^ swp[s]) == out) perm[s][n++] = t;
        a.kind = RK_ANY;
        if (shaped && q.ntq == 1) a.kind = RK_1_0;
        else if (shaped && q.ntq == 2) a.kind = h == 0 ? RK_2_0 : RK_2_1;
        else if (shaped && q.ntq == 4) a.kind = h == 0 ? RK_4_0 : h == 1 ? RK_4_1 : RK_4_2;
        a.k = gp.k0 + s;
        a.nmem = q.nmem;
        a.ntq = q.ntq;
        a.m = q.m;
        for (int t = 0; t < q.ntq; t++) {
            a.tau0 |= (hs.tau0[perm[s][t]] ^ swp[s]) << t;
            a.tau1 |= (hs.tau1[perm[s][t]] ^ swp[s]) << t;
            a.sg[t] = hs.par[perm[s][t]] ? -1.0 : 1.0;
        }
        for (int j = 0; j < gp.nb; j++)
            a.lam |= (uint64_t)(__builtin_popcountll(cols[(size_t)j] & q.lambda) & 1) << j;
        number[s].assign((size_t)gp.stage_size[s], 0);
        for (int j = 0; j < q.nmem; j++) {
            a.mpar |= (uint32_t)(q.mpar[j] & 1) << j;
            for (int t = 0; t < q.ntq; t++) number[s][(size_t)q.in_idx[j][perm[s][t]]] = q.ntq * j + t;
        }
    }
    for (int i = 0; i < gp.stage_size[0]; i++) g.zin[number[0][(size_t)i]] = before(gp.z_in[(size_t)i]);
    for (int s = 0; s < gp.d; s++) {
        const GroupPlan::Step &q = gp.step[s];
        for (int j = 0; j < q.nmem; j++)
            for (int tau = 0; tau < q.m; tau++) {
                const int old = q.out_idx[j][tau ^ swp[s]];
                if (s + 1 < gp.d) g.st[s].out[j][tau] = (unsigned char)number[s + 1][(size_t)old];
                else g.zout[q.m * j + tau] = after(gp.z_out[(size_t)old]);
            }
    }
    return true;
}

struct GradEngine {
    HPlan plan;
    int dev = 0, sms = 0, cap = 1024, bs = 1;   // cap: strings per host batch, a multiple of bs
    std::vector<GradPass> passes;
    std::vector<size_t> entries;       // of the table before pass i; the last one (after all passes) is 1
    int q = 1;                         // every q-th pass keeps its table
    std::vector<size_t> kept_off;      // offset (entries) of pass i's kept table in a string's slot (i % q == 0)
    size_t kept_n = 0, seg_stride = 0; // entries per string: kept tables; one table of a segment, or a lambda table
    double2 *d_kept = nullptr, *d_seg = nullptr, *d_pair[2] = {nullptr, nullptr};
    double *d_M = nullptr, *partials = nullptr, *d_grad = nullptr;
    double2 *d_z = nullptr;
    int8_t *d_bits = nullptr;
    int *d_item = nullptr;
    unsigned int *d_counter = nullptr;
    cudaStream_t stream = nullptr;
    cudaGraphExec_t graph = nullptr;

    ~GradEngine() {
        int prev = 0;
        cudaGetDevice(&prev);
        cudaSetDevice(dev);
        if (graph) cudaGraphExecDestroy(graph);
        cudaFree(d_kept);
        cudaFree(d_seg);
        cudaFree(d_pair[0]);
        cudaFree(d_pair[1]);
        cudaFree(d_M);
        cudaFree(partials);
        cudaFree(d_grad);
        cudaFree(d_z);
        cudaFree(d_bits);
        cudaFree(d_item);
        cudaFree(d_counter);
        if (stream) cudaStreamDestroy(stream);
        cudaSetDevice(prev);
    }

    // Kept tables for an interval of n passes; returns the device bytes a string needs.
    size_t lay_out(int n) {
        q = n;
        kept_off.assign(passes.size(), 0);
        kept_n = 0;
        for (size_t i = 0; i < passes.size(); i += (size_t)n) {
            kept_off[i] = kept_n;
            kept_n += entries[i];
        }
        return 16 * (kept_n + (size_t)(n - 1) * seg_stride + 2 * seg_stride) + (size_t)max_blocks() * 8 * sizeof(double);
    }
    // Blocks of a launch over all its strings: four rounds of four per SM; every block ends in a block reduction and an
    // atomic, so a thread walks several classes.
    int max_blocks() const { return sms * 16; }
    dim3 grid_of(const GradPass &g) const {
        const uint64_t want = std::min<uint64_t>(((1ULL << g.nb) + GRAD_THREADS - 1) / GRAD_THREADS,
                                                 std::max(1, max_blocks() / bs));
        uint64_t gx = 1;   // a power of two: ClassWalk splits a class index into thread and Gray-walk bits
        while (gx * 2 <= want) gx *= 2;
        return dim3((unsigned)gx, (unsigned)bs);
    }
    GradCtx ctx() const { return GradCtx{d_M, d_bits, d_item, plan.ns}; }

    // Where the table before pass i lives while `seg0` is the first pass of the segment being worked on.
    double2 *table(size_t i, size_t *stride) const {
        if (i % (size_t)q == 0) {
            *stride = kept_n;
            return d_kept + kept_off[i];
        }
        *stride = (size_t)(q - 1) * seg_stride;
        return d_seg + (i % (size_t)q - 1) * seg_stride;
    }
    static size_t fwd_smem(const GradPass &g) { return (size_t)(g.ssz[0] + (g.d == 2 ? g.ssz[1] : 0)) * 16 * GRAD_THREADS; }
    static size_t bwd_smem(const GradPass &g) {
        return (size_t)(g.ssz[0] + g.ssz[1] + (g.d == 2 ? g.ssz[2] : 0)) * 16 * GRAD_THREADS;
    }
    // Kernels whose passes need more shared memory than a launch has by default; asked for before the first sweep and not in
    // an open, which would load the kernels.
    cudaError_t allow_smem() const {
        const int most = GRAD_MAX_VALUES * 16 * GRAD_THREADS;   // of the largest pass
        cudaError_t e = cudaSuccess;
        for (int d = 1; d <= 2; d++) {
            size_t f = 0, b = 0;
            for (const GradPass &g : passes)
                if (g.d == d) { f = std::max(f, fwd_smem(g)); b = std::max(b, bwd_smem(g)); }
            const void *fk = d == 2 ? (const void *)k_gr_fwd<2> : (const void *)k_gr_fwd<1>;
            const void *bk = d == 2 ? (const void *)k_gr_bwd<2> : (const void *)k_gr_bwd<1>;
            // the reverse pass's static sums count too
            if (e == cudaSuccess && f > 47 * 1024) e = cudaFuncSetAttribute(fk, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
            if (e == cudaSuccess && b > 47 * 1024) e = cudaFuncSetAttribute(bk, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        }
        return e;
    }
    cudaError_t fwd(size_t i, const double2 *in, size_t is, double2 *out, size_t os) {
        const GradPass &g = passes[i];
        const size_t sm = fwd_smem(g);
        if (g.d == 2) k_gr_fwd<2><<<grid_of(g), GRAD_THREADS, sm, stream>>>(g, in, is, out, os, ctx());
        else k_gr_fwd<1><<<grid_of(g), GRAD_THREADS, sm, stream>>>(g, in, is, out, os, ctx());
        return cudaGetLastError();
    }
    cudaError_t bwd(size_t i, const double2 *T, size_t ts, const double2 *lo, double2 *li) {
        const GradPass &g = passes[i];
        const size_t sm = bwd_smem(g);
        if (g.d == 2)
            k_gr_bwd<2><<<grid_of(g), GRAD_THREADS, sm, stream>>>(g, T, ts, lo, li, seg_stride, ctx(), partials, d_counter,
                                                                  d_grad);
        else
            k_gr_bwd<1><<<grid_of(g), GRAD_THREADS, sm, stream>>>(g, T, ts, lo, li, seg_stride, ctx(), partials, d_counter,
                                                                  d_grad);
        return cudaGetLastError();
    }

    // The sequence of one launch of bs strings (captured once as a graph).
    cudaError_t enqueue() {
        const dim3 one(1, (unsigned)bs);
        const size_t np = passes.size();
        k_gr_begin<<<one, 1, 0, stream>>>(d_kept, kept_n);
        cudaError_t e = cudaGetLastError();
        // forward: tables that are not kept pass through the pair that holds lambda later
        const double2 *in = d_kept;
        size_t is = kept_n;
        for (size_t i = 0; i < np && e == cudaSuccess; i++) {
            double2 *out = d_pair[i & 1];
            size_t os = seg_stride;
            if (i + 1 < np && (i + 1) % (size_t)q == 0) out = table(i + 1, &os);
            e = fwd(i, in, is, out, os);
            in = out;
            is = os;
        }
        if (e != cudaSuccess) return e;
        int cur = in == d_pair[0] ? 1 : 0;   // lambda starts in the buffer that does not hold T_ns
        k_gr_final<<<one, 1, 0, stream>>>(in, is, d_pair[cur], seg_stride, d_z, ctx());
        e = cudaGetLastError();
        for (size_t c = (np - 1) / (size_t)q * (size_t)q; e == cudaSuccess; c -= (size_t)q) {
            const size_t end = std::min(c + (size_t)q, np);
            for (size_t i = c; i + 1 < end && e == cudaSuccess; i++) {   // the segment's tables again
                size_t a, b;
                const double2 *src = table(i, &a);
                double2 *dst = table(i + 1, &b);
                e = fwd(i, src, a, dst, b);
            }
            for (size_t i = end; i-- > c && e == cudaSuccess; cur ^= 1) {
                size_t a;
                const double2 *T = table(i, &a);
                e = bwd(i, T, a, d_pair[cur], d_pair[cur ^ 1]);
            }
            if (c == 0) break;
        }
        if (e != cudaSuccess) return e;
        k_gr_next<<<1, 1, 0, stream>>>(d_item, bs);
        return cudaGetLastError();
    }
};

}  // namespace gsb

using namespace gsb;

#define GR_CK(x)                                                                                                  \
    do {                                                                                                          \
        cudaError_t e_ = (x);                                                                                     \
        if (e_ != cudaSuccess) return fail(GSB_E_CUDA, std::string("CUDA error: ") + cudaGetErrorString(e_) + " at " #x); \
    } while (0)

struct gsb_grad {
    GradEngine E;
};

extern "C" {

int gsb_grad_open_text(const char *text, size_t len, int device, int every, gsb_grad **out) {
    if (!text || !out) return fail(GSB_E_USAGE, "null argument");
    *out = nullptr;
    if (every < 1 || every > 64) return fail(GSB_E_USAGE, "checkpoint interval must be 1..64");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) return fail(GSB_E_CUDA, "no CUDA device is visible");
    if (device < 0 || device >= ndev) return fail(GSB_E_USAGE, "device out of range");
    gsb_grad *h = new gsb_grad();
    GradEngine &E = h->E;
    std::string err;
    int rc = parse_plan_text(text, len, E.plan, err);
    if (!rc) rc = validate_plan(E.plan, err);
    if (rc) {
        delete h;
        return fail(rc, err);
    }
    const HPlan &p = E.plan;
    if (p.ns < 1) {
        delete h;
        return fail(GSB_E_USAGE, "plan has no steps");
    }
    const HStep &lastst = p.st[(size_t)p.ns - 1];
    if (lastst.nk != 0 || lastst.m != 1) {
        delete h;
        return fail(GSB_E_USAGE, "the last step must leave a single entry (nk = 0, m = 1)");
    }
    E.dev = device;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    struct Restore {
        int p;
        ~Restore() { cudaSetDevice(p); }
    } restore{prev};
    cudaDeviceGetAttribute(&E.sms, cudaDevAttrMultiProcessorCount, device);
    for (int k = 0; k < p.ns;) {
        GradPass g;
        GroupPlan gp;
        int d = 2;
        while (d > 0 && !(plan_group(p, k, d, 0, 30, gp) && make_pass(p, gp, g))) d--;
        if (d == 0) {
            delete h;
            return fail(GSB_E_PLAN_LAYOUT, "step " + std::to_string(k) + " does not fit a pass of the adjoint sweep");
        }
        E.passes.push_back(g);
        E.entries.push_back(((size_t)1 << p.st[(size_t)k].nk) * p.st[(size_t)k].tqs.size());
        E.seg_stride = std::max(E.seg_stride, E.entries.back());
        k += d;
    }
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    // The default interval of four steps keeps the table before every pass (half of all tables: less memory than
    // checkpoints and the segments between them took), longer ones every (every / 4)-th; where that does not fit, fewer.
    size_t per_string = E.lay_out(std::max(1, every / 4));
    for (int n = E.q + 1; per_string > free_b / 10 * 9 && n <= (int)E.passes.size(); n++) per_string = E.lay_out(n);
    if (per_string > free_b / 10 * 9) {
        delete h;
        return fail(GSB_E_ALLOC, "kept tables, segment tables and lambda need " + std::to_string(per_string) +
                                     " bytes; the device has " + std::to_string(free_b) + " free");
    }
    // strings per launch: a power of two up to 32, each with its own tables, within half of the free device memory
    E.bs = 1;
    while (E.bs < 32 && (size_t)(2 * E.bs) * per_string <= free_b / 2) E.bs *= 2;
    const size_t bs = (size_t)E.bs;
    cudaError_t e = cudaStreamCreateWithFlags(&E.stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&E.d_kept, bs * E.kept_n * 16);
    if (e == cudaSuccess && E.q > 1) e = cudaMalloc(&E.d_seg, bs * (size_t)(E.q - 1) * E.seg_stride * 16);
    for (auto &b : E.d_pair)
        if (e == cudaSuccess) e = cudaMalloc(&b, bs * E.seg_stride * 16);
    if (e == cudaSuccess) e = cudaMalloc(&E.d_M, (size_t)p.ns * 8 * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&E.partials, std::max<size_t>((size_t)E.max_blocks(), bs) * 8 * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&E.d_grad, (size_t)E.cap * (size_t)p.ns * 4 * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&E.d_z, (size_t)E.cap * sizeof(double2));
    if (e == cudaSuccess) e = cudaMalloc(&E.d_bits, (size_t)E.cap * (size_t)p.ns);
    if (e == cudaSuccess) e = cudaMalloc(&E.d_item, sizeof(int));
    if (e == cudaSuccess) e = cudaMalloc(&E.d_counter, bs * sizeof(unsigned int));
    if (e == cudaSuccess) e = cudaMemsetAsync(E.d_counter, 0, bs * sizeof(unsigned int), E.stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(E.stream);
    if (e != cudaSuccess) {
        delete h;
        return fail(GSB_E_ALLOC, std::string("device allocation: ") + cudaGetErrorString(e));
    }
    *out = h;
    return 0;
}

int gsb_grad_close(gsb_grad *h) {
    delete h;
    return 0;
}

int gsb_grad_run(gsb_grad *h, const double *M, const int8_t *bits, int64_t nstr, double *z, double *dz) {
    if (!h) return fail(GSB_E_STATE, "null handle");
    if (nstr < 0 || (nstr && (!M || !bits || !z || !dz))) return fail(GSB_E_USAGE, "null argument");
    GradEngine &E = h->E;
    const int ns = E.plan.ns;
    for (int64_t i = 0; i < nstr * ns; i++)
        if (bits[i] != 0 && bits[i] != 1) return fail(GSB_E_USAGE, "bits must be 0 or 1");
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(E.dev);
    struct Restore {
        int p;
        ~Restore() { cudaSetDevice(p); }
    } restore{prev};
    GR_CK(cudaMemcpyAsync(E.d_M, M, (size_t)ns * 8 * sizeof(double), cudaMemcpyHostToDevice, E.stream));
    if (!E.graph) {
        GR_CK(E.allow_smem());
        cudaGraph_t gr = nullptr;
        GR_CK(cudaStreamBeginCapture(E.stream, cudaStreamCaptureModeThreadLocal));
        cudaError_t e = E.enqueue();
        cudaError_t e2 = cudaStreamEndCapture(E.stream, &gr);
        if (e != cudaSuccess) {
            if (gr) cudaGraphDestroy(gr);
            GR_CK(e);
        }
        GR_CK(e2);
        e = cudaGraphInstantiate(&E.graph, gr, 0);
        cudaGraphDestroy(gr);
        GR_CK(e);
    }
    for (int64_t off = 0; off < nstr; off += E.cap) {
        const int64_t nb = std::min<int64_t>(E.cap, nstr - off);
        const int64_t launches = (nb + E.bs - 1) / E.bs;   // the last launch's unused slots run all-zero strings
        GR_CK(cudaMemcpyAsync(E.d_bits, bits + off * ns, (size_t)(nb * ns), cudaMemcpyHostToDevice, E.stream));
        if (launches * E.bs > nb)
            GR_CK(cudaMemsetAsync(E.d_bits + nb * ns, 0, (size_t)((launches * E.bs - nb) * ns), E.stream));
        k_gr_set_item<<<1, 1, 0, E.stream>>>(E.d_item, 0);
        GR_CK(cudaGetLastError());
        for (int64_t i = 0; i < launches; i++) GR_CK(cudaGraphLaunch(E.graph, E.stream));
        GR_CK(cudaMemcpyAsync(z + 2 * off, E.d_z, (size_t)nb * 16, cudaMemcpyDeviceToHost, E.stream));
        GR_CK(cudaMemcpyAsync(dz + off * ns * 4, E.d_grad, (size_t)(nb * ns) * 4 * sizeof(double),
                              cudaMemcpyDeviceToHost, E.stream));
        GR_CK(cudaStreamSynchronize(E.stream));
    }
    return 0;
}

int gsb_grad_info(const gsb_grad *h, int *n, int *nsteps, int *R) {
    if (!h) return fail(GSB_E_STATE, "null handle");
    if (n) *n = h->E.plan.n;
    if (nsteps) *nsteps = h->E.plan.ns;
    if (R) *R = h->E.plan.R;
    return 0;
}

}  // extern "C"
