// Batched evaluation of many instances of uneven width in one persistent launch (the batching form).
//
// Work: for every instance i (its own in-place plan, ns_i steps, width R_i) and each of its npre prefixes, the
// forced bits of steps [0, K_i) are applied once, the live table before step K_i is kept, and each of nsuf suffixes
// resumes from it through steps [K_i, ns_i): one log2 Pr per (prefix, suffix) string.  Strings that share a prefix
// share its DP work (the reference's prefix / resume, gsamp2.cpp:162-208, done in memory).
//
// A work item is (instance, prefix).  Items sit in three queues, each sorted by decreasing cost: the widest instances are
// run by a cluster of CTAs ("cluster team"), wide ones by a CTA ("block team"), narrow ones (R <= small_R) by one warp
// ("warp team").  The kernel is persistent: every cluster first takes cluster items, then each of its CTAs block items,
// then each warp warp items, with one atomic per item.  A team owns an arena of 2^R entries and a second table of the
// same size in its slot, so a whole item runs without any grid-wide synchronisation.  Warp items of up to width BATCH_NEAR_R
// have both in shared memory and a function of their own (near_item), one step per pass.
//
// An item's steps run in passes of up to three (gsb_fuse.h), which read and write the table once: a thread takes a few
// classes at a time through the pass's steps, and their values between two steps sit in shared-memory slots of its own.
// Each step's code is compiled for its dataflow shape and member count (step_chunk).  The last pass of the prefix writes the
// second table and the first pass of every suffix reads it, so the table that the suffixes share is neither saved nor
// restored.  After a pass the team sums the written norm; the one-pass chain logic (power-of-two rescaling,
// gsamp2.cpp:59-70) runs redundantly in every thread of the team.
// Block size, the narrow-width threshold and CTAs per SM are chosen by an autotuner that times the actual batch; each
// shape's launch is captured once as a CUDA graph (queue reset + kernel).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <exception>
#include <map>
#include <new>
#include <string>
#include <thread>
#include <tuple>
#include <vector>

#include "gsb.h"
#include "gsb_common.h"
#include "gsb_fuse.h"
#include "gsb_plan.h"
#include "gsb_step.h"

namespace gsb {

namespace cg = cooperative_groups;

// Shape of a step's dataflow: with m = 2 and every x = 1 term in the other output than its offset's x = 0 term, the host
// orders the offsets so that the x = 0 terms of the first NTQ - H go to output 0 and those of the last H to output 1
// (relabelling the outputs where that makes H <= NTQ / 2).  BK_ANY: everything else, with runtime tables.
enum { BK_ANY = 0, BK_1_0, BK_2_0, BK_2_1, BK_4_0, BK_4_1, BK_4_2 };

// One step inside a pass.  Every stage's values are numbered so that member j reads values ntq j + t; out[j][tau]: the
// number of its outputs in the next stage (m j + tau in the last one).  Class sign: parity(class & lam) ^ bit j of mpar.
struct BStep {
    double M[8];             // M[b][x] (re, im)
    uint32_t lam, mpar;
    int kind, nmem, ntq, m;
    int tau0, tau1, par;     // bit t: offset t's x = 0 / x = 1 output, x = 1 sign
    unsigned char out[16][2];
    int pad;
};

// A pass of d steps: class p has base address XOR of col[j] over the bits of p; its value i of the first (last) stage
// sits at base ^ zin[i] (zout[i]).  mid[s]: values of the stage after step s (s < d - 1), chunk: classes taken at a time.
struct alignas(16) BPass {
    int d, nb, chunk, mid[2];
    uint32_t col[24], zin[32], zout[32];
    BStep st[FUSE_MAX_STEPS];
};
static_assert(sizeof(BPass) % 16 == 0, "descriptors are copied in 16-byte words");
constexpr int BATCH_WORDS = (int)(sizeof(BPass) / 16), BATCH_NEAR_WORDS = 32;   // of a descriptor; of one with a single step
static_assert(offsetof(BPass, st) + sizeof(BStep) <= 16 * BATCH_NEAR_WORDS, "one word per lane of a warp");
// Slots of a thread: the values between two steps of a chunk's classes.  More classes per chunk spread a step's
// descriptor loads over more work, fewer leave room for more CTAs: 512 instances of widths 7-20 in complex64 took 22.7,
// 21.8 and 41 ms at 128, 256 and 512 B.
constexpr int BATCH_SLOT_BYTES = 256;
constexpr int BATCH_CLUSTER = 8;      // CTAs of a cluster team
constexpr int BATCH_MAX_BLOCK = 512;
// Instances up to this width take one step per pass, and a warp keeps both tables of their items in its lanes' slots (2^8
// entries of complex128 twice: 8 KB).  A warp's item is a chain of dependent passes with a table read in each, so what bounds
// it is the latency of those reads and of the code between them: through L2, and through the code of the wide passes, 320
// items of widths 1-3 took 67 us in complex64 and 75 us in complex128 (single steps with generic code 43 and 41 us, now 23 and
// 23), 4,000 items of widths 5-9 321 and 376 us (226 and 227; now 162 and 205).
constexpr int BATCH_NEAR_R = 8;

struct BInst {
    int ns, R, K, n;
    int list_off, npass[2];  // in the list of passes: those of the prefix, then those of a suffix
    int first[2];            // the first pass of each
    int64_t pre_off;         // prefix bits: [npre][K]
    int64_t suf_off;         // suffix bits: [npre][nsuf][ns - K]
    int64_t out_off;         // log2 Pr: [npre][nsuf]
};

struct BatchArgs {
    const BPass *passes;     // every pass that some prefix length has needed
    const BInst *inst;
    const int *list;         // the passes of the current prefix lengths, by instance
    const int *items_wide, *items_big, *items_small;   // item = inst * npre + prefix
    int n_wide, n_big, n_small, npre, nsuf;
    const int8_t *pre_bits, *suf_bits;
    double *log2p;
    unsigned int *queues;    // [0] block-team queue, [1] warp-team queue, [2] cluster-team queue
    void *wide_arena;        // per cluster: two tables of 2^wide_R entries
    void *big_arena;         // per CTA: two tables of 2^big_R entries
    void *small_arena;       // per warp: two tables of 2^small_R entries
    int wide_R, big_R, small_R;
};

// Teams.  sum() gives every thread the same total (fixed order) and is also the barrier between two passes: partial sums
// alternate between two buffers, so a block needs one __syncthreads and a cluster one cluster barrier per pass.
struct BlockTeam {
    static constexpr bool WARP = false;
    int buf = 0;
    __device__ int rank() const { return threadIdx.x; }
    __device__ int size() const { return blockDim.x; }
    __device__ int log2size() const { return __ffs((int)blockDim.x) - 1; }   // blockDim.x: a power of two
    __device__ int local() const { return threadIdx.x; }     // threads that share this block's descriptor buffers
    __device__ int nlocal() const { return blockDim.x; }
    __device__ void sync() const { __syncthreads(); }
    __device__ double sum(double v) {
        __shared__ double red[2][BATCH_MAX_BLOCK / 32];
        v = warp_sum(v);
        const int nw = (int)(blockDim.x >> 5);
        if ((threadIdx.x & 31) == 0) red[buf][threadIdx.x >> 5] = v;
        __syncthreads();
        double t = 0;
        for (int i = 0; i < nw; i++) t += red[buf][i];
        buf ^= 1;
        return t;
    }
};

struct WarpTeam {
    static constexpr bool WARP = true;
    __device__ int rank() const { return threadIdx.x & 31; }
    __device__ int size() const { return 32; }
    __device__ int log2size() const { return 5; }
    __device__ int local() const { return threadIdx.x & 31; }
    __device__ int nlocal() const { return 32; }
    __device__ void sync() const { __syncwarp(); }
    __device__ double sum(double v) const {
        __syncwarp();
        return warp_sum(v);
    }
};

// The CTAs of a cluster.
struct ClusterTeam {
    static constexpr bool WARP = false;
    int buf = 0;
    __device__ int rank() const { return (int)(cg::this_cluster().block_rank() * blockDim.x + threadIdx.x); }
    __device__ int size() const { return (int)(cg::this_cluster().num_blocks() * blockDim.x); }
    __device__ int log2size() const { return __ffs(size()) - 1; }
    __device__ int local() const { return threadIdx.x; }
    __device__ int nlocal() const { return blockDim.x; }
    __device__ void sync() const { cg::this_cluster().sync(); }
    __device__ double sum(double v) {
        __shared__ double red[2][BATCH_MAX_BLOCK / 32], part[2][BATCH_CLUSTER];
        cg::cluster_group cl = cg::this_cluster();
        v = warp_sum(v);
        const int nw = (int)(blockDim.x >> 5), nc = (int)cl.num_blocks();
        if ((threadIdx.x & 31) == 0) red[buf][threadIdx.x >> 5] = v;
        __syncthreads();
        if ((int)threadIdx.x < nc) {   // thread i tells CTA i
            double t = 0;
            for (int i = 0; i < nw; i++) t += red[buf][i];
            *cl.map_shared_rank(&part[buf][cl.block_rank()], (int)threadIdx.x) = t;
        }
        cl.sync();
        double t = 0;
        for (int i = 0; i < nc; i++) t += part[buf][i];
        buf ^= 1;
        return t;
    }
};

template <typename E> struct ArithOf;
template <> struct ArithOf<float2> { typedef float T; };
template <> struct ArithOf<double2> { typedef double T; };

__device__ __forceinline__ float2 mk2(float r, float i) { return make_float2(r, i); }
__device__ __forceinline__ double2 mk2(double r, double i) { return make_double2(r, i); }
__device__ __forceinline__ float signed_by(float x, int neg) { return __int_as_float(__float_as_int(x) ^ (neg << 31)); }
__device__ __forceinline__ double signed_by(double x, int neg) {
    return __hiloint2double(__double2hiint(x) ^ (neg << 31), __double2loint(x));
}

// Classes n0 .. n0 + cn - 1 of a thread's walk: rank | (gray(n) << ls), the first one at `base` with index `cls`.
struct Chunk {
    uint32_t base, cls, n0, cn;
    int ls;
};
__device__ __forceinline__ void chunk_next(const BPass &p, const Chunk &k, uint32_t n, uint32_t &base, uint32_t &cls) {
    const int j = k.ls + __ffs((int)n) - 1;   // gray(n) = gray(n - 1) ^ 2^ctz(n)
    base ^= p.col[j];
    cls ^= 1u << j;
}

// What bounds the launch is the latency of the table reads (16 warps per SM; 27 % of the issue slots, a quarter of the HBM
// peak), so reads are issued early.  Measured against single-step passes with generic code: 96 instances of widths 7-20
// 12.0 -> 4.6 ms in complex64 and 17.7 -> 6.3 ms in complex128, 512 instances 46.2 -> 21.8 ms; fused passes with runtime
// tables alone took 7.1 ms and 32 ms (3.3 times the instructions).  Twice the warps at 64 registers measured the same.
//
// A shaped step on the classes of a chunk.  FIRST reads the table, other steps
// slots a..; LAST writes the table and returns the squared norm written, other steps slots b... NM: members, 0 for
// a runtime count.  The step's offsets, signs and row stay in registers for the whole chunk.
template <typename E, typename T, int NTQ, int H, int NM, bool FIRST, bool LAST>
__device__ __noinline__ double step_chunk(const BPass &p, const BStep &s, const int8_t *bit, double scale, const E *in,
                                          E *out, E *slots, int stride, int a, int b, const Chunk k) {
    const double *M = s.M + 4 * bit[0];
    const T m0r = (T)(scale * M[0]), m0i = (T)(scale * M[1]), m1r = (T)(scale * M[2]), m1i = (T)(scale * M[3]);
    T sg[NTQ];
#pragma unroll
    for (int t = 0; t < NTQ; t++) sg[t] = (s.par >> t) & 1 ? (T)-1 : (T)1;
    const uint32_t lam = s.lam, mpar = s.mpar;
    constexpr int MU = NM ? NM : 1;
    uint32_t zi[MU][NTQ], zo[MU][2];   // NM > 0: the members' offsets, in registers
    if (NM)
#pragma unroll
        for (int j = 0; j < MU; j++) {
            if (FIRST)
#pragma unroll
                for (int t = 0; t < NTQ; t++) zi[j][t] = p.zin[NTQ * j + t];
#pragma unroll
            for (int tau = 0; tau < 2; tau++) zo[j][tau] = LAST ? p.zout[2 * j + tau] : (uint32_t)(s.out[j][tau] * stride);
        }
    const int nm = NM ? NM : s.nmem, sin = NTQ * nm, sout = 2 * nm;
    E *src = slots + a * stride, *dst = slots + b * stride;
    uint32_t base = k.base, cls = k.cls;
    double nb = 0;
    // the next class's values in registers (complex64: up to 8; complex128 values took registers and ran 10 % slower)
    constexpr bool UPFRONT = sizeof(E) == 8;
    constexpr bool AHEAD = FIRST && NM > 0 && NM * NTQ <= 8 && sizeof(E) == 8;
    E v[MU][NTQ], ahead[AHEAD ? MU : 1][NTQ];
    auto load = [&](uint32_t at, E (&x)[MU][NTQ]) {
#pragma unroll
        for (int j = 0; j < MU; j++)
#pragma unroll
            for (int t = 0; t < NTQ; t++) x[j][t] = in[at ^ zi[j][t]];
    };
    if constexpr (AHEAD) load(base, ahead);
    for (uint32_t n = k.n0;;) {
        const int cs = __popc(cls & lam);
        T nn = 0;
        auto member = [&](int j, const E (&v)[NTQ], const uint32_t (&oj)[2]) {
            // x = 0 sums (X) and signed x = 1 sums (Z) of the two outputs
            T Xr[2] = {0, 0}, Xi[2] = {0, 0}, Zr[2] = {0, 0}, Zi[2] = {0, 0};
#pragma unroll
            for (int t = 0; t < NTQ; t++) {
                const int o = t < NTQ - H ? 0 : 1;
                const bool f = t == 0 || (H > 0 && t == NTQ - H);   // the first term of its sums
                Xr[o] = f ? v[t].x : Xr[o] + v[t].x;
                Xi[o] = f ? v[t].y : Xi[o] + v[t].y;
                Zr[1 - o] = f ? sg[t] * v[t].x : fma(sg[t], v[t].x, Zr[1 - o]);
                Zi[1 - o] = f ? sg[t] * v[t].y : fma(sg[t], v[t].y, Zi[1 - o]);
            }
            const int neg = (cs ^ (int)(mpar >> j)) & 1;
            const T wr = signed_by(m1r, neg), wi = signed_by(m1i, neg);
#pragma unroll
            for (int tau = 0; tau < 2; tau++) {
                T re, im;
                if (H == 0 && tau == 0) {          // x = 0 terms only
                    re = m0r * Xr[0] - m0i * Xi[0];
                    im = m0r * Xi[0] + m0i * Xr[0];
                } else if (H == 0) {               // x = 1 terms only
                    re = wr * Zr[1] - wi * Zi[1];
                    im = wr * Zi[1] + wi * Zr[1];
                } else {
                    re = m0r * Xr[tau] - m0i * Xi[tau] + wr * Zr[tau] - wi * Zi[tau];
                    im = m0r * Xi[tau] + m0i * Xr[tau] + wr * Zi[tau] + wi * Zr[tau];
                }
                if (LAST) {
                    out[base ^ oj[tau]] = mk2(re, im);
                    nn += re * re + im * im;
                } else {
                    dst[oj[tau]] = mk2(re, im);
                }
            }
        };
        uint32_t nbase = base, ncls = cls;
        const bool more = n + 1 < k.n0 + k.cn;
        if (more) chunk_next(p, k, n + 1, nbase, ncls);
        if constexpr (NM > 0) {
            // every value of the class is loaded before any is used, and with AHEAD the next class's as well: a few dozen
            // warps per SM have to cover the L2 and HBM latency
            if constexpr (AHEAD) {
#pragma unroll
                for (int j = 0; j < MU; j++)
#pragma unroll
                    for (int t = 0; t < NTQ; t++) v[j][t] = ahead[j][t];
                if (more) load(nbase, ahead);
            } else if constexpr (FIRST && UPFRONT) {
                load(base, v);
            } else if constexpr (!FIRST) {
#pragma unroll
                for (int j = 0; j < MU; j++)
#pragma unroll
                    for (int t = 0; t < NTQ; t++) v[j][t] = src[(NTQ * j + t) * stride];
            }
#pragma unroll
            for (int j = 0; j < NM; j++) {
                if constexpr (FIRST && !UPFRONT)
#pragma unroll
                    for (int t = 0; t < NTQ; t++) v[j][t] = in[base ^ zi[j][t]];
                member(j, v[j], zo[j]);
            }
        } else {
            for (int j = 0; j < nm; j++) {
#pragma unroll
                for (int t = 0; t < NTQ; t++)
                    v[0][t] = FIRST ? in[base ^ p.zin[NTQ * j + t]] : src[(NTQ * j + t) * stride];
#pragma unroll
                for (int tau = 0; tau < 2; tau++) zo[0][tau] = LAST ? p.zout[2 * j + tau] : (uint32_t)(s.out[j][tau] * stride);
                member(j, v[0], zo[0]);
            }
        }
        nb += (double)nn;
        n++;
        if (!more) break;
        base = nbase;
        cls = ncls;
        if (!FIRST) src += sin * stride;
        if (!LAST) dst += sout * stride;
    }
    return nb;
}

// The same for any step (runtime tables; one or two outputs).
template <typename E, typename T, bool FIRST, bool LAST>
__device__ __noinline__ double step_chunk_any(const BPass &p, const BStep &s, const int8_t *bit, double scale, const E *in,
                                              E *out, E *slots, int stride, int a, int b, const Chunk k) {
    const double *M = s.M + 4 * bit[0];
    const T m0r = (T)(scale * M[0]), m0i = (T)(scale * M[1]), m1r = (T)(scale * M[2]), m1i = (T)(scale * M[3]);
    const int ntq = s.ntq, m = s.m, nm = s.nmem;
    E *src = slots + a * stride, *dst = slots + b * stride;
    uint32_t base = k.base, cls = k.cls;
    double nb = 0;
    for (uint32_t n = k.n0;;) {
        T nn = 0;
        for (int j = 0; j < nm; j++) {
            T a0r = 0, a0i = 0, a1r = 0, a1i = 0, b0r = 0, b0i = 0, b1r = 0, b1i = 0;
            for (int t = 0; t < ntq; t++) {
                const E v = FIRST ? in[base ^ p.zin[ntq * j + t]] : src[(ntq * j + t) * stride];
                if ((s.tau0 >> t) & 1) { a1r += v.x; a1i += v.y; } else { a0r += v.x; a0i += v.y; }
                const T yr = signed_by(v.x, (s.par >> t) & 1), yi = signed_by(v.y, (s.par >> t) & 1);
                if ((s.tau1 >> t) & 1) { b1r += yr; b1i += yi; } else { b0r += yr; b0i += yi; }
            }
            const int neg = (__popc(cls & s.lam) ^ (int)(s.mpar >> j)) & 1;
            const T wr = signed_by(m1r, neg), wi = signed_by(m1i, neg);
            for (int tau = 0; tau < m; tau++) {
                const T xr = tau ? a1r : a0r, xi = tau ? a1i : a0i, zr = tau ? b1r : b0r, zi = tau ? b1i : b0i;
                const T re = m0r * xr - m0i * xi + wr * zr - wi * zi, im = m0r * xi + m0i * xr + wr * zi + wi * zr;
                if (LAST) {
                    out[base ^ p.zout[m * j + tau]] = mk2(re, im);
                    nn += re * re + im * im;
                } else {
                    dst[s.out[j][tau] * stride] = mk2(re, im);
                }
            }
        }
        nb += (double)nn;
        if (++n >= k.n0 + k.cn) break;
        chunk_next(p, k, n, base, cls);
        if (!FIRST) src += ntq * nm * stride;
        if (!LAST) dst += m * nm * stride;
    }
    return nb;
}

template <typename E, typename T, bool FIRST, bool LAST>
__device__ __forceinline__ double step_on(const BPass &p, const BStep &s, const int8_t *bit, double scale, const E *in, E *out,
                                          E *slots, int stride, int a, int b, const Chunk &k) {
#define GSB_BK(KIND, NTQ, H)                                                                                       \
    case KIND:                                                                                                     \
        switch (s.nmem) {                                                                                          \
            case 1: return step_chunk<E, T, NTQ, H, 1, FIRST, LAST>(p, s, bit, scale, in, out, slots, stride, a, b, k); \
            case 2: return step_chunk<E, T, NTQ, H, 2, FIRST, LAST>(p, s, bit, scale, in, out, slots, stride, a, b, k); \
            case 4: return step_chunk<E, T, NTQ, H, 4, FIRST, LAST>(p, s, bit, scale, in, out, slots, stride, a, b, k); \
            default: return step_chunk<E, T, NTQ, H, 0, FIRST, LAST>(p, s, bit, scale, in, out, slots, stride, a, b, k); \
        }
    switch (s.kind) {
        GSB_BK(BK_1_0, 1, 0)
        GSB_BK(BK_2_0, 2, 0)
        GSB_BK(BK_2_1, 2, 1)
        GSB_BK(BK_4_0, 4, 0)
        GSB_BK(BK_4_1, 4, 1)
        GSB_BK(BK_4_2, 4, 2)
        default: return step_chunk_any<E, T, FIRST, LAST>(p, s, bit, scale, in, out, slots, stride, a, b, k);
    }
#undef GSB_BK
}

// One pass of a team from the table `in` to the table `out` (the same one, or the item's other one), the first step's
// outputs scaled; returns the squared norm of this thread's outputs.
template <typename E>
__device__ __noinline__ double team_pass(const BPass &p, uint32_t r, int ls, const E *in, E *out, const int8_t *bits,
                                         double scale, E *slots, int stride) {
    typedef typename ArithOf<E>::T T;
    if (p.nb < ls && r >= (1u << p.nb)) return 0;
    Chunk k;
    k.base = 0;
    k.cls = r;
    k.ls = ls;
    for (int j = 0; j < min(p.nb, ls); j++)
        if ((r >> j) & 1) k.base ^= p.col[j];
    const uint32_t count = p.nb > ls ? 1u << (p.nb - ls) : 1;
    k.cn = min(count, (uint32_t)p.chunk);   // powers of two
    double nb = 0;
    for (k.n0 = 0; k.n0 < count; k.n0 += k.cn) {
        if (k.n0) {
            // from the previous chunk's first class: gray(n0) ^ gray(n0 - cn) has the bits log2 cn - 1 (cn > 1) and above
            const uint32_t f = k.n0 - k.cn, d = (k.n0 ^ (k.n0 >> 1)) ^ (f ^ (f >> 1));
            for (uint32_t x = d; x; x &= x - 1) k.base ^= p.col[ls + __ffs((int)x) - 1];
            k.cls ^= d << ls;
        }
        const int b1 = 0, b2 = (int)k.cn * p.mid[0];
        if (p.d == 1) {
            nb += step_on<E, T, true, true>(p, p.st[0], bits, scale, in, out, slots, stride, 0, 0, k);
        } else {
            step_on<E, T, true, false>(p, p.st[0], bits, scale, in, out, slots, stride, 0, b1, k);
            if (p.d == 2) {
                nb += step_on<E, T, false, true>(p, p.st[1], bits + 1, 1.0, in, out, slots, stride, b1, 0, k);
            } else {
                step_on<E, T, false, false>(p, p.st[1], bits + 1, 1.0, in, out, slots, stride, b1, b2, k);
                nb += step_on<E, T, false, true>(p, p.st[2], bits + 2, 1.0, in, out, slots, stride, b2, 0, k);
            }
        }
    }
    return nb;
}

// A pass of one step by a warp, of at most 2^BATCH_NEAR_R classes: short code for any shape with NTQ offsets.  The classes are
// the step's cosets; columns past the last one are 0.
template <typename E, int NTQ>
__device__ __forceinline__ double near_step(const BPass &p, const E *in, E *out, int bit, double scale) {
    typedef typename ArithOf<E>::T T;
    const BStep &s = p.st[0];
    const uint32_t r = threadIdx.x & 31;
    if (r >> min(p.nb, 5)) return 0;
    uint32_t base = 0, cls = r, z[NTQ];
#pragma unroll
    for (int j = 0; j < 5; j++)
        if ((r >> j) & 1) base ^= p.col[j];
#pragma unroll
    for (int t = 0; t < NTQ; t++) z[t] = p.zin[t];
    const uint32_t z0 = p.zout[0], z1 = p.zout[1], lam = s.lam, count = p.nb > 5 ? 1u << (p.nb - 5) : 1;
    const int m = s.m, tau0 = s.tau0, tau1 = s.tau1, par = s.par ^ (s.mpar & 1 ? (1 << NTQ) - 1 : 0);
    const double *M = s.M + 4 * bit;
    const T m0r = (T)(scale * M[0]), m0i = (T)(scale * M[1]), m1r = (T)(scale * M[2]), m1i = (T)(scale * M[3]);
    double nb = 0;
    for (uint32_t n = 0;;) {
        E v[NTQ];
#pragma unroll
        for (int t = 0; t < NTQ; t++) v[t] = in[base ^ z[t]];
        T a0r = 0, a0i = 0, a1r = 0, a1i = 0, b0r = 0, b0i = 0, b1r = 0, b1i = 0;
#pragma unroll
        for (int t = 0; t < NTQ; t++) {
            if ((tau0 >> t) & 1) { a1r += v[t].x; a1i += v[t].y; } else { a0r += v[t].x; a0i += v[t].y; }
            const int neg = (par >> t) & 1;
            const T yr = signed_by(v[t].x, neg), yi = signed_by(v[t].y, neg);
            if ((tau1 >> t) & 1) { b1r += yr; b1i += yi; } else { b0r += yr; b0i += yi; }
        }
        const int neg = __popc(cls & lam) & 1;
        const T wr = signed_by(m1r, neg), wi = signed_by(m1i, neg);
        T re = m0r * a0r - m0i * a0i + wr * b0r - wi * b0i, im = m0r * a0i + m0i * a0r + wr * b0i + wi * b0r;
        out[base ^ z0] = mk2(re, im);
        T nn = re * re + im * im;
        if (m == 2) {
            re = m0r * a1r - m0i * a1i + wr * b1r - wi * b1i;
            im = m0r * a1i + m0i * a1r + wr * b1i + wi * b1r;
            out[base ^ z1] = mk2(re, im);
            nn += re * re + im * im;
        }
        nb += (double)nn;
        if (++n >= count) break;
        const int j = 5 + __ffs((int)n) - 1;
        base ^= p.col[j];
        cls ^= 1u << j;
    }
    return nb;
}
template <typename E>
__device__ __noinline__ double near_pass(const BPass &p, const E *in, E *out, int bit, double scale) {
    switch (p.st[0].ntq) {
        case 1: return near_step<E, 1>(p, in, out, bit, scale);
        case 2: return near_step<E, 2>(p, in, out, bit, scale);
        default: return near_step<E, 4>(p, in, out, bit, scale);
    }
}

// Norms: a class's squared outputs are summed in the arena's precision (at most 32 of them), classes and threads in FP64.  A
// pass's norm only picks the power of two that scales the next one; the result is the norm of the last step's single entry.
struct ChainState {
    double prev, lsc, scale;
    int ek, dead;
};

// The one-pass chain scalars after a write of norm nb (gsamp2.cpp:59-70, executor write_epilogue).
__device__ __forceinline__ void chain_update(ChainState &cs, double nb) {
    cs.lsc += cs.ek;
    cs.prev = nb;
    if (!(nb > 0)) {
        cs.dead = 1;
        return;
    }
    int ex = 0;
    frexp(nb, &ex);
    cs.ek = (ex - 1) >> 1;
    cs.scale = ldexp(1.0, -cs.ek);
}

// The n passes list[0 .. n - 1] of `passes` (the first is number p0) with their bits (the first pass's step first): read from
// `first`, otherwise the arena, the last one written to `last`, otherwise the arena.  desc: two descriptor buffers; the next
// pass's descriptor is fetched during a pass, its number in the pass before.  Ends behind a team barrier (the last sum): tables complete, buffers free.
template <typename E, typename TM>
__device__ void run_passes(TM &tm, const BPass *passes, const int *list, int p0, int n, int words, const int8_t *bits,
                           const E *first, E *arena, E *last, BPass *desc, E *slots, int stride, ChainState &cs) {
    constexpr int PER = (BATCH_WORDS + 31) / 32;
    const int l = tm.local(), nl = tm.nlocal();
    for (int i = l; i < words; i += nl) reinterpret_cast<int4 *>(desc)[i] = reinterpret_cast<const int4 *>(passes + p0)[i];
    int coming = n > 1 ? list[1] : 0;
    tm.sync();
    int k = 0;
    for (int i = 0; i < n; i++) {
        const BPass &p = desc[i & 1];
        int4 next[PER];
        if (i + 1 < n)
#pragma unroll
            for (int q = 0; q < PER; q++)
                if (l + q * nl < words) next[q] = reinterpret_cast<const int4 *>(passes + coming)[l + q * nl];
        coming = i + 2 < n ? list[i + 2] : 0;
        const E *from = i == 0 ? first : arena;
        E *to = i == n - 1 ? last : arena;
        double nb;
        if (TM::WARP && p.d == 1 && p.nb <= BATCH_NEAR_R && p.st[0].nmem == 1) nb = near_pass<E>(p, from, to, bits[k], cs.scale);
        else nb = team_pass<E>(p, (uint32_t)tm.rank(), tm.log2size(), from, to, bits + k, cs.scale, slots, stride);
        k += p.d;
        if (i + 1 < n)
#pragma unroll
            for (int q = 0; q < PER; q++)
                if (l + q * nl < words) reinterpret_cast<int4 *>(desc + ((i + 1) & 1))[l + q * nl] = next[q];
        chain_update(cs, tm.sum(nb));
        if (cs.dead) break;
    }
}

template <typename E, typename TM>
__device__ void run_item(TM &tm, const BatchArgs &a, int item, E *arena, E *kept, BPass *desc, E *slots, int stride) {
    const int ii = item / a.npre, pre = item % a.npre;
    const BInst in = a.inst[ii];
    const int8_t *pb = a.pre_bits + in.pre_off + (int64_t)pre * in.K;
    if (tm.rank() == 0) arena[0] = mk2((typename ArithOf<E>::T)1, (typename ArithOf<E>::T)0);
    ChainState cs{1.0, 0.0, 1.0, 0, 0};
    const int *list = a.list + in.list_off;
    const int words = in.R <= BATCH_NEAR_R ? BATCH_NEAR_WORDS : BATCH_WORDS;
    run_passes<E, TM>(tm, a.passes, list, in.first[0], in.npass[0], words, pb, arena, arena, kept, desc, slots, stride, cs);
    const ChainState at_k = cs;
    const int nsuf_steps = in.ns - in.K;
    for (int sidx = 0; sidx < a.nsuf; sidx++) {
        cs = at_k;
        double lp = -INFINITY;
        if (!cs.dead) {
            const int8_t *sb = a.suf_bits + in.suf_off + ((int64_t)pre * a.nsuf + sidx) * nsuf_steps;
            run_passes<E, TM>(tm, a.passes, list + in.npass[0], in.first[1], in.npass[1], words, sb, kept, arena, arena, desc,
                              slots, stride, cs);
            if (!cs.dead) lp = log2(cs.prev) + 2.0 * cs.lsc - in.n;
        }
        if (tm.rank() == 0) a.log2p[in.out_off + (int64_t)pre * a.nsuf + sidx] = lp;
    }
}

// The same for a near instance by a warp: every pass is one step, its descriptor one word per lane.
template <typename E>
__device__ __forceinline__ void near_passes(const BPass *passes, const int *list, int p0, int n, const int8_t *bits,
                                            const E *first, E *tab, E *last, BPass *desc, ChainState &cs) {
    const int lane = threadIdx.x & 31;
    reinterpret_cast<int4 *>(desc)[lane] = reinterpret_cast<const int4 *>(passes + p0)[lane];
    int bit = bits[0], coming = n > 1 ? list[1] : 0;
    __syncwarp();
#pragma unroll 1
    for (int i = 0; i < n; i++) {
        const BPass &p = desc[i & 1];
        int4 next = make_int4(0, 0, 0, 0);
        int next_bit = 0;
        if (i + 1 < n) {
            next = reinterpret_cast<const int4 *>(passes + coming)[lane];
            next_bit = bits[i + 1];
        }
        coming = i + 2 < n ? list[i + 2] : 0;
        const E *from = i == 0 ? first : tab;
        E *to = i == n - 1 ? last : tab;
        const int ntq = p.st[0].ntq;
        double nb;
        if (ntq == 1) nb = near_step<E, 1>(p, from, to, bit, cs.scale);
        else if (ntq == 2) nb = near_step<E, 2>(p, from, to, bit, cs.scale);
        else nb = near_step<E, 4>(p, from, to, bit, cs.scale);
        reinterpret_cast<int4 *>(desc + ((i + 1) & 1))[lane] = next;
        bit = next_bit;
        __syncwarp();
        chain_update(cs, warp_sum(nb));
        if (cs.dead) break;
    }
}
template <typename E>
__device__ __noinline__ void near_item(const BatchArgs &a, int item, E *tab, BPass *desc) {
    const int ii = item / a.npre, pre = item % a.npre;
    const BInst in = a.inst[ii];
    E *kept = tab + (1 << BATCH_NEAR_R);
    if ((threadIdx.x & 31) == 0) tab[0] = mk2((typename ArithOf<E>::T)1, (typename ArithOf<E>::T)0);
    ChainState cs{1.0, 0.0, 1.0, 0, 0};
    const int *list = a.list + in.list_off;
    near_passes<E>(a.passes, list, in.first[0], in.npass[0], a.pre_bits + in.pre_off + (int64_t)pre * in.K, tab, tab, kept, desc,
                   cs);
    const ChainState at_k = cs;
    const int nsuf_steps = in.ns - in.K;
    for (int sidx = 0; sidx < a.nsuf; sidx++) {
        cs = at_k;
        double lp = -INFINITY;
        if (!cs.dead) {
            near_passes<E>(a.passes, list + in.npass[0], in.first[1], in.npass[1],
                           a.suf_bits + in.suf_off + ((int64_t)pre * a.nsuf + sidx) * nsuf_steps, kept, tab, tab, desc, cs);
            if (!cs.dead) lp = log2(cs.prev) + 2.0 * cs.lsc - in.n;
        }
        if ((threadIdx.x & 31) == 0) a.log2p[in.out_off + (int64_t)pre * a.nsuf + sidx] = lp;
    }
}

// Dynamic shared memory of a block: two descriptors per warp (a block or cluster team uses the first two), then the
// threads' slots.
static size_t batch_smem(int block) {
    return (size_t)(block / 32) * 2 * sizeof(BPass) + (size_t)BATCH_SLOT_BYTES * (size_t)block;
}

constexpr size_t BATCH_MAX_SMEM = (227 << 10) - 2048;   // dynamic, beside the teams' static sums

template <typename E>
__global__ void __launch_bounds__(BATCH_MAX_BLOCK) k_batch(const __grid_constant__ BatchArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int warps = (int)(blockDim.x >> 5), w = (int)(threadIdx.x >> 5);
    BPass *desc = reinterpret_cast<BPass *>(smem);
    E *slots = reinterpret_cast<E *>(smem + (size_t)warps * 2 * sizeof(BPass)) + threadIdx.x;
    const int stride = (int)blockDim.x;
    __shared__ int s_item;
    if (a.n_wide > 0) {
        cg::cluster_group cl = cg::this_cluster();
        const size_t wide = (size_t)1 << a.wide_R;
        E *arena = reinterpret_cast<E *>(a.wide_arena) + (size_t)(blockIdx.x / cl.num_blocks()) * 2 * wide;
        ClusterTeam ct;
        for (;;) {
            if (cl.block_rank() == 0 && threadIdx.x == 0) {
                const int it = (int)atomicAdd(&a.queues[2], 1u);
                for (unsigned r = 0; r < cl.num_blocks(); r++) *cl.map_shared_rank(&s_item, r) = it;
            }
            cl.sync();
            const int it = s_item;
            cl.sync();
            if (it >= a.n_wide) break;
            run_item<E, ClusterTeam>(ct, a, a.items_wide[it], arena, arena + wide, desc, slots, stride);
        }
    }
    const size_t big = (size_t)1 << a.big_R, small = (size_t)1 << a.small_R;
    E *arena = reinterpret_cast<E *>(a.big_arena) + (size_t)blockIdx.x * 2 * big;
    BlockTeam bt;
    for (;;) {
        if (threadIdx.x == 0) s_item = (int)atomicAdd(&a.queues[0], 1u);
        __syncthreads();
        const int it = s_item;
        __syncthreads();
        if (it >= a.n_big) break;
        run_item<E, BlockTeam>(bt, a, a.items_big[it], arena, arena + big, desc, slots, stride);
    }
    E *wa = reinterpret_cast<E *>(a.small_arena) + ((size_t)blockIdx.x * warps + (size_t)w) * 2 * small;
    E *ws = reinterpret_cast<E *>(smem + (size_t)warps * 2 * sizeof(BPass)) + (size_t)w * (32 * BATCH_SLOT_BYTES / sizeof(E));
    WarpTeam wt;
    // Where there are narrow items only, every warp's first one is its own, dealt out over the blocks: the blocks that start
    // first would otherwise take eight each.
    const bool dealt = a.n_wide == 0 && a.n_big == 0;
    const int warps_all = (int)gridDim.x * warps;
    for (int it = dealt ? w * (int)gridDim.x + (int)blockIdx.x : -1;; it = -1) {
        if (it < 0) {
            if ((threadIdx.x & 31) == 0) it = (int)atomicAdd(&a.queues[1], 1u) + (dealt ? warps_all : 0);
            it = __shfl_sync(0xffffffffu, it, 0);
        }
        if (it >= a.n_small) break;
        const int item = a.items_small[it];
        if (a.inst[item / a.npre].R <= BATCH_NEAR_R) near_item<E>(a, item, ws, desc + 2 * w);
        else run_item<E, WarpTeam>(wt, a, item, wa, wa + small, desc + 2 * w, ws + (threadIdx.x & 31), 32);
    }
}

struct BatchShape {
    int block = 256, small_R = 12, per_sm = 2;
    bool operator<(const BatchShape &o) const {
        return std::tie(block, small_R, per_sm) < std::tie(o.block, o.small_R, o.per_sm);
    }
};

struct BatchEngine {
    int prec = 64, dev = 0, sms = 0;
    size_t esize = 8;
    std::vector<HPlan> plans;
    std::vector<int> K;             // prefix lengths that the list was made for
    struct Lists {
        int off, npre, nsuf, pre0, suf0;   // in the list; passes and first pass of the prefix and of a suffix
    };
    std::vector<Lists> lists;
    // per instance, entry 3 k + d - 1: the number of the pass of steps k .. k + d - 1 in d_passes, or one of these
    enum { UNKNOWN = -1, NO_PASS = -2 };
    std::vector<std::vector<int>> known;
    size_t table_n = 0, table_cap = 0;   // passes in d_passes, and room
    int *d_list = nullptr;
    std::vector<double> cost;       // per instance: entries moved by one prefix + its suffixes (relative)
    BPass *d_passes = nullptr;
    BInst *d_inst = nullptr;
    int *d_items = nullptr;
    int8_t *d_pre = nullptr, *d_suf = nullptr;
    double *d_out = nullptr;
    unsigned int *d_q = nullptr;
    void *d_arena = nullptr;
    size_t arena_bytes = 0;
    size_t limit = SIZE_MAX;        // of the arenas' bytes, where clusters can be done without (shape_layout)
    int npre = 0, nsuf = 0;
    int64_t pre_cap = 0, suf_cap = 0, out_cap = 0, out_total = 0;   // bytes, bytes, results: room; results set
    std::vector<BInst> h_inst;
    cudaStream_t stream = nullptr;
    BatchShape shape;
    bool tuned = false;
    std::map<BatchShape, cudaGraphExec_t> graphs;

    ~BatchEngine() {
        int prev = 0;
        cudaGetDevice(&prev);
        cudaSetDevice(dev);
        for (auto &kv : graphs) cudaGraphExecDestroy(kv.second);
        cudaFree(d_passes);
        cudaFree(d_list);
        cudaFree(d_inst);
        cudaFree(d_items);
        cudaFree(d_pre);
        cudaFree(d_suf);
        cudaFree(d_out);
        cudaFree(d_q);
        cudaFree(d_arena);
        if (stream) cudaStreamDestroy(stream);
        cudaSetDevice(prev);
    }

    int max_R() const {
        int r = 0;
        for (const HPlan &p : plans) r = std::max(r, p.R);
        return r;
    }
};

}  // namespace gsb

using namespace gsb;

#define BT_CK(x)                                                                                                  \
    do {                                                                                                          \
        cudaError_t e_ = (x);                                                                                     \
        if (e_ != cudaSuccess) return fail(GSB_E_CUDA, std::string("CUDA error: ") + cudaGetErrorString(e_) + " at " #x); \
    } while (0)

struct gsb_batch {
    BatchEngine E;
};

// Items of a shape: the widest instances to the cluster-team queue, wide ones to the block-team queue, narrow ones to the
// warp-team queue, each in decreasing cost, and the sizes of the team arenas.
struct BatchLayout {
    std::vector<int> wide, big, small;
    int wide_R = 0, big_R = 0, small_R = 0, grid = 0;
    size_t bytes = 0;
};
static BatchLayout team_layout(const BatchEngine &E, const BatchShape &sh, bool clusters) {
    BatchLayout L;
    std::vector<int> order(E.plans.size());
    for (size_t i = 0; i < order.size(); i++) order[i] = (int)i;
    std::sort(order.begin(), order.end(), [&](int x, int y) { return E.cost[(size_t)x] > E.cost[(size_t)y]; });
    L.grid = E.sms * sh.per_sm / BATCH_CLUSTER * BATCH_CLUSTER;
    // An item that would keep one CTA busy for longer than an even share of the whole batch goes to a cluster: a
    // cluster spends part of its time on barriers, so it pays only where one CTA would be the batch's tail.  Thresholds of
    // 1/4, 1/2, 1 and 2 shares took 5.6, 5.2, 4.7 and 5.6 ms on 96 instances of widths 7-20 (no clusters: 10 ms, the time of
    // one width-20 item), 27.4, 24.4, 21.8 and 21.8 ms on 512, 2.4, 0.79, 0.80 and 0.80 ms on 200 of widths up to 15.
    // Below width 15 a cluster's steps are barriers only (8 instances of width 12: 0.33 ms against 0.11 ms).
    double total = 0;
    for (double c : E.cost) total += c * E.npre;
    const double share = total / L.grid;
    for (int i : order) {
        const int R = E.plans[(size_t)i].R;
        const bool small = R <= sh.small_R, wide = clusters && !small && R >= 15 && E.cost[(size_t)i] > share;
        auto &q = small ? L.small : wide ? L.wide : L.big;
        for (int p = 0; p < E.npre; p++) q.push_back(i * E.npre + p);
        int &r = small ? L.small_R : wide ? L.wide_R : L.big_R;
        r = std::max(r, R);
    }
    const size_t warps = (size_t)L.grid * (size_t)(sh.block / 32);
    L.bytes = E.esize * 2 * ((L.wide.empty() ? 0 : (size_t)(L.grid / BATCH_CLUSTER) << L.wide_R) +
                             ((size_t)L.grid << L.big_R) + (warps << L.small_R));
    return L;
}

// Cluster teams have arenas of their own beside those of the block teams, which need no less where a second instance of the
// same width is left to them: within E.limit, or else the block teams take every wide instance if that needs less.
static BatchLayout shape_layout(const BatchEngine &E, const BatchShape &sh) {
    BatchLayout L = team_layout(E, sh, true);
    if (L.bytes > E.limit && !L.wide.empty()) {
        BatchLayout B = team_layout(E, sh, false);
        if (B.bytes < L.bytes) L = B;
    }
    return L;
}

// The pass of steps gp.k0 .. gp.k0 + gp.d - 1; false when one class's values between the steps exceed `slots`.
static bool make_pass(const HPlan &p, const GroupPlan &gp, int slots, BPass &g) {
    memset(&g, 0, sizeof g);
    int kept = 0;
    for (int s = 0; s + 1 < gp.d; s++) kept += g.mid[s] = gp.stage_size[s + 1];
    if (kept > slots || gp.nb > 24) return false;
    g.d = gp.d;
    g.nb = gp.nb;
    g.chunk = 1;
    while (g.chunk < 32 && 2 * g.chunk * kept <= slots) g.chunk *= 2;
    std::vector<uint64_t> cols;
    for (int j = 0; j < gp.L; j++) cols.push_back(1ULL << j);
    cols.insert(cols.end(), gp.bhi.begin(), gp.bhi.end());
    for (int j = 0; j < gp.nb; j++) g.col[j] = (uint32_t)cols[(size_t)j];
    std::vector<int> number[FUSE_MAX_STEPS + 1];   // of the plan's stage values: member-major in the step that reads them
    int perm[FUSE_MAX_STEPS][4], swp[FUSE_MAX_STEPS];
    for (int s = 0; s < gp.d; s++) {
        const HStep &hs = p.st[(size_t)(gp.k0 + s)];
        const GroupPlan::Step &q = gp.step[s];
        BStep &a = g.st[s];
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
        a.kind = BK_ANY;
        if (shaped && q.ntq == 1) a.kind = BK_1_0;
        else if (shaped && q.ntq == 2) a.kind = h == 0 ? BK_2_0 : BK_2_1;
        else if (shaped && q.ntq == 4) a.kind = h == 0 ? BK_4_0 : h == 1 ? BK_4_1 : BK_4_2;
        a.nmem = q.nmem;
        a.ntq = q.ntq;
        a.m = q.m;
        for (int b = 0; b < 2; b++)
            for (int x = 0; x < 2; x++) {
                a.M[4 * b + 2 * x] = hs.Mr[b][x];
                a.M[4 * b + 2 * x + 1] = hs.Mi[b][x];
            }
        for (int t = 0; t < q.ntq; t++) {
            a.tau0 |= (hs.tau0[perm[s][t]] ^ swp[s]) << t;
            a.tau1 |= (hs.tau1[perm[s][t]] ^ swp[s]) << t;
            a.par |= hs.par[perm[s][t]] << t;
        }
        for (int j = 0; j < gp.nb; j++)
            a.lam |= (uint32_t)(__builtin_popcountll(cols[(size_t)j] & q.lambda) & 1) << j;
        number[s].assign((size_t)gp.stage_size[s], 0);
        for (int j = 0; j < q.nmem; j++) {
            a.mpar |= (uint32_t)(q.mpar[j] & 1) << j;
            for (int t = 0; t < q.ntq; t++) number[s][(size_t)q.in_idx[j][perm[s][t]]] = q.ntq * j + t;
        }
    }
    for (int i = 0; i < gp.stage_size[0]; i++) g.zin[number[0][(size_t)i]] = (uint32_t)gp.z_in[(size_t)i];
    for (int s = 0; s < gp.d; s++) {
        const GroupPlan::Step &q = gp.step[s];
        for (int j = 0; j < q.nmem; j++)
            for (int tau = 0; tau < q.m; tau++) {
                const int old = q.out_idx[j][tau ^ swp[s]];
                if (s + 1 < gp.d) g.st[s].out[j][tau] = (unsigned char)number[s + 1][(size_t)old];
                else g.zout[q.m * j + tau] = (uint32_t)gp.z_out[(size_t)old];
            }
    }
    return true;
}

// Passes of steps k0 .. k1 - 1, each as long as its classes' slots allow, appended to `list`; pass_at(k, d): the number of the pass
// of steps k .. k + d - 1, or NO_PASS or UNKNOWN, which ends the list and is returned (as is NO_PASS where not even a single
// step fits; otherwise 0).  A narrow instance is run by one warp by default, and fusing leaves its lanes few classes with a
// long chain of work each: up to width 12 passes of several steps have at least 2^8 classes (300 instances of widths up to
// 12: 0.63 ms with any number of classes, 0.43 at 2^5, 0.36 at 2^8).  Block and cluster teams are faster fused throughout
// (60 instances of widths 8-14: 0.27 against 0.33 ms).
static int least_classes(const HPlan &p) { return p.R <= 12 ? 8 : 0; }
template <typename F>
static int passes_of(const HPlan &p, int k0, int k1, F pass_at, std::vector<int> &list) {
    const int least = least_classes(p);
    for (int k = k0; k < k1;) {
        int d = 1, pass = BatchEngine::NO_PASS;   // a pass has at most the 2^nk cosets of each of its steps as classes
        while (p.R > BATCH_NEAR_R && d < FUSE_MAX_STEPS && k + d < k1 &&
               std::min(p.st[(size_t)k].nk, p.st[(size_t)(k + d)].nk) >= least)
            d++;
        for (; d > 0 && (pass = pass_at(k, d)) == BatchEngine::NO_PASS; d--) {}
        if (pass < 0) return pass;
        list.push_back(pass);
        k += d;
    }
    return 0;
}

// The pass lists for prefix lengths K.  A pass is derived once, when a list first needs it (10 us; the host's cores side by
// side), and stays in the device's table: other prefix lengths need few new ones or none.  Two set_strings with other prefix
// lengths: 300 instances of widths 4-5 5.4 ms with a table made for each call, 100 of width 11 3.8 ms; now 0.5 and 0.23.
static int batch_passes(BatchEngine &E, const int *K) {
    const size_t n = E.plans.size();
    if (E.K.size() == n && std::equal(E.K.begin(), E.K.end(), K)) return 0;
    constexpr int FRESH = 1 << 28;   // a derived pass's number until it has one in the device's table
    const int slots = BATCH_SLOT_BYTES / (int)E.esize;
    if (E.known.empty())
        for (const HPlan &p : E.plans) E.known.emplace_back((size_t)(FUSE_MAX_STEPS * p.ns), BatchEngine::UNKNOWN);
    std::vector<std::vector<int>> rows(n);       // E.known with this call's passes, of the instances that needed some
    std::vector<std::vector<BPass>> derived(n);
    std::vector<int> list, off(n), pre(n);
    std::vector<size_t> todo;
    // the lists with the passes at hand; false: no pass fits a step of instance *bad
    auto assemble = [&](size_t *bad) {
        list.clear();
        todo.clear();
        for (size_t i = 0; i < n; i++) {
            const HPlan &p = E.plans[i];
            const std::vector<int> &row = rows[i].empty() ? E.known[i] : rows[i];
            auto at = [&](int k, int d) { return row[(size_t)(FUSE_MAX_STEPS * k + d - 1)]; };
            off[i] = (int)list.size();
            int rc = passes_of(p, 0, K[i], at, list);
            pre[i] = (int)list.size() - off[i];
            if (!rc) rc = passes_of(p, K[i], p.ns, at, list);
            *bad = i;
            if (rc == BatchEngine::NO_PASS) return false;
            if (rc) todo.push_back(i);
        }
        return true;
    };
    auto derive = [&](size_t i) {
        const HPlan &p = E.plans[i];
        std::vector<int> row = E.known[i], any;
        auto at = [&](int k, int d) {
            int &x = row[(size_t)(FUSE_MAX_STEPS * k + d - 1)];
            if (x != BatchEngine::UNKNOWN) return x;
            BPass g;
            GroupPlan gp;
            x = BatchEngine::NO_PASS;
            if (plan_group(p, k, d, 0, 24, gp) && (d == 1 || gp.nb >= least_classes(p)) && make_pass(p, gp, slots, g)) {
                x = FRESH + (int)derived[i].size();
                derived[i].push_back(g);
            }
            return x;
        };
        if (!passes_of(p, 0, K[i], at, any)) passes_of(p, K[i], p.ns, at, any);
        rows[i].swap(row);
    };
    size_t bad = 0;
    std::vector<BPass> fresh;
    bool fits = assemble(&bad);
    if (fits && !todo.empty()) {
        const unsigned nt = std::min({(unsigned)todo.size(), 16u, std::max(1u, std::thread::hardware_concurrency())});
        std::atomic<size_t> next{0};
        std::atomic<bool> memory{true};
        auto work = [&] {
            for (size_t j; (j = next++) < todo.size();) {
                try {
                    derive(todo[j]);
                } catch (const std::bad_alloc &) {
                    memory = false;
                }
            }
        };
        std::vector<std::thread> th;
        th.reserve(nt);
        try {
            for (unsigned t = 1; t < nt; t++) th.emplace_back(work);
        } catch (const std::exception &) {   // no more threads: those there are, and this one, take all instances
        }
        work();
        for (std::thread &t : th) t.join();
        if (!memory) return fail(GSB_E_ALLOC, "no host memory for the batch's passes");
        for (size_t i : todo) {
            for (int &x : rows[i])
                if (x >= FRESH) x += (int)(E.table_n + fresh.size()) - FRESH;
            fresh.insert(fresh.end(), derived[i].begin(), derived[i].end());
        }
        fits = assemble(&bad);
    }
    if (!fits) return fail(GSB_E_PLAN_LAYOUT, "instance " + std::to_string(bad) + " does not fit the batch kernel's passes");
    // until the new passes are on the device the engine keeps the old lists, with the offsets that belong to them
    const size_t need = E.table_n + fresh.size();
    cudaError_t e = cudaSuccess;
    if (!E.d_list) {   // at most one pass per step
        size_t steps = 0;
        for (const HPlan &p : E.plans) steps += (size_t)p.ns;
        e = cudaMalloc(&E.d_list, steps * sizeof(int));
    }
    if (e == cudaSuccess && need > E.table_cap) {
        const size_t cap = E.table_n ? need + need / 2 : need;
        BPass *d = nullptr;
        e = cudaMalloc(&d, cap * sizeof(BPass));
        if (e == cudaSuccess && E.table_n) e = cudaMemcpy(d, E.d_passes, E.table_n * sizeof(BPass), cudaMemcpyDeviceToDevice);
        if (e == cudaSuccess) {
            for (auto &kv : E.graphs) cudaGraphExecDestroy(kv.second);   // they point at the old table
            E.graphs.clear();
            cudaFree(E.d_passes);
            E.d_passes = d;
            E.table_cap = cap;
        } else {
            cudaFree(d);
        }
    }
    if (e == cudaSuccess && !fresh.empty())
        e = cudaMemcpy(E.d_passes + E.table_n, fresh.data(), fresh.size() * sizeof(BPass), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(E.d_list, list.data(), list.size() * sizeof(int), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return fail(GSB_E_CUDA, std::string("the batch's pass table: ") + cudaGetErrorString(e));
    E.table_n = need;
    for (size_t i = 0; i < n; i++)
        if (!rows[i].empty()) E.known[i].swap(rows[i]);
    E.lists.resize(n);
    for (size_t i = 0; i < n; i++) {
        const int end = i + 1 < n ? off[i + 1] : (int)list.size(), suf = off[i] + pre[i];
        E.lists[i] = BatchEngine::Lists{off[i], pre[i], end - suf, list[(size_t)off[i]], list[(size_t)suf]};
    }
    E.K.assign(K, K + n);
    return 0;
}

static int batch_graph(BatchEngine &E, const BatchShape &sh, cudaGraphExec_t *out) {
    auto it = E.graphs.find(sh);
    if (it != E.graphs.end()) {
        *out = it->second;
        return 0;
    }
    BatchLayout L = shape_layout(E, sh);
    if (L.bytes > E.arena_bytes) {
        cudaFree(E.d_arena);
        E.d_arena = nullptr;
        E.arena_bytes = 0;
        for (auto &kv : E.graphs) cudaGraphExecDestroy(kv.second);   // they point at the old arena
        E.graphs.clear();
        cudaError_t e = cudaMalloc(&E.d_arena, L.bytes);
        if (e == cudaErrorMemoryAllocation) {   // no room for the cluster teams' arenas: without them, from now on
            E.limit = L.bytes - 1;
            const size_t tried = L.bytes;
            L = shape_layout(E, sh);
            if (L.bytes < tried) {
                cudaGetLastError();
                e = cudaMalloc(&E.d_arena, L.bytes);
            }
        }
        if (e != cudaSuccess) E.d_arena = nullptr;
        BT_CK(e);
        E.arena_bytes = L.bytes;
    }
    for (auto &kv : E.graphs) cudaGraphExecDestroy(kv.second);   // they point at the old items
    E.graphs.clear();
    cudaFree(E.d_items);
    E.d_items = nullptr;
    std::vector<int> items(L.wide);
    items.insert(items.end(), L.big.begin(), L.big.end());
    items.insert(items.end(), L.small.begin(), L.small.end());
    BT_CK(cudaMalloc(&E.d_items, std::max<size_t>(items.size(), 1) * sizeof(int)));
    if (!items.empty())
        BT_CK(cudaMemcpy(E.d_items, items.data(), items.size() * sizeof(int), cudaMemcpyHostToDevice));
    BatchArgs a;
    a.passes = E.d_passes;
    a.inst = E.d_inst;
    a.list = E.d_list;
    a.items_wide = E.d_items;
    a.items_big = a.items_wide + L.wide.size();
    a.items_small = a.items_big + L.big.size();
    a.n_wide = (int)L.wide.size();
    a.n_big = (int)L.big.size();
    a.n_small = (int)L.small.size();
    a.npre = E.npre;
    a.nsuf = E.nsuf;
    a.pre_bits = E.d_pre;
    a.suf_bits = E.d_suf;
    a.log2p = E.d_out;
    a.queues = E.d_q;
    char *mem = static_cast<char *>(E.d_arena);
    a.wide_arena = mem;
    if (a.n_wide) mem += E.esize * 2 * ((size_t)(L.grid / BATCH_CLUSTER) << L.wide_R);
    a.big_arena = mem;
    a.small_arena = mem + E.esize * 2 * ((size_t)L.grid << L.big_R);
    a.wide_R = L.wide_R;
    a.big_R = L.big_R;
    a.small_R = L.small_R;
    const size_t smem = batch_smem(sh.block);
    const void *fn = E.prec == 128 ? (const void *)k_batch<double2> : (const void *)k_batch<float2>;
    // asked for here and not in an open, which would load both precisions' kernels
    BT_CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BATCH_MAX_SMEM));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)L.grid);
    cfg.blockDim = dim3((unsigned)sh.block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = E.stream;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = BATCH_CLUSTER;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = a.n_wide ? 1 : 0;   // clusters only where an item needs one
    cudaGraph_t g = nullptr;
    BT_CK(cudaStreamBeginCapture(E.stream, cudaStreamCaptureModeThreadLocal));
    cudaMemsetAsync(E.d_q, 0, 3 * sizeof(unsigned int), E.stream);
    void *kargs[] = {&a};
    const cudaError_t e0 = cudaLaunchKernelExC(&cfg, fn, kargs);
    cudaError_t e = e0;
    cudaError_t e2 = cudaStreamEndCapture(E.stream, &g);
    if (e != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        BT_CK(e);
    }
    BT_CK(e2);
    cudaGraphExec_t ex = nullptr;
    e = cudaGraphInstantiate(&ex, g, 0);
    cudaGraphDestroy(g);
    BT_CK(e);
    E.graphs[sh] = ex;
    *out = ex;
    return 0;
}

extern "C" {

int gsb_batch_open(const char *const *texts, const size_t *lens, int ninst, int precision, int device, gsb_batch **out) {
    if (!texts || !lens || !out || ninst < 1) return fail(GSB_E_USAGE, "bad argument");
    *out = nullptr;
    if (precision != 64 && precision != 128) return fail(GSB_E_USAGE, "precision must be 64 or 128");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) return fail(GSB_E_CUDA, "no CUDA device is visible");
    if (device < 0 || device >= ndev) return fail(GSB_E_USAGE, "device out of range");
    gsb_batch *h = new gsb_batch();
    BatchEngine &E = h->E;
    E.prec = precision;
    E.esize = precision == 128 ? 16 : 8;
    E.dev = device;
    E.plans.resize((size_t)ninst);
    for (int i = 0; i < ninst; i++) {
        std::string err;
        int rc = parse_plan_text(texts[i], lens[i], E.plans[(size_t)i], err);
        if (!rc) rc = validate_plan(E.plans[(size_t)i], err);
        if (!rc && E.plans[(size_t)i].ns < 2) {
            rc = GSB_E_USAGE;
            err = "a batched instance needs at least 2 steps";
        }
        if (!rc && E.plans[(size_t)i].R > 24) {
            rc = GSB_E_USAGE;
            err = "batched instances are limited to width 24 (one team arena each)";
        }
        if (rc) {
            delete h;
            return fail(rc, "instance " + std::to_string(i) + ": " + err);
        }
    }
    for (const HPlan &p : E.plans) {
        double c = 0;
        for (int k = 0; k < p.ns; k++) {
            const HStep &s = p.st[(size_t)k];
            c += std::ldexp(1.0, s.nk) * (double)((int)s.tqs.size() + s.m);
        }
        E.cost.push_back(c);
    }
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    struct Restore {
        int p;
        ~Restore() { cudaSetDevice(p); }
    } restore{prev};
    cudaDeviceGetAttribute(&E.sms, cudaDevAttrMultiProcessorCount, device);
    cudaError_t e = cudaStreamCreateWithFlags(&E.stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&E.d_q, 3 * sizeof(unsigned int));
    if (e != cudaSuccess) {
        delete h;
        return fail(GSB_E_ALLOC, std::string("device allocation: ") + cudaGetErrorString(e));
    }
    *out = h;
    return 0;
}

int gsb_batch_close(gsb_batch *h) {
    delete h;
    return 0;
}

int gsb_batch_set_strings(gsb_batch *h, const int *K, int npre, int nsuf, const int8_t *prefix_bits,
                          const int8_t *suffix_bits) {
    if (!h || !K || npre < 1 || nsuf < 1 || !prefix_bits || !suffix_bits) return fail(GSB_E_USAGE, "bad argument");
    BatchEngine &E = h->E;
    const int ninst = (int)E.plans.size();
    std::vector<BInst> inst((size_t)ninst);
    int64_t po = 0, so = 0, oo = 0;
    for (int i = 0; i < ninst; i++) {
        const HPlan &p = E.plans[(size_t)i];
        if (K[i] < 1 || K[i] >= p.ns) return fail(GSB_E_USAGE, "prefix length must be in [1, ns) for instance " + std::to_string(i));
        BInst b;
        b.ns = p.ns;
        b.R = p.R;
        b.K = K[i];
        b.n = p.n;
        b.pre_off = po;
        b.suf_off = so;
        b.out_off = oo;
        po += (int64_t)npre * K[i];
        so += (int64_t)npre * nsuf * (p.ns - K[i]);
        oo += (int64_t)npre * nsuf;
        inst[(size_t)i] = b;
    }
    for (int64_t i = 0; i < po; i++)
        if (prefix_bits[i] != 0 && prefix_bits[i] != 1) return fail(GSB_E_USAGE, "bits must be 0 or 1");
    for (int64_t i = 0; i < so; i++)
        if (suffix_bits[i] != 0 && suffix_bits[i] != 1) return fail(GSB_E_USAGE, "bits must be 0 or 1");
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(E.dev);
    struct Restore {
        int p;
        ~Restore() { cudaSetDevice(p); }
    } restore{prev};
    if (int rc = batch_passes(E, K)) return rc;
    for (int i = 0; i < ninst; i++) {
        const BatchEngine::Lists &l = E.lists[(size_t)i];
        inst[(size_t)i].list_off = l.off;
        inst[(size_t)i].npass[0] = l.npre;
        inst[(size_t)i].npass[1] = l.nsuf;
        inst[(size_t)i].first[0] = l.pre0;
        inst[(size_t)i].first[1] = l.suf0;
    }
    // Buffers grow and stay: a call whose strings fit them keeps the graphs as well, unless it has other counts.  No d_inst (the
    // last of the buffers): none yet, or a call that found no memory for them.
    const bool grow = !E.d_inst || po > E.pre_cap || so > E.suf_cap || oo > E.out_cap;
    if (grow || npre != E.npre || nsuf != E.nsuf) {
        for (auto &kv : E.graphs) cudaGraphExecDestroy(kv.second);
        E.graphs.clear();
    }
    if (grow) {
        const int64_t pre = std::max(po, E.pre_cap), suf = std::max(so, E.suf_cap), res = std::max(oo, E.out_cap);
        E.pre_cap = E.suf_cap = E.out_cap = 0;
        cudaFree(E.d_pre);
        cudaFree(E.d_suf);
        cudaFree(E.d_out);
        cudaFree(E.d_inst);
        E.d_pre = nullptr;
        E.d_suf = nullptr;
        E.d_out = nullptr;
        E.d_inst = nullptr;
        BT_CK(cudaMalloc(&E.d_pre, (size_t)pre));
        BT_CK(cudaMalloc(&E.d_suf, (size_t)suf));
        BT_CK(cudaMalloc(&E.d_out, (size_t)res * sizeof(double)));
        BT_CK(cudaMalloc(&E.d_inst, (size_t)ninst * sizeof(BInst)));
        E.pre_cap = pre;
        E.suf_cap = suf;
        E.out_cap = res;
    }
    E.out_total = oo;
    E.npre = npre;
    E.nsuf = nsuf;
    BT_CK(cudaMemcpy(E.d_inst, inst.data(), (size_t)ninst * sizeof(BInst), cudaMemcpyHostToDevice));
    BT_CK(cudaMemcpy(E.d_pre, prefix_bits, (size_t)po, cudaMemcpyHostToDevice));
    BT_CK(cudaMemcpy(E.d_suf, suffix_bits, (size_t)so, cudaMemcpyHostToDevice));
    E.h_inst = inst;
    return 0;
}

// Run the batch with the current shape (the tuned one after gsb_batch_tune); log2p: per instance [npre][nsuf].
int gsb_batch_run(gsb_batch *h, double *log2p, float *ms) {
    if (!h || !log2p) return fail(GSB_E_USAGE, "null argument");
    BatchEngine &E = h->E;
    if (!E.d_inst) return fail(GSB_E_STATE, "no strings set (gsb_batch_set_strings)");
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(E.dev);
    struct Restore {
        int p;
        ~Restore() { cudaSetDevice(p); }
    } restore{prev};
    cudaGraphExec_t ex;
    if (int rc = batch_graph(E, E.shape, &ex)) return rc;
    cudaEvent_t e0, e1;
    BT_CK(cudaEventCreate(&e0));
    BT_CK(cudaEventCreate(&e1));
    BT_CK(cudaEventRecord(e0, E.stream));
    BT_CK(cudaGraphLaunch(ex, E.stream));
    BT_CK(cudaEventRecord(e1, E.stream));
    BT_CK(cudaMemcpyAsync(log2p, E.d_out, (size_t)E.out_total * sizeof(double), cudaMemcpyDeviceToHost, E.stream));
    BT_CK(cudaStreamSynchronize(E.stream));
    float t = 0;
    cudaEventElapsedTime(&t, e0, e1);
    if (ms) *ms = t;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return 0;
}

// The largest block the batch kernel of this precision can launch with (its registers per thread bound it), or 0.
static int batch_max_block(const BatchEngine &E) {
    cudaFuncAttributes fa{};
    const cudaError_t e = E.prec == 128 ? cudaFuncGetAttributes(&fa, k_batch<double2>) : cudaFuncGetAttributes(&fa, k_batch<float2>);
    return e == cudaSuccess ? fa.maxThreadsPerBlock : 0;
}

int gsb_batch_set_shape(gsb_batch *h, int block, int small_R, int per_sm) {
    if (!h || (block != 64 && block != 128 && block != 256 && block != 512 && block != 1024) || small_R < 0 ||
        small_R > 24 || per_sm < 1 || per_sm > 16 || block * per_sm > 2048)
        return fail(GSB_E_USAGE, "bad shape");
    if (block > batch_max_block(h->E)) return fail(GSB_E_USAGE, "block larger than the batch kernel can launch");
    h->E.shape = BatchShape{block, small_R, per_sm};
    return 0;
}

int gsb_batch_get_shape(const gsb_batch *h, int *block, int *small_R, int *per_sm) {
    if (!h) return fail(GSB_E_STATE, "null handle");
    if (block) *block = h->E.shape.block;
    if (small_R) *small_R = h->E.shape.small_R;
    if (per_sm) *per_sm = h->E.shape.per_sm;
    return 0;
}

// Autotuner: times every candidate shape on the current strings (one warm-up and `reps` timed runs each, CUDA
// events on the batch stream) and keeps the fastest.  Candidates whose arenas exceed `max_bytes` are skipped.
int gsb_batch_tune(gsb_batch *h, int reps, size_t max_bytes, int *block, int *small_R, int *per_sm, float *best_ms) {
    if (!h || reps < 1) return fail(GSB_E_USAGE, "bad argument");
    BatchEngine &E = h->E;
    if (!E.d_inst) return fail(GSB_E_STATE, "no strings set (gsb_batch_set_strings)");
    std::vector<double> out((size_t)std::max<int64_t>(E.out_total, 1));
    float best = 1e30f;
    E.limit = max_bytes;
    BatchShape bs = E.shape;
    const int maxR = E.max_R();
    const int max_block = batch_max_block(E);   // shapes the kernel cannot launch are skipped
    for (int blk : {128, 256, 512})
        for (int sr : {0, 8, 10, 12, 14})
            for (int ps : {1, 2, 4}) {
                if (blk * ps > 2048 || sr > maxR + 1 || blk > max_block) continue;
                BatchShape sh{blk, sr, ps};
                if (shape_layout(E, sh).bytes > max_bytes) continue;
                if (batch_smem(blk) > BATCH_MAX_SMEM) continue;
                E.shape = sh;
                float ms = 0, tot = 0;
                if (int rc = gsb_batch_run(h, out.data(), &ms)) return rc;
                for (int r = 0; r < reps; r++) {
                    if (int rc = gsb_batch_run(h, out.data(), &ms)) return rc;
                    tot += ms;
                }
                if (tot / reps < best) {
                    best = tot / reps;
                    bs = sh;
                }
            }
    E.shape = bs;
    E.tuned = true;
    if (block) *block = bs.block;
    if (small_R) *small_R = bs.small_R;
    if (per_sm) *per_sm = bs.per_sm;
    if (best_ms) *best_ms = best;
    return 0;
}

}  // extern "C"
