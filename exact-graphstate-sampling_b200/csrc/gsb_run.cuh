// Runs of small steps: consecutive steps whose columns span at most 2^RUN_DIM addresses, walked by one CTA per string.
//
// The two ends of every item, and the whole of a narrow one, are steps of a few thousand entries at most.  As launches of
// their own, or as steps over the arena in global memory, they are bound by latency alone: the arena version of this
// kernel took 2.5 us per step (two block barriers around scalar work in one thread, and dependent loads of the
// descriptor, the state and the table), 54 us for each end of a 'chain' string at width 19 (now 40 for 64 strings side by
// side; both cold).  Calls on 20 steps: one 'prob' 142 us (now 55, with one pass per step), 1024 strings by 'chain' 0.53 ms
// (now 0.114), 100 samples 0.25 ms (now 0.146).  What is left is the latency of FP64 sums, shuffles and instruction fetches,
// step after step.  Here
//   * the live table sits in shared memory in compact coordinates: the addresses that the run's steps touch span a
//     subspace of dimension D <= RUN_DIM, the host picks a basis of it (the widest step's columns first, so that its
//     neighbouring cosets are neighbouring entries) and rewrites every step's columns in that basis;
//   * sums and rotations are FP64 for both arenas; entries are held in the arena's type (complex64 rounds every store);
//   * one barrier per pass: warp sums go to alternating buffers, every thread adds them in the same order and keeps the
//     run's scalars itself, so bits, scales and deaths are uniform without a broadcast;
//   * the next step's descriptor is fetched during a step, forced bits and uniforms before the first one, and
//     logarithms and conditionals are formed after the last one, one step per thread.
// A run may start from the unit table (`begin`), end the item (`finish`), or both: then nothing touches the arena and a
// single launch evaluates any number of strings (`direct`, one CTA each).
#pragma once
#include "gsb_kernels.cuh"

namespace gsb {

constexpr int RUN_DIM = 12;        // 64 KB of shared memory in complex128: three CTAs per SM
constexpr int RUN_THREADS = 512;

// One step in its run's compact coordinates; the entry after a run's last step gives the live table it leaves.
struct RunStep {
    double M[2][2][2];             // [b][x] (re, im)
    uint32_t tk[RUN_DIM], tq[4], g, rhoc;
    int nk, ntq, m;
    int tau0, tau1, par;           // bit t: offset t's x = 0 / x = 1 output, x = 1 sign
};
static_assert(sizeof(RunStep) % 8 == 0 && sizeof(RunStep) <= 32 * 8, "one 8-byte word per lane of a warp");

struct RunArgs {
    const RunStep *rs;             // entries of steps k0 .. k1 (k1: the table left)
    const StepArgs *sa;            // the engine's steps (arena columns of steps k0 and k1)
    int k0, k1, dim;
    int norm;                      // branch norms of the steps whose bit is drawn ('chain' passes: none)
    int begin, finish, direct;     // direct: begin and finish, item = blockIdx.y, no state
    double *logp, *aux;            // finish: per item
};

// Sums of v over the block, to every thread, in a fixed order; also a barrier.
template <int ND>
__device__ __forceinline__ void run_sum(double (&v)[ND], double (*red)[2][RUN_THREADS / 32], int &buf) {
#pragma unroll
    for (int i = 0; i < ND; i++) v[i] = warp_sum(v[i]);
    const int nw = (int)(blockDim.x >> 5);
    if (nw == 1) {
        __syncwarp();
        return;
    }
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int i = 0; i < ND; i++) red[buf][i][threadIdx.x >> 5] = v[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ND; i++) {
        double t = red[buf][i][0];
        for (int w = 1; w < nw; w++) t += red[buf][i][w];
        v[i] = t;
    }
    buf ^= 1;
}

__device__ __forceinline__ double flip_sign(double x, int neg) {
    return __hiloint2double(__double2hiint(x) ^ (neg << 31), __double2loint(x));
}

// One pass over a step's cosets: the written branch `bv` scaled by sc (WRITE: sum[0] = its norm), or both branch norms.
// Thread t takes cosets t, t + T, ...: UB of them at a time, all their loads before any store (cosets share no slot).
// The loop's bounds and the cosets' high bits are uniform; only the low bits' base and sign are the thread's own.
template <typename E, int NTQ, bool WRITE>
__device__ __forceinline__ void run_pass_n(const RunStep &s, E *tab, int bv, double sc, double (&sum)[2]) {
    constexpr int UB = NTQ == 4 ? 2 : 4;
    const uint32_t N = 1u << s.nk, T = blockDim.x, tid = threadIdx.x;
    const int lt = __ffs((int)T) - 1;
    const uint32_t per = N > T ? N >> lt : 1;
    if (tid >= N) return;
    uint32_t lo = 0;
#pragma unroll
    for (int j = 0; j < 9; j++)   // T <= 2^9
        if ((tid >> j) & 1) lo ^= s.tk[j];
    const int plo = __popc(tid & s.rhoc);
    const double m0r = s.M[bv][0][0], m0i = s.M[bv][0][1], m1r = s.M[bv][1][0], m1i = s.M[bv][1][1];
#pragma unroll 1
    for (uint32_t h0 = 0; h0 < per; h0 += UB) {
        uint32_t b0 = lo;
        for (uint32_t h = h0 >> 1, j = (uint32_t)lt + 1; h; h >>= 1, j++)
            if (h & 1) b0 ^= s.tk[j];
        E v[UB][NTQ];
        uint32_t base[UB];
#pragma unroll
        for (int u = 0; u < UB; u++) {
            if (h0 + (uint32_t)u >= per) break;
            base[u] = b0 ^ (u & 1 ? s.tk[lt] : 0u) ^ (u & 2 ? s.tk[lt + 1] : 0u);
#pragma unroll
            for (int t = 0; t < NTQ; t++) v[u][t] = tab[base[u] ^ s.tq[t]];
        }
#pragma unroll
        for (int u = 0; u < UB; u++) {
            if (h0 + (uint32_t)u >= per) break;
            const int pc = plo ^ __popc(((h0 + (uint32_t)u) << lt) & s.rhoc);
            double s00r = 0, s00i = 0, s01r = 0, s01i = 0, s10r = 0, s10i = 0, s11r = 0, s11i = 0;
#pragma unroll
            for (int t = 0; t < NTQ; t++) {
                const double xr = (double)v[u][t].x, xi = (double)v[u][t].y;
                if ((s.tau0 >> t) & 1) { s01r += xr; s01i += xi; }
                else { s00r += xr; s00i += xi; }
                const int neg = (pc ^ (s.par >> t)) & 1;
                const double yr = flip_sign(xr, neg), yi = flip_sign(xi, neg);
                if ((s.tau1 >> t) & 1) { s11r += yr; s11i += yi; }
                else { s10r += yr; s10i += yi; }
            }
            if (WRITE) {
                double r = m0r * s00r - m0i * s00i + m1r * s10r - m1i * s10i;
                double i = m0r * s00i + m0i * s00r + m1r * s10i + m1i * s10r;
                r *= sc;
                i *= sc;
                store_entry(tab + base[u], r, i);
                sum[0] += r * r + i * i;
                if (s.m == 2) {
                    r = m0r * s01r - m0i * s01i + m1r * s11r - m1i * s11i;
                    i = m0r * s01i + m0i * s01r + m1r * s11i + m1i * s11r;
                    r *= sc;
                    i *= sc;
                    store_entry(tab + (base[u] ^ s.g), r, i);
                    sum[0] += r * r + i * i;
                }
            } else {
#pragma unroll
                for (int b = 0; b < 2; b++) {
                    const double p0r = s.M[b][0][0], p0i = s.M[b][0][1], p1r = s.M[b][1][0], p1i = s.M[b][1][1];
                    double r = p0r * s00r - p0i * s00i + p1r * s10r - p1i * s10i;
                    double i = p0r * s00i + p0i * s00r + p1r * s10i + p1i * s10r;
                    sum[b] += r * r + i * i;
                    if (s.m == 2) {
                        r = p0r * s01r - p0i * s01i + p1r * s11r - p1i * s11i;
                        i = p0r * s01i + p0i * s01r + p1r * s11i + p1i * s11r;
                        sum[b] += r * r + i * i;
                    }
                }
            }
        }
    }
}

template <bool WRITE, typename E>
__device__ __forceinline__ void run_pass(const RunStep &s, E *tab, int bv, double sc, double (&sum)[2]) {
    if (s.ntq == 4) run_pass_n<E, 4, WRITE>(s, tab, bv, sc, sum);
    else if (s.ntq == 2) run_pass_n<E, 2, WRITE>(s, tab, bv, sc, sum);
    else run_pass_n<E, 1, WRITE>(s, tab, bv, sc, sum);
}

// A step whose bit is drawn from its branch norms, with at most two cosets per thread: the cosets' sums stay in registers
// between the norms and the write, which then reads nothing and forms no sums again (100 samples of 20 steps: 155 -> 148 us a
// call; a 'prob' of two passes per step 74 -> 67).
struct CosetSums {
    double x[2][2], z[2][2];   // [tau][re, im]: x = 0 and signed x = 1 sums
    uint32_t base;
};
template <typename E, int NTQ>
__device__ __forceinline__ void coset_sums(const RunStep &s, const E *tab, uint32_t per, CosetSums (&c)[2]) {
    const uint32_t T = blockDim.x, tid = threadIdx.x;
    const int lt = __ffs((int)T) - 1;
    uint32_t lo = 0;
#pragma unroll
    for (int j = 0; j < 9; j++)
        if ((tid >> j) & 1) lo ^= s.tk[j];
    const int plo = __popc(tid & s.rhoc);
    E v[2][NTQ];
#pragma unroll
    for (int u = 0; u < 2; u++) {
        if ((uint32_t)u >= per) break;
        c[u].base = u ? lo ^ s.tk[lt] : lo;
#pragma unroll
        for (int t = 0; t < NTQ; t++) v[u][t] = tab[c[u].base ^ s.tq[t]];
    }
#pragma unroll
    for (int u = 0; u < 2; u++) {
        if ((uint32_t)u >= per) break;
        const int pc = plo ^ (u ? (int)(s.rhoc >> lt) : 0);
#pragma unroll
        for (int tau = 0; tau < 2; tau++) c[u].x[tau][0] = c[u].x[tau][1] = c[u].z[tau][0] = c[u].z[tau][1] = 0;
#pragma unroll
        for (int t = 0; t < NTQ; t++) {
            const double xr = (double)v[u][t].x, xi = (double)v[u][t].y;
            if ((s.tau0 >> t) & 1) { c[u].x[1][0] += xr; c[u].x[1][1] += xi; }
            else { c[u].x[0][0] += xr; c[u].x[0][1] += xi; }
            const int neg = (pc ^ (s.par >> t)) & 1;
            const double yr = flip_sign(xr, neg), yi = flip_sign(xi, neg);
            if ((s.tau1 >> t) & 1) { c[u].z[1][0] += yr; c[u].z[1][1] += yi; }
            else { c[u].z[0][0] += yr; c[u].z[0][1] += yi; }
        }
    }
}
template <typename E>
__device__ __forceinline__ void coset_sums_any(const RunStep &s, const E *tab, uint32_t per, CosetSums (&c)[2]) {
    if (s.ntq == 4) coset_sums<E, 4>(s, tab, per, c);
    else if (s.ntq == 2) coset_sums<E, 2>(s, tab, per, c);
    else coset_sums<E, 1>(s, tab, per, c);
}
// Output tau of a coset under row b, times sc.
__device__ __forceinline__ void coset_out(const RunStep &s, const CosetSums &c, int b, int tau, double sc, double &r, double &i) {
    const double m0r = s.M[b][0][0], m0i = s.M[b][0][1], m1r = s.M[b][1][0], m1i = s.M[b][1][1];
    const double xr = c.x[tau][0], xi = c.x[tau][1], zr = c.z[tau][0], zi = c.z[tau][1];
    r = (m0r * xr - m0i * xi + m1r * zr - m1i * zi) * sc;
    i = (m0r * xi + m0i * xr + m1r * zi + m1i * zr) * sc;
}
__device__ __forceinline__ void coset_norms(const RunStep &s, uint32_t per, const CosetSums (&c)[2], double (&sum)[2]) {
#pragma unroll
    for (int u = 0; u < 2; u++) {
        if ((uint32_t)u >= per) break;
#pragma unroll
        for (int b = 0; b < 2; b++)
#pragma unroll
            for (int tau = 0; tau < 2; tau++) {
                if (tau >= s.m) break;
                double r, i;
                coset_out(s, c[u], b, tau, 1.0, r, i);
                sum[b] += r * r + i * i;
            }
    }
}
template <typename E>
__device__ __forceinline__ void coset_write(const RunStep &s, E *tab, uint32_t per, const CosetSums (&c)[2], int bv, double sc,
                                            double (&sum)[2]) {
#pragma unroll
    for (int u = 0; u < 2; u++) {
        if ((uint32_t)u >= per) break;
#pragma unroll
        for (int tau = 0; tau < 2; tau++) {
            if (tau >= s.m) break;
            double r, i;
            coset_out(s, c[u], bv, tau, sc, r, i);
            store_entry(tab + (tau ? c[u].base ^ s.g : c[u].base), r, i);
            sum[0] += r * r + i * i;
        }
    }
}

// Shared memory of a run: the table, two step descriptors, the warp sums, and per step two saved scalars, the uniform
// and the bit.
inline size_t run_smem(int dim, int nsteps, size_t esize) {
    return (esize << dim) + 2 * sizeof(RunStep) + 4 * (RUN_THREADS / 32) * sizeof(double) + (size_t)nsteps * 25 + 8;
}

template <typename E>
__global__ void __launch_bounds__(RUN_THREADS) k_run(const RunArgs ra, E *__restrict__ mem, const Ctx c0) {
    const Ctx cx = slot_ctx(c0);
    mem += (size_t)blockIdx.y * cx.arena;
    DevState *st = cx.st;
    const int item = ra.direct ? (int)blockIdx.y : st->item;
    const int tid = (int)threadIdx.x, T = (int)blockDim.x, n = ra.k1 - ra.k0;
    if (!ra.direct) {
        if (ra.begin ? item >= st->nitems : *(volatile int *)&st->dead) {
            // a slot without an item, or an item that died before: nothing to run, but its end is still to be recorded
            __syncthreads();
            if (tid) return;
            if (ra.begin) st->dead = 1;
            if (!ra.finish) return;
            st->item = item + (int)gridDim.y;
            if (item >= st->nitems) return;
            ra.logp[item] = -INFINITY;
            if (ra.aux) ra.aux[item] = cx.driver == DRV_HYBRID ? st->logscale : st->aux;
            return;
        }
    }
    extern __shared__ __align__(16) unsigned char smem[];
    E *tab = reinterpret_cast<E *>(smem);
    RunStep *steps = reinterpret_cast<RunStep *>(smem + (sizeof(E) << ra.dim));
    double(*red)[2][RUN_THREADS / 32] = reinterpret_cast<double(*)[2][RUN_THREADS / 32]>(steps + 2);
    double *va = reinterpret_cast<double *>(red + 2), *vb = va + n, *un = vb + n;
    int8_t *bit = reinterpret_cast<int8_t *>(un + n);
    const size_t row = (size_t)item * (size_t)cx.ns;

    double prev = 1, lsc = 0, logscale = 0, logp = 0, sc = 1, n0 = 0, n1 = 0;
    int ek = 0, bv = 0;
    if (!ra.begin) {
        prev = st->prev; lsc = st->lsc; logscale = st->logscale; logp = st->logp;
        sc = st->sc; n0 = st->n0; n1 = st->n1; ek = st->ek; bv = st->bv;
    }
    for (int i = tid; i < n; i += T) {
        bit[i] = cx.forced ? cx.forced[row + ra.k0 + i] : (int8_t)-1;
        un[i] = cx.unif ? cx.unif[row + ra.k0 + i] : 0.0;
    }
    constexpr int WORDS = (int)sizeof(RunStep) / 8;
    if (tid < WORDS) reinterpret_cast<uint64_t *>(steps)[tid] = reinterpret_cast<const uint64_t *>(ra.rs)[tid];
    if (ra.begin && tid == 0) store_entry(tab, 1.0, 0.0);
    __syncthreads();
    if (!ra.begin) {
        const StepArgs &a = ra.sa[ra.k0];
        for (uint32_t c = (uint32_t)tid; c < 1u << steps[0].nk; c += (uint32_t)T) {
            uint64_t g = 0;
            uint32_t l = 0;
            for (uint32_t h = c, j = 0; h; h >>= 1, j++)
                if (h & 1) { g ^= a.tk[j]; l ^= steps[0].tk[j]; }
            for (int t = 0; t < steps[0].ntq; t++) tab[l ^ steps[0].tq[t]] = mem[g ^ a.tq[t]];
        }
        __syncthreads();
    }

    // An item dies where a branch has probability 0, not where a norm is not a number: a NaN goes on to the results, as the
    // epilogues of the wide steps let it.
    int buf = 0, died = -1;
    for (int k = 0; k < n; k++) {
        const RunStep &s = steps[k & 1];
        uint64_t next = 0;
        if (tid < WORDS) next = reinterpret_cast<const uint64_t *>(ra.rs + k + 1)[tid];
        double sum[2] = {0, 0};
        const int f = bit[k];
        const uint32_t N = 1u << s.nk;
        const bool pair = N <= 2u * (uint32_t)T;   // at most two cosets per thread
        const uint32_t per = (uint32_t)tid >= N ? 0 : N > (uint32_t)T ? 2 : 1;
        CosetSums c[2];
        if (cx.driver == DRV_CHAIN1) {
            run_pass<true>(s, tab, f, sc, sum);
            if (tid < WORDS) reinterpret_cast<uint64_t *>(steps + ((k + 1) & 1))[tid] = next;
            double nb[1] = {sum[0]};
            run_sum<1>(nb, red, buf);
            if (tid == 0) { va[k] = ldexp(nb[0], 2 * ek); vb[k] = 2 * prev; }
            lsc += ek;
            prev = nb[0];
            if (prev <= 0) { died = k; break; }
            int ex;
            frexp(prev, &ex);
            ek = (ex - 1) >> 1;
            sc = ldexp(1.0, -ek);
        } else if (cx.driver == DRV_CHAIN) {
            if (pair) {
                coset_sums_any(s, tab, per, c);
                coset_norms(s, per, c, sum);
            } else {
                run_pass<false>(s, tab, 0, 1.0, sum);
            }
            run_sum<2>(sum, red, buf);
            n0 = sum[0];
            n1 = sum[1];
            const double p1 = n1 / (n0 + n1);
            bv = f >= 0 ? f : un[k] < p1;
            const double pb = bv ? p1 : 1 - p1;
            if (tid == 0) { va[k] = pb; bit[k] = (int8_t)bv; }
            if (pb <= 0) { died = k; break; }
            sc = rsqrt(bv ? n1 : n0);
            sum[0] = 0;
            if (pair) coset_write(s, tab, per, c, bv, sc, sum);
            else run_pass<true>(s, tab, bv, sc, sum);
            if (tid < WORDS) reinterpret_cast<uint64_t *>(steps + ((k + 1) & 1))[tid] = next;
            if (k + 1 < n || ra.finish) {
                __syncthreads();
            } else {   // the stored table's norm, for the pass that follows the run
                double nb[1] = {sum[0]};
                run_sum<1>(nb, red, buf);
                prev = nb[0];
            }
        } else {   // DRV_HYBRID
            if (f >= 0) bv = f;
            const bool drawn = f < 0 && ra.norm;
            if (drawn) {
                if (pair) {
                    coset_sums_any(s, tab, per, c);
                    coset_norms(s, per, c, sum);
                } else {
                    run_pass<false>(s, tab, 0, 1.0, sum);
                }
                run_sum<2>(sum, red, buf);
                n0 = sum[0];
                n1 = sum[1];
                bv = un[k] < n1 / (n0 + n1);
                sum[0] = 0;
            }
            if (drawn && pair) coset_write(s, tab, per, c, bv, rsqrt(prev), sum);
            else run_pass<true>(s, tab, bv, rsqrt(prev), sum);
            if (tid < WORDS) reinterpret_cast<uint64_t *>(steps + ((k + 1) & 1))[tid] = next;
            double nb[1] = {sum[0]};
            run_sum<1>(nb, red, buf);
            if (tid == 0) { va[k] = nb[0] / 2; vb[k] = prev; bit[k] = (int8_t)bv; }
            prev = nb[0];
            if (prev <= 0) { died = k; break; }
        }
    }
    __syncthreads();

    // per step, one thread each: conditionals, bits, and the terms of the running logarithms (added below in step order)
    const int done = died < 0 ? n : died + 1;
    for (int i = tid; i < n; i += T) {
        const size_t o = row + (size_t)(ra.k0 + i);
        if (cx.driver == DRV_CHAIN1) {
            cx.cond_out[o] = i < done && i != died ? va[i] / vb[i] : 0.0;
        } else if (cx.driver == DRV_CHAIN) {
            cx.bits_out[o] = i < done && i != died ? bit[i] : cx.forced ? cx.forced[o] : (int8_t)0;
            if (i < done) va[i] = log2(va[i]);
        } else {
            cx.cond_out[o] = i < done && i != died ? va[i] : 0.0;
            if (i >= done || i == died) {
                const int f = cx.forced[o];
                cx.bits_out[o] = (int8_t)(f < 0 ? 0 : f);
            } else {
                cx.bits_out[o] = bit[i];
            }
            if (i < done) { va[i] = log2(va[i]); vb[i] = 0.5 * log2(vb[i]); }
        }
    }
    if (died >= 0)   // the steps after the run
        for (int k = ra.k1 + tid; k < (cx.driver == DRV_HYBRID ? cx.k1 : cx.ns); k += T) {
            const size_t o = row + (size_t)k;
            if (cx.driver != DRV_CHAIN) cx.cond_out[o] = 0;
            if (cx.driver == DRV_CHAIN) cx.bits_out[o] = cx.forced ? cx.forced[o] : (int8_t)0;
            else if (cx.driver == DRV_HYBRID) cx.bits_out[o] = (int8_t)(cx.forced[o] < 0 ? 0 : cx.forced[o]);
        }
    __syncthreads();
    if (!ra.direct && died < 0) {   // the table left, to the arena
        const RunStep &s = steps[n & 1];
        const StepArgs &a = ra.sa[ra.k1];
        for (uint32_t c = (uint32_t)tid; c < 1u << s.nk; c += (uint32_t)T) {
            uint64_t g = 0;
            uint32_t l = 0;
            for (uint32_t h = c, j = 0; h; h >>= 1, j++)
                if (h & 1) { g ^= a.tk[j]; l ^= s.tk[j]; }
            for (int t = 0; t < s.ntq; t++) mem[g ^ a.tq[t]] = tab[l ^ s.tq[t]];
        }
    }
    if (tid) return;
    if (cx.driver != DRV_CHAIN1)
        for (int i = 0; i < done; i++) {
            if (i != died) logp += va[i];
            if (cx.driver == DRV_HYBRID) logscale += vb[i];
        }
    if (died >= 0) logp = -INFINITY;
    if (ra.finish) {
        ra.logp[item] = cx.driver != DRV_CHAIN1 ? logp : died >= 0 ? -INFINITY : log2(prev) + 2.0 * lsc - cx.ns;
        if (ra.aux) ra.aux[item] = cx.driver == DRV_HYBRID ? logscale : ra.begin ? 0.0 : st->aux;
    }
    if (ra.direct) return;
    st->prev = prev; st->lsc = lsc; st->logscale = logscale; st->logp = logp;
    st->sc = sc; st->n0 = n0; st->n1 = n1; st->ek = ek; st->bv = bv;
    st->dead = died >= 0;
    if (ra.begin) { st->counter = 0; st->trx = 0; st->aux = 0; }
    if (ra.finish) st->item = item + (int)gridDim.y;
}

}  // namespace gsb
