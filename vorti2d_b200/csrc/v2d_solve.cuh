// The solve with the multifrontal factors (v2d_mf.cu): work items over the
// fronts, as one dataflow launch or one launch per level and sweep.
//
// After the factorization each front's storage holds, row-major f x f,
//   [0,S) x [0,S)   A11^-1,
//   [S,f) x [0,S)   -G, G = A21 A11^-1,
//   [0,S) x [S,f)   H = A11^-1 A12,
// so every row of the solve is one contiguous dot product with a vector
// gathered once per work item (t = the right-hand side on the pivots):
//   forward,  r <  S:  z_r = t_r (kept for the backward sweep)
//             r >= S:  u_r = w_r + F[r, 0:S] . t[0:S]      contribution to the parent
//   backward, r <  S:  x_r = F[r, 0:f] . v[0:f]            v = (t, -x_struct)
// A front's forward rows need only its children's contributions and its
// backward rows only its own z and its ancestors' x: one dependent step per
// level and sweep.  G and H hold as many entries as A21 and A12, so a solve
// still reads sum S (2f - S) factor entries.
#pragma once

#include "v2d_factor.cuh"
#include "v2d_async.cuh"
#include "v2d_internal.cuh"

namespace v2d {
namespace {

__device__ __forceinline__ bool stopped(const int *a, const int *b)
{
    return (a && *a) || (b && *b);
}

constexpr int kSolveThreads = 256;   // threads that compute a work item
constexpr int kGatherRegs = 4;   // gathered entries per thread whose indices load before the wait
constexpr int kRowGroup = 4;     // rows a warp sums at once
constexpr int kStages = 2;       // matrix chunks in flight ahead of the rows

// A work item and how its rows are staged (plan_chunks): `group` rows per
// chunk of shared memory, `pitch` elements apart, or (segment > 0) one row per
// warp and `segment` columns of it per chunk.
struct SolveItem : SolveItemDev {
    int r0, rows, group, pitch, segment, index;
};

__device__ __forceinline__ SolveItem load_item(const SolveItemDev *items, int i)
{
    SolveItem it;
    static_cast<SolveItemDev &>(it) = items[i];
    it.index = i;
    it.r0 = it.kind == 0 ? max(it.rb, it.S) : it.rb;   // first row with a product
    it.rows = it.kind < 2 ? max(0, it.re - it.r0) : 0;
    it.group = it.pitch = it.segment = 0;
    return it;
}

// How an item's rows are cut into chunks of at most `bytes` of shared memory:
// backward rows are contiguous (pitch f), forward ones (S of f columns) are
// padded to 16 bytes each.  Where fewer rows fit than half the warps, each warp
// takes one row and a chunk holds a segment of those rows (a multiple of 32
// columns: a lane's columns keep their order).
template <class T>
__device__ __forceinline__ void plan_chunks(SolveItem &it, int bytes, int nw)
{
    if (it.rows == 0) return;
    constexpr int E = 16 / (int)sizeof(T);
    it.pitch = it.kind == 1 ? it.f : (it.S + E - 1) / E * E + E;
    int g = (bytes - 32) / (it.pitch * (int)sizeof(T));
    if (g >= nw) g = g / nw * nw;
    it.group = 2 * g < min(nw, it.rows) ? 0 : min(g, it.rows);
    if (it.group > 0) return;
    const int seg = ((bytes - 32) / (nw * (int)sizeof(T)) - E) / 32 * 32;
    if (seg < 64) return;   // hardly any shared memory left: read from global memory
    it.segment = seg;
    it.pitch = seg + E;
}

// Values on their way between items carry their own readiness: before a
// dataflow solve z, upd and x are filled with 0xff bytes (unset: a NaN that no
// arithmetic makes), and an item reads an entry again until it is set.  FP64
// arithmetic may hand on an operand's NaN, so a store replaces this one, which a
// caller's matrix could hold, by the ordinary NaN (no measurable cost).  One word
// is one message, so neither side needs an ordering between words: no counter, no
// release fence after an item's writes (about 0.8 us) and no separate poll before
// its gather (about 0.6 us).
template <class T> struct Unset;
template <> struct Unset<float> {
    __device__ __forceinline__ static bool is(float v) { return __float_as_uint(v) == 0xffffffffu; }
};
template <> struct Unset<double> {
    __device__ __forceinline__ static bool is(double v)
    {
        return __double_as_longlong(v) == -1LL;
    }
};

// Reads of one entry before a CTA gives up (each sleeps 50 ns: about a second
// in all), unless WaitLimits says otherwise.
constexpr int kFlowSpins = 1 << 21;

__device__ __forceinline__ float ld_relaxed(const float *p)
{
    float v;
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ double ld_relaxed(const double *p)
{
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed(float *p, float v)
{
    if (Unset<float>::is(v)) v = __int_as_float(0x7fffffff);
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed(double *p, double v)
{
    if (Unset<double>::is(v)) v = __longlong_as_double(0x7ff8000000000000LL);
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

// The vector of an item, entries e < n (n = count(), or 0 for nothing), each pulled
// through the index maps; the first kGatherRegs per thread have their indices (and
// the scaled right-hand side) loaded by pre(), which needs no other item.
//   forward: t on the pivots, then w on the item's own contribution rows
//   backward: z on the pivots, then -x on the struct variables
// run() stores it to shared memory; it waits for entries not set yet, unless
// the launches before have set them all (Wait = false).  False when a wait ran
// out.
template <class T, int NT> struct SolveGather {
    int a[kGatherRegs], b[kGatherRegs];
    T v[kGatherRegs];

    __device__ __forceinline__ static int count(const SolveItem &it)
    {
        return it.kind == 0 ? it.S + it.rows : it.f;
    }
    __device__ __forceinline__ static void index(const SolveItem &it, const MfDev &D, const T *rhs,
                                                 const double *__restrict__ rs, int e, int &a,
                                                 int &b, T &v)
    {
        if (it.kind == 1) {
            a = D.vars[it.vo + e];
            if (e < it.S) a = ~(it.vo + e);
            return;
        }
        const int p = e < it.S ? e : it.r0 + e - it.S;
        a = it.cu0 >= 0 ? D.inv0[it.vo + p] : -1;
        b = it.cu1 >= 0 ? D.inv1[it.vo + p] : -1;
        v = T(0);
        if (p < it.S) {
            const int r = D.vars[it.vo + p];
            v = (T)(rs[r] * (double)rhs[r]);
        }
    }
    __device__ __forceinline__ void pre(const SolveItem &it, int n, const MfDev &D, const T *rhs,
                                        const double *__restrict__ rs)
    {
#pragma unroll
        for (int k = 0; k < kGatherRegs; ++k) {
            a[k] = b[k] = -1;
            v[k] = T(0);
            const int e = threadIdx.x + k * NT;
            if (e < n) index(it, D, rhs, rs, e, a[k], b[k], v[k]);
        }
    }
    template <bool Wait>
    __device__ __forceinline__ bool run(const SolveItem &it, int n, const MfDev &D, const T *rhs,
                                        const double *__restrict__ rs, const T *zbuf, const T *upd,
                                        const T *x, T *dst, volatile int *err, int limit)
    {
        for (int e0 = threadIdx.x; e0 < n; e0 += kGatherRegs * NT) {
            if (e0 >= kGatherRegs * NT) {
#pragma unroll
                for (int k = 0; k < kGatherRegs; ++k)
                    if (e0 + k * NT < n) index(it, D, rhs, rs, e0 + k * NT, a[k], b[k], v[k]);
            }
            const T *p[2][kGatherRegs];
            T u[2][kGatherRegs];
#pragma unroll
            for (int k = 0; k < kGatherRegs; ++k) {
                p[0][k] = p[1][k] = nullptr;
                if (e0 + k * NT < n) {
                    if (it.kind == 1) {
                        p[0][k] = a[k] < 0 ? zbuf + ~a[k] : x + a[k];
                    } else {
                        if (a[k] >= 0) p[0][k] = upd + it.cu0 + a[k];
                        if (b[k] >= 0) p[1][k] = upd + it.cu1 + b[k];
                    }
                }
            }
            for (int spin = 0;; ++spin) {
                bool unset = false;
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int k = 0; k < kGatherRegs; ++k)
                        if (spin == 0 || (p[h][k] && Unset<T>::is(u[h][k])))
                            u[h][k] = p[h][k] ? ld_relaxed(p[h][k]) : T(0);
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int k = 0; k < kGatherRegs; ++k) unset = unset || Unset<T>::is(u[h][k]);
                if (!Wait || !unset) break;
                if (spin >= limit || ((spin & 63) == 63 && *err)) return false;
                __nanosleep(50);
            }
#pragma unroll
            for (int k = 0; k < kGatherRegs; ++k)
                if (e0 + k * NT < n)
                    dst[e0 + k * NT] = it.kind == 1 ? (a[k] < 0 ? u[0][k] : -u[0][k])
                                                    : v[k] + u[0][k] + u[1][k];
        }
        return true;
    }
};

// Sums of four values over the warp, value u in the lanes [8 u, 8 u + 8): the
// additions of a butterfly (xor 16, 8, 4, 2, 1) with six shuffles for the
// four instead of five for each.
template <class T>
__device__ __forceinline__ T warp_sum4(const T (&a)[4])
{
    constexpr unsigned M = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool h = lane & 16, l = lane & 8;
    const T k0 = (h ? a[2] : a[0]) + __shfl_xor_sync(M, h ? a[0] : a[2], 16);
    const T k1 = (h ? a[3] : a[1]) + __shfl_xor_sync(M, h ? a[1] : a[3], 16);
    T v = (l ? k1 : k0) + __shfl_xor_sync(M, l ? k0 : k1, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(M, v, o);
    return v;
}

// Rows [0, n) of a chunk, one warp per row and kRowGroup rows of a
// warp at once: row(i) gives the address of local row i, in shared or global
// memory.  A lane sums its columns left to right, so a row's sum does not
// depend on where it is read from or on how the rows are cut into chunks.
template <class T, int NT, class Row, class Out>
__device__ __forceinline__ void sum_rows(int n, int len, const T *vec, Row row, Out out)
{
    constexpr int nw = NT / 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int i = wid; i < n; i += kRowGroup * nw) {
        const T *p[kRowGroup];
#pragma unroll
        for (int u = 0; u < kRowGroup; ++u) p[u] = row(min(i + u * nw, n - 1));
        const int mine = i + (lane >> 3) * nw;   // the row whose sum this lane gets
        const int to = mine < n && (lane & 7) == 0 ? out.target(mine) : 0;
        T a[kRowGroup] = {};
        if (i + nw >= n) {          // a single row
#pragma unroll 8
            for (int c = lane; c < len; c += 32) a[0] += p[0][c] * vec[c];
        } else {
#pragma unroll 2
            for (int c = lane; c < len; c += 32) {
                const T x = vec[c];
#pragma unroll
                for (int u = 0; u < kRowGroup; ++u) a[u] += p[u][c] * x;
            }
        }
        const T s = warp_sum4(a);
        if (mine < n && (lane & 7) == 0) out.store(mine, to, s);
    }
}

// Where an item's row sums go.
template <class T> struct SolveOut {
    const SolveItem &it;
    const MfDev &D;
    const T *vec;
    T *upd, *x;
    int base;   // item row of local row 0
    __device__ __forceinline__ int target(int i) const
    {
        const int r = it.r0 + base + i;
        return it.kind == 0 ? it.uo + r - it.S : D.vars[it.vo + r];
    }
    __device__ __forceinline__ void store(int i, int to, T s) const
    {
        if (it.kind == 0)
            st_relaxed(upd + to, vec[it.S + base + i] + s);
        else
            st_relaxed(x + to, s);
    }
};

// One launch per level and sweep: block i runs item i0 + i (its
// dependencies are the previous launches).
template <class T>
__global__ void __launch_bounds__(kSolveThreads, 2) k_solve_level(
    const MfDev D, const T *F, const T *rhs, const double *__restrict__ rs, T *zbuf, T *upd, T *x,
    const SolveItemDev *__restrict__ items, int i0, const int *stop_a, const int *stop_b)
{
    constexpr int NT = kSolveThreads;
    if (stopped(stop_a, stop_b)) return;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T *vec = reinterpret_cast<T *>(smem_raw);
    const SolveItem it = load_item(items, i0 + blockIdx.x);
    SolveGather<T, NT> g;
    const int n = SolveGather<T, NT>::count(it);
    g.pre(it, n, D, rhs, rs);
    g.template run<false>(it, n, D, rhs, rs, zbuf, upd, x, vec, nullptr, 0);
    __syncthreads();
    if (it.kind == 0)
        for (int r = it.rb + (int)threadIdx.x; r < min(it.re, it.S); r += NT)
            st_relaxed(zbuf + it.vo + r, vec[r]);
    const T *A = F + it.fo + (long long)it.r0 * it.f;
    sum_rows<T, NT>(it.rows, it.kind == 0 ? it.S : it.f, vec,
                    [&](int i) { return A + (long long)i * it.f; },
                    SolveOut<T>{it, D, vec, upd, x, 0});
}

// Global nanosecond timer (per-item traces of the dataflow solve).
__device__ __forceinline__ unsigned long long globaltimer_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

struct FlowShared {
    unsigned long long full[kStages], empty[kStages], dfull[2], dempty[2];
    SolveItem item[2];
    volatile int quit;   // a wait ran out: the others end
    int ok, leave;       // leave: the threads that compute end after the next barrier
};

// The whole solve as one launch of work items in the plan's order (forward
// bottom-up, then backward top-down).  A CTA takes items by ticket and runs
// them one after the other; an item's gather waits for the values of the items
// it depends on (Unset).  The plan checks that those come earlier in the order,
// and a CTA runs its items in ticket order, so the first unfinished item is
// always one whose CTA is at it and whose dependencies are met: no co-resident
// grid is needed.  A wait that runs out (or an error seen while waiting) sets
// bar->err (bit 2) and *stop_a (so GMRES stops instead of using an unfinished
// preconditioner) and ends the CTA: the threads that compute leave together, by
// `leave`, which is only set between an item's start and its first barrier, and
// the producer warp once its copies have landed.
//
// What an item reads besides the vectors of other items -- its table entry and
// the factor rows, most of the solve's bytes -- depends on no other item, so a
// producer warp fetches it while the NT other threads are still at the item
// before: it takes the next ticket, writes the item into shared memory and
// copies its rows into kStages chunks of shared memory (mbarriers), refilled as
// they are read.  An item then costs its dependency wait, one gather and the
// row sums from shared memory, instead of a chain of dependent global loads.
//
// Two forms (the autotuner picks one): MINB resident CTAs per SM, 2 or 3, with
// the shared memory split between them.  A launch runs the items [item0,
// item1) with the ticket counter tickets[slot] (from -1): the whole table, or
// (split form) the lower levels' forward items, the upper levels, the lower levels' backward
// items as three launches in stream order -- an item then only waits for items
// of its own launch or of an earlier, finished one.  The lower launches use NT
// = 128 threads and a vector for their own largest front, so more of their many
// small items are in flight per SM.  vbytes: the vector's bytes; cbytes: each
// chunk's.
template <class T, int MINB, int NT = kSolveThreads>
__global__ void __launch_bounds__(NT + 32, MINB) k_solve_flow(
    const MfDev D, const T *F, const T *rhs, const double *__restrict__ rs, T *zbuf, T *upd, T *x,
    const SolveItemDev *__restrict__ items, int item0, int item1, int vbytes, int cbytes,
    int *tickets, int slot, MfBarrier *bar, const int *stop_a, const int *stop_b,
    const WaitLimits limits, unsigned long long *trace)
{
    constexpr int nw = NT / 32;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ FlowShared sh;
    T *vec = reinterpret_cast<T *>(smem_raw);
    unsigned char *chunk0 = smem_raw + vbytes;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&sh.full[s], 32);   // the producer's lanes
            mbar_init(&sh.empty[s], nw);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&sh.dfull[s], 1);
            mbar_init(&sh.dempty[s], 1);
        }
        sh.quit = sh.leave = 0;
        sh.ok = !stopped(stop_a, stop_b);   // read once: all of the CTA's threads agree
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (!sh.ok) return;
    auto give_up = [&]() {
        atomicOr(&bar->err, 2);
        if (stop_a) atomicExch(const_cast<int *>(stop_a), 1);
        sh.quit = 1;
    };
    if (threadIdx.x >= NT) {   // ---------------------------------- producer
        const int lane = threadIdx.x & 31;
        // the next item's ticket and table entry are fetched while this one's
        // rows are copied
        auto take = [&]() {
            SolveItem it;
            do {
                int i = 0;
                if (lane == 0) i = item0 + 1 + atomicAdd(tickets + slot, 1);
                i = __shfl_sync(0xffffffffu, i, 0);
                it.index = -1;
                it.kind = it.S = it.rows = 0;
                if (i >= item1) break;
                it = load_item(items, i);
                if (trace && lane < 3 && (lane == 0 || it.kind > 1)) trace[3 * i + lane] = globaltimer_ns();
            } while (it.kind > 1);   // the items gather for themselves
            return it;
        };
        // b's phase n has ended (a reader that gave up ends it too)
        auto freed = [&](unsigned long long *b, int n) {
            const bool done = mbar_wait(b, n & 1, &sh.quit, limits.pipe);
            return __all_sync(0xffffffffu, done && !sh.quit) != 0;
        };
        int ks = 0;   // chunks issued
        bool ok = true;
        SolveItem next = take();
        for (int k = 0; ok; ++k) {
            SolveItem it = next;
            if (it.index >= 0) {
                next = take();
                plan_chunks<T>(it, cbytes, nw);
            }
            ok = k < 2 || freed(&sh.dempty[k & 1], (k >> 1) - 1);
            if (!ok) break;
            if (lane == 0) {
                sh.item[k & 1] = it;
                mbar_arrive(&sh.dfull[k & 1]);
            }
            if (it.index < 0) break;
            const int len = it.kind == 0 ? it.S : it.f;
            const T *A = F + it.fo + (long long)it.r0 * it.f;
            // the chunk's stage once its readers are done with it
            auto stage = [&]() -> unsigned char * {
                const int s = ks % kStages;
                if (ks >= kStages && !freed(&sh.empty[s], ks / kStages - 1)) return nullptr;
                return chunk0 + (size_t)s * cbytes;
            };
            if (it.group > 0) {
                for (int c = 0; c < it.rows; c += it.group, ++ks) {
                    const int n = min(it.group, it.rows - c);
                    unsigned char *dst = stage();
                    ok = dst != nullptr;
                    if (!ok) break;
                    unsigned long long *full = &sh.full[ks % kStages];
                    const T *src = A + (long long)c * it.f;
                    if (it.kind == 1) {   // contiguous rows: one bulk copy
                        if (lane == 0) {
                            const unsigned mis = (unsigned)((unsigned long long)src & 15);
                            const unsigned bytes = (mis + n * it.f * (unsigned)sizeof(T) + 15) & ~15u;
                            mbar_expect(full, bytes);
                            bulk_copy(dst, (const char *)src - mis, bytes, full);
                        } else {
                            mbar_arrive(full);
                        }
                    } else {
                        // rows of S of f columns (f is even: a row starts on 8
                        // bytes), copied from the 16-byte boundary before each
                        auto row = [&](int r, const char *&p) {
                            p = (const char *)(src + (long long)r * it.f);
                            const unsigned mis = (unsigned)((unsigned long long)p & 15);
                            p -= mis;
                            return (mis + len * (unsigned)sizeof(T) + 15) & ~15u;
                        };
                        const char *p;
                        unsigned bytes = 0;
                        for (int r = lane; r < n; r += 32) bytes += row(r, p);
                        if (bytes > 0) mbar_expect(full, bytes);
                        else mbar_arrive(full);
                        for (int r = lane; r < n; r += 32) {
                            bytes = row(r, p);
                            bulk_copy(dst + (size_t)r * it.pitch * sizeof(T), p, bytes, full);
                        }
                    }
                }
            } else if (it.segment > 0) {   // one row per warp, in column segments
                for (int c = 0; c < it.rows && ok; c += nw) {
                    const int n = min(nw, it.rows - c);
                    for (int b = 0; b < len; b += it.segment, ++ks) {
                        unsigned char *dst = stage();
                        ok = dst != nullptr;
                        if (!ok) break;
                        unsigned long long *full = &sh.full[ks % kStages];
                        const int w = min(it.segment, len - b);
                        if (lane < n) {
                            const char *src = (const char *)(A + (long long)(c + lane) * it.f + b);
                            const unsigned mis = (unsigned)((unsigned long long)src & 15);
                            const unsigned bytes = (mis + w * (unsigned)sizeof(T) + 15) & ~15u;
                            mbar_expect(full, bytes);
                            bulk_copy(dst + (size_t)lane * it.pitch * sizeof(T), src - mis, bytes, full);
                        } else {
                            mbar_arrive(full);
                        }
                    }
                }
            }
        }
        if (!ok && lane == 0) give_up();
        // the CTA may end before its readers have awaited every copy: let them land
        for (int c = max(0, ks - kStages); c < ks; ++c)
            mbar_wait(&sh.full[c % kStages], (c / kStages) & 1, nullptr, kPipeSpins);
        return;
    }
    // -------------------------------------------------------------- the items
    auto sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory"); };
    int ks = 0;
    for (int k = 0;; ++k) {
        // (without an item nothing is gathered: a branch or a vote here costs every
        // item, 181 x 181 FP64 126.5 us a solve against 127.7 with a vote)
        const bool have = mbar_wait(&sh.dfull[k & 1], (k >> 1) & 1, &sh.quit, limits.pipe);
        const SolveItem &it = sh.item[k & 1];   // stays until dempty
        const int ne = have ? SolveGather<T, NT>::count(it) : 0;
        if (!have) sh.leave = 1;
        SolveGather<T, NT> g;
        g.pre(it, ne, D, rhs, rs);
        if (!g.template run<true>(it, ne, D, rhs, rs, zbuf, upd, x, vec, &bar->err, limits.gather))
            sh.leave = 1;
        sync();
        if (sh.leave) goto left;
        if (it.index < 0) return;
        if (trace && threadIdx.x == 0) trace[3 * it.index + 1] = globaltimer_ns();
        if (it.kind == 0)
            for (int r = it.rb + (int)threadIdx.x; r < min(it.re, it.S); r += NT)
                st_relaxed(zbuf + it.vo + r, vec[r]);
        const int len = it.kind == 0 ? it.S : it.f;
        const T *A = F + it.fo + (long long)it.r0 * it.f;
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        // chunk ks in shared memory; the producer may refill its stage after release().
        // Where the wait runs out the rows go on with what is there: nobody uses
        // the result, and a way out of here would cost every chunk a vote.
        auto chunk = [&]() -> const T * {
            const int s = ks % kStages;
            if (!mbar_wait(&sh.full[s], (ks / kStages) & 1, &sh.quit, limits.pipe)) give_up();
            return reinterpret_cast<const T *>(chunk0 + (size_t)s * cbytes);
        };
        auto release = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.empty[ks % kStages]);
        };
        // a row's offset from the 16-byte boundary it was copied from
        auto offset = [&](const T *p) { return (int)(((unsigned long long)p & 15) / sizeof(T)); };
        if (it.group > 0) {
            for (int c = 0; c < it.rows; c += it.group, ++ks) {
                const T *B = chunk();
                const T *first = A + (long long)c * it.f;
                sum_rows<T, NT>(
                    min(it.group, it.rows - c), len, vec,
                    [&](int i) {
                        return B + (size_t)i * it.pitch +
                               offset(it.kind == 1 ? first : first + (long long)i * it.f);
                    },
                    SolveOut<T>{it, D, vec, upd, x, c});
                release();
            }
        } else if (it.segment > 0) {
            for (int c = 0; c < it.rows; c += nw) {
                const int r = c + wid;
                const SolveOut<T> out{it, D, vec, upd, x, 0};
                const int to = r < it.rows ? out.target(r) : 0;
                T a[4] = {};
                for (int b = 0; b < len; b += it.segment, ++ks) {
                    const T *B = chunk();
                    if (r < it.rows) {
                        B += (size_t)wid * it.pitch + offset(A + (long long)r * it.f + b);
                        const int w = min(it.segment, len - b);
#pragma unroll 8
                        for (int e = lane; e < w; e += 32) a[0] += B[e] * vec[b + e];
                    }
                    release();
                }
                const T sum = warp_sum4(a);
                if (lane == 0 && r < it.rows) out.store(r, to, sum);
            }
        } else {
            sum_rows<T, NT>(it.rows, len, vec, [&](int i) { return A + (long long)i * it.f; },
                            SolveOut<T>{it, D, vec, upd, x, 0});
        }
        sync();   // the vector and the item may be replaced
        if (threadIdx.x == 0) {
            if (trace) trace[3 * it.index + 2] = globaltimer_ns();
            mbar_arrive(&sh.dempty[k & 1]);
        }
    }
left:
    give_up();
}

}  // namespace
}  // namespace v2d
