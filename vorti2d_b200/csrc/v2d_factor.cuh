// Numeric phase of the multifrontal factorization (v2d_mf.cu): batched dense
// kernels over the fronts of one tree level.
//
// Each front (S pivots of f variables, row-major f x f) is eliminated by
// blocked Gauss-Jordan steps of kPiv pivots.  A step on the pivots K = [k, e)
// of a front A does, in place,
//   X = A_KK^-1                          k_assemble, k_update (X replaces A_KK)
//   R = X A_KJ for all columns J != K    k_row_block     (R replaces A_KJ)
//   A_IJ -= A_IK R, A_IK = -A_IK X       k_update, every row I outside K
// and leaves, after the last step, exactly what a solve multiplies with:
//   [0,S) x [0,S)   A11^-1
//   [0,S) x [S,f)   H = A11^-1 A12
//   [S,f) x [0,S)   -G, G = A21 A11^-1
//   [S,f) x [S,f)   the Schur complement, the parent's contribution block.
// The whole front is updated in each step by one uniform rank-kPiv product,
// so a level needs three launches per step and no separate triangular
// solves, inverses or products of the factors; the price is 2 S f^2 flops
// instead of the 4/3 S^3 + 4 S^2 m + 2 S m^2 (m = f - S) of LU, inverses, G
// and H: 1.5 times as many on a front without contribution rows, 1.09 times
// at f = 2 S, almost none more on wide fronts.
//
// Pivoting is partial among 32 rows: a pivot block is inverted as two 32 x 32
// diagonal blocks one after the other, each by implicit row exchanges inside X
// (no permutation leaves the block), so a block whose leading half is singular
// fails although the whole is regular.  The row scaling applied at assembly keeps
// the blocks well scaled, and the FP64 Krylov iteration around the factors absorbs
// the restriction.  X is computed in FP64 in both precisions: on a 181 x 181
// Jacobian one FP32 solve then reduces the residual to 5e-6, against 2e-2 with an
// FP32 X and 9e-2 with FP32 LU factors and their explicit inverses (one and two
// GMRES iterations more).
#pragma once

#include <algorithm>

#include "v2d_async.cuh"
#include "v2d_internal.cuh"

namespace v2d {
namespace {

constexpr int kPiv = 64;      // pivots per elimination step
constexpr int kTile = 64;     // output tile of the step's products
constexpr int kSlice = 32;    // inner columns per operand slice
// rs[r] = 1 / max_c |a_rc| (1 for an empty row).
__global__ void k_rowscale(int n, const int *__restrict__ rowptr, const double *__restrict__ val,
                           double *rs)
{
    V2D_GRID_STRIDE(r, n)
    {
        double m = 0.0;
        for (int p = rowptr[r]; p < rowptr[r + 1]; ++p) m = fmax(m, fabs(val[p]));
        rs[r] = m > 0.0 ? 1.0 / m : 1.0;
    }
}

// Every front's own matrix entries, row-scaled, into the zeroed fronts: one
// entry per position, so a plain store (a read of the zero would cost a second
// trip to memory), four entries of a thread in flight (513 x 513 FP64: 0.56 ms
// with += and one entry at a time).
constexpr int kScatterEntries = 4;

template <class T>
__global__ void __launch_bounds__(256) k_scatter(long long n, const int *__restrict__ csr,
                                                 const int *__restrict__ row,
                                                 const long long *__restrict__ pos,
                                                 const double *__restrict__ val,
                                                 const double *__restrict__ rs, T *F)
{
    const long long e0 = (long long)blockIdx.x * (256 * kScatterEntries) + threadIdx.x;
    int c[kScatterEntries], r[kScatterEntries];
    long long p[kScatterEntries];
#pragma unroll
    for (int k = 0; k < kScatterEntries; ++k) {
        const long long e = e0 + 256 * k;
        c[k] = e < n ? csr[e] : -1;
        r[k] = e < n ? row[e] : 0;
        p[k] = e < n ? pos[e] : 0;
    }
    double v[kScatterEntries], s[kScatterEntries];
#pragma unroll
    for (int k = 0; k < kScatterEntries; ++k) {
        v[k] = c[k] >= 0 ? val[c[k]] : 0.0;
        s[k] = c[k] >= 0 ? rs[r[k]] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kScatterEntries; ++k)
        if (c[k] >= 0) F[p[k]] = (T)(v[k] * s[k]);
}

// inv[slot][voff[P] + cbmap[e]] = e for each front's contribution variables:
// the position of a parent's local variable in its child's contribution
// block (the arrays are preset to -1).
__global__ void k_invert_cbmap(int nf, const int *__restrict__ S, const int *__restrict__ f,
                               const int *__restrict__ voff, const int *__restrict__ uoff,
                               const int *__restrict__ parent, const int *__restrict__ child0,
                               const int *__restrict__ cbmap, int *inv0, int *inv1)
{
    for (int q = blockIdx.x; q < nf; q += gridDim.x) {
        const int pa = parent[q];
        if (pa < 0) continue;
        int *inv = child0[pa] == q ? inv0 : inv1;
        for (int e = threadIdx.x; e < f[q] - S[q]; e += blockDim.x)
            inv[voff[pa] + cbmap[uoff[q] + e]] = e;
    }
}

// A front of the level being assembled and its children's contribution
// blocks (null where it has no such child), with the inverse maps of its
// variables.
template <class T> struct Assembly {
    T *A;
    const T *src[2];
    const int *map[2];
    int f, w, fc[2];   // w: pivots of the first elimination step
};

struct AssemblyMaps {
    const int *S, *f, *voff, *child0, *child1, *inv0, *inv1;
    const long long *foff;
};

template <class T>
__device__ __forceinline__ Assembly<T> assembly_of(const AssemblyMaps &m, int q, T *F)
{
    Assembly<T> a;
    const int c[2] = {m.child0[q], m.child1[q]}, vo = m.voff[q];
    a.A = F + m.foff[q];
    a.f = m.f[q];
    a.w = min(kPiv, m.S[q]);
    a.map[0] = m.inv0 + vo;
    a.map[1] = m.inv1 + vo;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        a.src[u] = nullptr;
        a.fc[u] = 0;
        if (c[u] >= 0) {
            a.fc[u] = m.f[c[u]];
            const int sc = m.S[c[u]];
            a.src[u] = F + m.foff[c[u]] + (long long)sc * a.fc[u] + sc;
        }
    }
    return a;
}

// One warp's share of the extend-add: kExtRows rows x kExtCols columns of a
// front, each entry pulled from the children through the inverse maps (a
// fixed order of addition, no atomics, one pass for both children).  A lane
// keeps its columns' positions for all rows, and a row's loads are all in
// flight together; the first step's pivot block is left out (k_assemble adds
// it where it inverts it).
constexpr int kExtRows = 4, kExtCols = 256, kExtWarps = 8;

template <class T>
__device__ __forceinline__ void extend_rows(const Assembly<T> &a, int r0, int c0)
{
    constexpr int U = kExtCols / 32;
    const int lane = threadIdx.x & 31;
    int j[2][U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int c = c0 + lane + 32 * u;
#pragma unroll
        for (int h = 0; h < 2; ++h) j[h][u] = a.src[h] && c < a.f ? a.map[h][c] : -1;
    }
#pragma unroll 2
    for (int r = r0; r < min(r0 + kExtRows, a.f); ++r) {
        int i[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) i[h] = a.src[h] ? a.map[h][r] : -1;
        if (i[0] < 0 && i[1] < 0) continue;
        const T *s0 = a.src[0] + (long long)i[0] * a.fc[0], *s1 = a.src[1] + (long long)i[1] * a.fc[1];
        T *d = a.A + (long long)r * a.f + c0 + lane;
        T v[U], x0[U], x1[U];
        bool on[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool p0 = i[0] >= 0 && j[0][u] >= 0, p1 = i[1] >= 0 && j[1][u] >= 0;
            on[u] = (p0 || p1) && !(r < a.w && c0 + lane + 32 * u < a.w);
            v[u] = on[u] ? d[32 * u] : T(0);
            x0[u] = p0 ? s0[j[0][u]] : T(0);
            x1[u] = p1 ? s1[j[1][u]] : T(0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (on[u]) d[32 * u] = v[u] + x0[u] + x1[u];
    }
}

// ------------------------------------------------------- 64 x 64 products
// Asynchronous global -> shared copy of B bytes (B-aligned on both sides);
// ok == false writes zeros and reads nothing.
template <int B>
__device__ __forceinline__ void cp_async(void *dst, const void *src, bool ok)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (B == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src),
                     "r"(ok ? 16 : 0));
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(src), "n"(B),
                     "r"(ok ? B : 0));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void dmma_8x8x4(double &c0, double &c1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

// X = A_KK^-1 of one step's pivot block, in FP64, by four warps: for a level's
// first step by the CTA that adds the children's entries to that block
// (k_assemble), for every later step by the CTA that has just updated it in
// the step before (k_update): no launch and no round trip through memory in
// the chain of steps, and hidden behind the other CTAs on levels with many.
// The block sits in shared memory as 2 x 2 blocks of 32 and is inverted by
// block Gauss-Jordan: the 32 x 32 diagonal blocks one after the other in
// registers (invert32), the products between the blocks on the FP64 tensor
// cores.  The chain of pivot columns bounds it, not its 2 kPiv^3 flops: the code
// is kept short and rolled, since straight-line code that runs once waits for its
// own instructions.
constexpr int kInvThreads = 128;
constexpr int kHalf = kPiv / 2;
constexpr int kLdX = kPiv + 2;   // two wavefronts per fragment read, rows 16-byte aligned
constexpr int kPanel = 4;        // columns per panel of invert32, one per warp

// Shared memory of one pivot block's inversion.
struct PivotSmem {
    double M[kPiv * kLdX];
    double col[2][kPanel][kHalf];
    int piv[kHalf];
};

// Barrier of the inversion's four warps (the first of the CTA).
__device__ __forceinline__ void pivot_sync()
{
    asm volatile("bar.sync 1, %0;" ::"n"(kInvThreads) : "memory");
}

// The reciprocal of a pivot: Newton's iteration for 1 / x, y += y (1 - x y), twice
// from the hardware's approximation, which flushes subnormals: within 2 units in
// the last place for |x| in [2^-1021, 2^1021).  The chain of pivot columns waits
// for it: with the division in its place a factorization of 65 x 65 takes 526 us
// instead of 487, of 181 x 181 1.66 ms instead of 1.57.
__device__ __forceinline__ double reciprocal(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    y = fma(y, fma(-x, y, 1.0), y);
    return fma(y, fma(-x, y, 1.0), y);
}
// The bits of |x|'s high word, without the sign's; of numbers in that range.
constexpr unsigned kFastLo = 2u << 21, kFastHi = 2044u << 21;
__device__ __forceinline__ unsigned pivot_bits(double x) { return (unsigned)__double2hiint(x) << 1; }
__device__ __forceinline__ bool fast_pivot(unsigned bits)
{
    return bits - kFastLo < kFastHi - kFastLo;
}
// Of any number but 0: those outside the range are scaled into it.
__device__ __forceinline__ double reciprocal_scaled(double x)
{
    const unsigned bits = pivot_bits(x);
    const double s = fast_pivot(bits) ? 1.0 : bits < kFastLo ? 0x1p100 : 0x1p-100;
    return reciprocal(x * s) * s;
}

// y[i] = 1 / x[i] as invert32 takes it of a pivot.
__global__ void k_reciprocal(int n, const double *x, double *y)
{
    V2D_GRID_STRIDE(i, n)
    {
        y[i] = fast_pivot(pivot_bits(x[i])) ? reciprocal(x[i]) : reciprocal_scaled(x[i]);
    }
}

// In-place inverse of the n x n block at M (n <= 32, rows ld apart; padded by
// the identity in registers) by four warps: lane = row,
// column 4 i + w in register i of warp w.  Gauss-Jordan in panels of four
// columns, one of each warp: the warps exchange the panel through shared
// memory (one barrier) and each eliminates its four columns on its own copy
// and on its own other seven columns, the pivot rows by shuffles; then the
// registers rotate by one, so that the next panel is again in a[0] and the
// loop stays rolled.  Partial pivoting with implicit row exchanges: the pivot
// is the free row with the largest |a| to 15 bits (one warp reduction finds
// value and lane; each lane takes the reciprocal of its own candidate
// meanwhile).  A pivot row stays unscaled until the end (the updates are
// linear in it), so a column is one multiply-add per entry on every row, with
// multiplier 0 on the pivot row.  X[s][p_t] = M[p_s][t], p_s the pivot row of
// column s.  9.0e3 clocks; one warp with whole rows in registers 1.8e4, a
// barrier per column instead of per panel 1.0e4.
//
// Every: pivots of any size, and a column of zeros is left out; true if there was
// one.  Otherwise true, and nothing stored, if a pivot was zero or outside
// reciprocal's range (all four warps see the same pivots).
template <bool Every>
__device__ __forceinline__ bool invert32_pass(double *M, int ld, int n,
                                              double (*col)[kPanel][kHalf], int *piv)
{
    constexpr int R = kHalf / kPanel;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double a[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int c = kPanel * i + w;
        a[i] = lane < n && c < n ? M[lane * ld + c] : (lane == c ? 1.0 : 0.0);
    }
    bool bad = false, used = false;
    int step = 0;
    double scale = 0.0;
#pragma unroll 1
    for (int P = 0; P < R; ++P) {
        col[P & 1][w][lane] = a[0];
        pivot_sync();
        double pan[kPanel];
#pragma unroll
        for (int t = 0; t < kPanel; ++t) pan[t] = col[P & 1][t][lane];
#pragma unroll
        for (int t = 0; t < kPanel; ++t) {
            // the high word of |a| (its last five bits given up for the lane);
            // 0 for a row already used: one row at least is free
            const unsigned hi = pivot_bits(pan[t]) & ~63u;
            const unsigned best =
                __reduce_max_sync(0xffffffffu, used ? 0u : hi | 32u | (unsigned)lane);
            const double rinv = Every ? reciprocal_scaled(pan[t]) : reciprocal(pan[t]);
            const int p = best & 31;
            const bool me = lane == p;
            double inv = __shfl_sync(0xffffffffu, rinv, p);
            if (!Every) {
                bad = bad || !fast_pivot(best);
            } else if (best < 64u) {
                inv = 0.0;
                bad = true;
            }
            const double m = me ? 0.0 : pan[t] * inv;
#pragma unroll
            for (int j = 0; j < kPanel; ++j)
                if (j != t) pan[j] -= m * __shfl_sync(0xffffffffu, pan[j], p);
            pan[t] = me ? 1.0 : -m;
#pragma unroll
            for (int i = 1; i < R; ++i) a[i] -= m * __shfl_sync(0xffffffffu, a[i], p);
            if (me) {
                used = true;
                step = kPanel * P + t;
                scale = inv;
                if (w == 0) piv[step] = lane;
            }
        }
#pragma unroll
        for (int i = 1; i < R; ++i) a[i - 1] = a[i];
        a[R - 1] = w == 0 ? pan[0] : w == 1 ? pan[1] : w == 2 ? pan[2] : pan[3];
    }
    pivot_sync();
    if (!Every && bad) return true;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int c = piv[kPanel * i + w];
        if (step < n && c < n) M[step * ld + c] = a[i] * scale;
    }
    return bad;
}

// Returns whether a pivot column was zero.
__device__ __forceinline__ bool invert32(double *M, int ld, int n, double (*col)[kPanel][kHalf],
                                         int *piv)
{
    return invert32_pass<false>(M, ld, n, col, piv) && invert32_pass<true>(M, ld, n, col, piv);
}

// The w x w block at sm.M (padded to 64 x 64 by the identity) inverted in
// place by the CTA's first four warps; sm.M must be visible to them.
__device__ __forceinline__ void invert_block(PivotSmem &sm, int w, int *flag)
{
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    bool bad = false;
    const int nh = w > kHalf ? 2 : 1;
#pragma unroll 1
    for (int h = 0; h < nh; ++h) {
        // the step's block X, its row O, its column C and the rest Y
        double *X = sm.M + h * (kHalf * kLdX + kHalf), *Y = sm.M + (1 - h) * (kHalf * kLdX + kHalf);
        double *O = sm.M + (h ? kHalf * kLdX : kHalf), *C = sm.M + (h ? kHalf : kHalf * kLdX);
        bad |= invert32(X, kLdX, kHalf, sm.col, sm.piv);
        pivot_sync();
        if (nh == 1) break;
#pragma unroll 1
        for (int i = 0; i < 3; ++i) {   // O = X O, Y -= C O, C = -C X; a warp's 8 rows
            const double *L = i == 0 ? X : C, *B = i == 2 ? X : O;
            double *D = i == 0 ? O : i == 1 ? Y : C;
            double acc[4][2] = {};
#pragma unroll 2
            for (int k4 = 0; k4 < kHalf; k4 += 4) {
                const double a = L[(8 * wid + g) * kLdX + k4 + t];
#pragma unroll
                for (int n = 0; n < 4; ++n)
                    dmma_8x8x4(acc[n][0], acc[n][1], a, B[(k4 + t) * kLdX + 8 * n + g]);
            }
            pivot_sync();
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                double *d = D + (8 * wid + g) * kLdX + 8 * n + 2 * t;
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    d[u] = i == 0 ? acc[n][u] : (i == 1 ? d[u] : 0.0) - acc[n][u];
            }
            pivot_sync();
        }
    }
    if (bad && tid == 0) atomicOr(flag, 1);
}

// sm.M's w x w block to the front (leading dimension f), four warps.
template <class T>
__device__ __forceinline__ void store_block(const PivotSmem &sm, int w, T *A, int f)
{
    const int c = threadIdx.x & (kPiv - 1);
#pragma unroll 8
    for (int r = threadIdx.x / kPiv; r < kPiv; r += kInvThreads / kPiv)
        if (r < w && c < w) A[(long long)r * f + c] = (T)sm.M[r * kLdX + c];
}

// A level's fronts get their children's contribution blocks, and the first
// step's pivot blocks are inverted: the first of a front's `per` CTAs adds the
// children's entries of that block, inverts it and stores X; the others (none
// on a level without children) add the rest, 32 rows x 256 columns each.  A
// front's CTAs are neighbours in the grid, here and in the step's kernels:
// with the first CTAs of all fronts in front the large levels lose their L2
// locality (8.8 against 7.1 ms on all levels of 1025 x 1025).
template <class T>
__global__ void __launch_bounds__(32 * kExtWarps) k_assemble(int q0, int per, int nc,
                                                             const AssemblyMaps m, T *F, int *flag)
{
    __shared__ __align__(16) PivotSmem sm;
    const int q = q0 + blockIdx.x / per, t = blockIdx.x % per;
    const Assembly<T> a = assembly_of(m, q, F);
    if (t > 0) {
        const int r0 = ((t - 1) / nc) * (kExtRows * kExtWarps) + (threadIdx.x >> 5) * kExtRows;
        const int c0 = ((t - 1) % nc) * kExtCols;
        if (r0 < a.f && c0 < a.f) extend_rows(a, r0, c0);
        return;
    }
    constexpr int R = kPiv * kPiv / (32 * kExtWarps), step = 32 * kExtWarps / kPiv;
    const int c = threadIdx.x & (kPiv - 1), r0 = threadIdx.x / kPiv;
    T v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = r0 + i * step;
        v[i] = (r < a.w && c < a.w) ? a.A[(long long)r * a.f + c] : (r == c ? T(1) : T(0));
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int j = a.src[h] && c < a.w ? a.map[h][c] : -1;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int r = r0 + i * step, k = j >= 0 && r < a.w ? a.map[h][r] : -1;
            if (k >= 0) v[i] += a.src[h][(long long)k * a.fc[h] + j];
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) sm.M[(r0 + i * step) * kLdX + c] = (double)v[i];
    __syncthreads();
    if (threadIdx.x >= kInvThreads) return;
    invert_block(sm, a.w, flag);
    store_block(sm, a.w, a.A, a.f);
}

// Accumulator of one 64 x 64 output tile of a CTA of 256 threads, fed
// kSlice-wide slices of its operands through shared memory.  A thread's
// outputs come in groups of kVec consecutive columns (each()).
//   double: FP64 tensor cores, mma.sync m8n8k4 (tcgen05 has no FP64 kind).
//           Warp w owns rows 32 (w / 4) .. + 32 and columns 16 (w % 4) .. +
//           16, i.e. 4 x 2 8x8 blocks; per k step of 4 a lane holds A[8 mi +
//           g][t], B[t][8 ni + g] and the outputs [8 mi + g][8 ni + 2 t + j]
//           (g = lane / 4, t = lane % 4).  Row strides of 36 and 72 doubles
//           spread a warp's 32 fragment reads evenly over the shared-memory
//           banks (two wavefronts, the minimum for 256 bytes).
//   float:  CUDA cores, each thread rows ty + 16 a and columns 4 tx .. + 4
//           (a, 4 of each); operands read four at a time.
template <class T> struct Tile;

template <> struct Tile<double> {
    static constexpr int kVec = 2;
    static constexpr int kLdA = kSlice + 4, kLdB = kTile + 8;
    struct Smem {
        double A[kTile][kLdA];
        double B[kSlice][kLdB];
    };
    double acc[4][2][2];
    // nr x nc: the tile's valid rows and columns (8 x 8 blocks beyond are skipped)
    __device__ __forceinline__ void mac(const Smem &s, int nr, int nc)
    {
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
        const int wr = (w >> 2) * 32, wc = (w & 3) * 16;
        if (wc >= nc) return;
        nr -= wr;
        // whole rows without a test between the products, so that the
        // fragment loads of the next ones are issued ahead
        if (nr > 24) {
#pragma unroll
            for (int k = 0; k < kSlice; k += 4) {
                double a[4], b[2];
#pragma unroll
                for (int ni = 0; ni < 2; ++ni) b[ni] = s.B[k + t][wc + 8 * ni + g];
#pragma unroll
                for (int mi = 0; mi < 4; ++mi) a[mi] = s.A[wr + 8 * mi + g][k + t];
#pragma unroll
                for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                    for (int ni = 0; ni < 2; ++ni)
                        dmma_8x8x4(acc[mi][ni][0], acc[mi][ni][1], a[mi], b[ni]);
            }
            return;
        }
#pragma unroll 2
        for (int k = 0; k < kSlice; k += 4) {
            double b[2];
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) b[ni] = s.B[k + t][wc + 8 * ni + g];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
                if (8 * mi < nr) {
                    const double a = s.A[wr + 8 * mi + g][k + t];
#pragma unroll
                    for (int ni = 0; ni < 2; ++ni)
                        dmma_8x8x4(acc[mi][ni][0], acc[mi][ni][1], a, b[ni]);
                }
        }
    }
    // fn(row, first column, the kVec accumulators)
    template <class Fn> __device__ __forceinline__ void each(Fn fn)
    {
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
        const int wr = (w >> 2) * 32, wc = (w & 3) * 16;
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) fn(wr + 8 * mi + g, wc + 8 * ni + 2 * t, acc[mi][ni]);
    }
};

template <> struct Tile<float> {
    static constexpr int kVec = 2;
    static constexpr int kLdA = kSlice + 4, kLdB = kTile;
    struct Smem {
        float A[kTile][kLdA];
        float B[kSlice][kLdB];
    };
    float acc[4][2][2];
    __device__ __forceinline__ void mac(const Smem &s, int, int)
    {
        const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
#pragma unroll 2
        for (int k = 0; k < kSlice; k += 4) {
            float4 av[4], bv[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) av[a] = *reinterpret_cast<const float4 *>(&s.A[ty + 16 * a][k]);
#pragma unroll
            for (int u = 0; u < 4; ++u) bv[u] = *reinterpret_cast<const float4 *>(&s.B[k + u][4 * tx]);
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const float x[4] = {av[a].x, av[a].y, av[a].z, av[a].w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    acc[a][0][0] += x[u] * bv[u].x;
                    acc[a][0][1] += x[u] * bv[u].y;
                    acc[a][1][0] += x[u] * bv[u].z;
                    acc[a][1][1] += x[u] * bv[u].w;
                }
            }
        }
    }
    template <class Fn> __device__ __forceinline__ void each(Fn fn)
    {
        const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) fn(ty + 16 * a, 4 * tx + 2 * b, acc[a][b]);
    }
};

template <class T> struct Pair;
template <> struct Pair<double> { using type = double2; };
template <> struct Pair<float> { using type = float2; };

// One slice of the operands: A rows [0, nr) x inner [k, k + kSlice) below ke
// of src (leading dimension lda), B inner rows x columns [0, nc).  Two
// elements per copy: f, S and every offset here are even (two unknowns per
// node), so rows are aligned to two elements and no pair straddles an edge.
template <class T>
__device__ __forceinline__ void stage_slice(typename Tile<T>::Smem &s, const T *a, long long lda,
                                            int nr, const T *b, long long ldb, int nc, int k,
                                            int ke)
{
    constexpr int B = 2 * (int)sizeof(T);
    constexpr int pa = kSlice / 2, pb = kTile / 2;
#pragma unroll
    for (int i = 0; i < kTile * pa / 256; ++i) {
        const int e = threadIdx.x + 256 * i, r = e / pa, t = 2 * (e % pa);
        const bool ok = r < nr && k + t < ke;
        cp_async<B>(&s.A[r][t], ok ? a + r * lda + k + t : a, ok);
    }
#pragma unroll
    for (int i = 0; i < kSlice * pb / 256; ++i) {
        const int e = threadIdx.x + 256 * i, t = e / pb, c = 2 * (e % pb);
        const bool ok = c < nc && k + t < ke;
        cp_async<B>(&s.B[t][c], ok ? b + (k + t) * ldb + c : b, ok);
    }
    cp_async_commit();
}

// acc += A B over the inner range [0, ke), ke <= 2 kSlice: both slices in
// flight at once, the second lands while the first is multiplied.
template <class T>
__device__ __forceinline__ void tile_product(Tile<T> &t, typename Tile<T>::Smem *sm, const T *a,
                                             long long lda, int nr, const T *b, long long ldb,
                                             int nc, int ke)
{
    static_assert(kPiv <= 2 * kSlice, "a step's inner range fits two slices");
    stage_slice<T>(sm[0], a, lda, nr, b, ldb, nc, 0, ke);
    if (ke > kSlice) {
        stage_slice<T>(sm[1], a, lda, nr, b, ldb, nc, kSlice, ke);
        cp_async_wait<1>();
        __syncthreads();
        t.mac(sm[0], nr, nc);
        cp_async_wait<0>();
        __syncthreads();
        t.mac(sm[1], nr, nc);
    } else {
        cp_async_wait<0>();
        __syncthreads();
        t.mac(sm[0], nr, nc);
    }
}

// Dynamic shared memory of k_row_block and k_update: two operand slices, or
// the next pivot block's inversion in their place.
template <class T> constexpr size_t tile_smem_bytes()
{
    return std::max(2 * sizeof(typename Tile<T>::Smem), sizeof(PivotSmem));
}

// R = X A_KJ of a step, in place, 64 columns per CTA (a front's blocks [0, nt)); blocks
// [nt, 2 nt) copy 64 rows of the pivot columns A_IK to the step's scratch C
// (front rows x kPiv, zero beyond the step's pivots; v0 = the level's first
// voff), where k_update reads them while it overwrites A_IK.
template <class T>
__global__ void __launch_bounds__(256) k_row_block(int q0, int k, int nt, int v0,
                                                   const int *__restrict__ S_,
                                                   const int *__restrict__ f_,
                                                   const long long *__restrict__ foff,
                                                   const int *__restrict__ voff, T *F, T *C)
{
    using P2 = typename Pair<T>::type;
    extern __shared__ __align__(16) unsigned char tile_raw[];
    const int q = q0 + blockIdx.x / (2 * nt), tile = blockIdx.x % (2 * nt);
    const int S = S_[q], f = f_[q];
    T *A = F + foff[q];
    const int w = min(kPiv, S - k), e = k + w;
    if (S <= k) return;
    if (tile >= nt) {
        const int r0 = (tile - nt) * kTile;
        const int nr = min(kTile, f - r0);
        T *Cq = C + (long long)(voff[q] - v0) * kPiv;
        for (int i = threadIdx.x; i < nr * (kPiv / 2); i += 256) {
            const int r = r0 + i / (kPiv / 2), t = 2 * (i % (kPiv / 2));
            P2 v;
            v.x = v.y = T(0);
            if (t < w) v = *reinterpret_cast<const P2 *>(A + (long long)r * f + k + t);
            *reinterpret_cast<P2 *>(Cq + (long long)r * kPiv + t) = v;
        }
        return;
    }
    const int c0 = tile * kTile;
    if (c0 >= f || (c0 >= k && min(c0 + kTile, f) <= e)) return;
    typename Tile<T>::Smem *sm = reinterpret_cast<typename Tile<T>::Smem *>(tile_raw);
    Tile<T> t;
    t.each([](int, int, T (&v)[2]) { v[0] = v[1] = T(0); });
    T *Ak = A + (long long)k * f;
    tile_product<T>(t, sm, Ak + k, f, w, Ak + c0, f, min(kTile, f - c0), w);
    // every entry of the block's rows in these columns is in shared memory
    t.each([&](int r, int cc, T (&v)[2]) {
        const int c = c0 + cc;
        if (r < w && c < f && !(c >= k && c < e)) {
            P2 o;
            o.x = v[0];
            o.y = v[1];
            *reinterpret_cast<P2 *>(Ak + (long long)r * f + c) = o;
        }
    });
}

// A_IJ -= C_I R_J on one 64 x 64 tile (rows outside the pivots), A_IK =
// -C_I X in the pivot columns (R_K = X in place).  Tile 0 of a front is the
// next step's pivot block, whose inverse this CTA stores in its place.
template <class T>
__global__ void __launch_bounds__(256, 3) k_update(int q0, int k, int nt, int v0,
                                                   const int *__restrict__ S_,
                                                   const int *__restrict__ f_,
                                                   const long long *__restrict__ foff,
                                                   const int *__restrict__ voff, T *F, const T *C,
                                                   int *flag)
{
    using P2 = typename Pair<T>::type;
    extern __shared__ __align__(16) unsigned char tile_raw[];
    const int q = q0 + blockIdx.x / (nt * nt), t = blockIdx.x % (nt * nt);
    const int S = S_[q], f = f_[q];
    const int w = min(kPiv, S - k), e = k + w;
    T *A = F + foff[q];
    const T *Cq = C + (long long)(voff[q] - v0) * kPiv;
    if (S <= k) return;
    // tiles in row order, the one of the next pivot block exchanged with the first
    const int next = e < S ? (e / kTile) * (nt + 1) : -1;
    const int t0 = next < 0 ? t : (t == 0 ? next : (t == next ? 0 : t));
    const int r0 = (t0 / nt) * kTile, c0 = (t0 % nt) * kTile;
    if (r0 >= f || c0 >= f || (r0 >= k && min(r0 + kTile, f) <= e)) return;
    typename Tile<T>::Smem *sm = reinterpret_cast<typename Tile<T>::Smem *>(tile_raw);
    Tile<T> acc;
    // the old entries, negated: loaded while the operands are on their way
    acc.each([&](int rr, int cc, T (&v)[2]) {
        const int r = r0 + rr, c = c0 + cc;
        v[0] = v[1] = T(0);
        if (r < f && c < f && !(c >= k && c < e)) {
            const P2 o = *reinterpret_cast<const P2 *>(A + (long long)r * f + c);
            v[0] = -o.x;
            v[1] = -o.y;
        }
    });
    tile_product<T>(acc, sm, Cq + (long long)r0 * kPiv, kPiv, min(kTile, f - r0),
                    A + (long long)k * f + c0, f, min(kTile, f - c0), w);
    const bool pivots = t0 == next;
    const int wn = pivots ? min(kPiv, S - e) : 0;   // the block's pivots
    PivotSmem &ps = *reinterpret_cast<PivotSmem *>(tile_raw);
    if (pivots) __syncthreads();   // the operands' buffers are free
    acc.each([&](int rr, int cc, T (&v)[2]) {
        const int r = r0 + rr, c = c0 + cc;
        if (pivots) {
            const bool in = rr < wn && cc < wn;
#pragma unroll
            for (int u = 0; u < 2; ++u)
                ps.M[rr * kLdX + cc + u] = in ? -(double)v[u] : (rr == cc + u ? 1.0 : 0.0);
            if (in) return;
        }
        if (r < f && c < f && !(r >= k && r < e)) {
            P2 o;
            o.x = -v[0];
            o.y = -v[1];
            *reinterpret_cast<P2 *>(A + (long long)r * f + c) = o;
        }
    });
    if (!pivots) return;
    __syncthreads();
    if (threadIdx.x >= kInvThreads) return;
    invert_block(ps, wn, flag);
    store_block(ps, wn, A + (long long)e * f + e, f);
}

// The update of a full step (64 pivots in every front) with FP64 fronts and
// many tiles: one CTA per SM, four producer warps that fetch the next tile's
// operands and old entries while eight warps multiply the current one.  A CTA
// takes strips of `len` tiles of a row of tiles from a counter, the next pivot
// blocks first; a strip's C_I is fetched once.  The FP64 tensor cores bound it
// (37 TF/s, 2.1 us per tile and SM): 16 fronts of 2562 take 0.53 ms, 24.9 TF/s,
// against 0.64 ms in k_update, whose reads of the old entries (64 bytes in each
// of 8 rows per load) hold up the products whether they come early or late.
// Measured and not taken, on the same fronts: bulk copies per row (0.85 ms),
// two groups of four warps in turn (0.59), two of eight that read the old
// entries themselves (0.65), strips with two CTAs per SM (0.76).
//
// No wait depends on another CTA, so none should run out; if one does, bit 4 of
// *err is set and the CTA ends.  Each side then leaves through a barrier that all
// of its threads reach: the producers' at the next ticket (stop, by the ticket's
// parity, so that a thread already past it cannot change what a slower one reads),
// the multiplying warps' at the next pivot tile or at the end (leave).
constexpr int kWideWarps = 8, kWideProducers = 128;

struct WideShared {
    struct Stage {
        double B[kPiv][kTile + 8], C[kTile][kTile + 8];
    } st[2];
    double A[2][kTile][kPiv + 4];
    unsigned long long full[2], empty[2];
    struct Work {
        int q, r0, c0, a;   // front (-1: no more), first row and column, A's buffer
    } tile[2];
    int ticket[2];
    volatile int quit;   // a wait ran out: the others end
    int stop[2], leave;  // ... and the producers, the multiplying warps leave together
};
static_assert(sizeof(PivotSmem) <= sizeof(WideShared::Stage), "the inversion uses a stage");

__global__ void __launch_bounds__(32 * kWideWarps + kWideProducers, 1)
    k_update_wide(int q0, int nq, int k, int nt, int len, int v0, const int *__restrict__ S_,
                  const int *__restrict__ f_, const long long *__restrict__ foff,
                  const int *__restrict__ voff, double *F, const double *C, int *ticket, int *flag,
                  int limit, int *err)
{
    extern __shared__ __align__(16) unsigned char tile_raw[];
    WideShared &sh = *reinterpret_cast<WideShared *>(tile_raw);
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&sh.full[s], kWideProducers + 1);
            mbar_init(&sh.empty[s], kWideWarps);
            sh.stop[s] = 0;
        }
        sh.quit = sh.leave = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int kt = k / kTile;   // the pivots' tile row and column
    if (wid >= kWideWarps) {
        const int ns = (nt + len - 1) / len, p = threadIdx.x - 32 * kWideWarps;
        const long long total = nq + (long long)nq * nt * ns;
        int n = 0, a = 0;
        bool failed = false;
        // the stage of the next tile once it is free; false: given up
        auto stage = [&](int q, int r0, int c0) {
            const int s = n & 1;
            if (n >= 2 && !mbar_wait(&sh.empty[s], ((n >> 1) - 1) & 1, &sh.quit, limit)) {
                atomicOr(err, 4);
                sh.quit = 1;
                failed = true;
                return false;
            }
            if (p == 0) {
                sh.tile[s] = {q, r0, c0, a};
                mbar_arrive(&sh.full[s]);
            }
            return true;
        };
        int next = p == 0 ? atomicAdd(ticket, 1) : 0;
        for (int i = 0;; ++i) {
            if (p == 0) sh.ticket[i & 1] = next;
            if (failed) sh.stop[i & 1] = 1;
            asm volatile("bar.sync 3, %0;" ::"n"(kWideProducers) : "memory");
            const int t = sh.ticket[i & 1];
            failed = sh.stop[i & 1];
            if (failed || t >= total) break;
            if (p == 0) next = atomicAdd(ticket, 1);
            const bool pivots = t < nq;
            const int u = t - nq, q = q0 + (pivots ? t : u / (nt * ns));
            const int S = S_[q], f = f_[q], rt = pivots ? kt + 1 : u / ns % nt;
            const int r0 = rt * kTile, nr = min(kTile, f - r0);
            if (nr <= 0 || rt == kt || (pivots && k + kPiv >= S)) continue;
            const double *A = F + foff[q], *R = A + (long long)k * f;
            const double *Ci = C + ((long long)(voff[q] - v0) + r0) * kPiv;
            const int j0 = pivots ? rt : u % ns * len, j1 = pivots ? rt + 1 : min(nt, j0 + len);
            const int pr = p / (kTile / 2), pc = 2 * (p % (kTile / 2));   // its rows, columns
            constexpr int step = kWideProducers / (kTile / 2);
            bool first = true;
            for (int j = j0; j < j1; ++j) {
                const int c0 = j * kTile, nc = min(kTile, f - c0);
                if (nc <= 0 || (!pivots && rt == kt + 1 && j == rt && k + kPiv < S)) continue;
                if (!stage(q, r0, c0)) break;
                WideShared::Stage &st = sh.st[n & 1];
                if (first)
#pragma unroll 4
                    for (int r = pr; r < nr; r += step)
                        cp_async<16>(&sh.A[a][r][pc], Ci + r * kPiv + pc, true);
                if (pc < nc) {
#pragma unroll 4
                    for (int r = pr; r < kPiv; r += step)
                        cp_async<16>(&st.B[r][pc], R + (long long)r * f + c0 + pc, true);
                    if (j != kt)   // the pivot columns are overwritten
#pragma unroll 4
                        for (int r = pr; r < nr; r += step)
                            cp_async<16>(&st.C[r][pc], A + (long long)(r0 + r) * f + c0 + pc, true);
                }
                mbar_arrive_copies(&sh.full[n & 1]);
                first = false;
                ++n;
            }
            if (!first) a ^= 1;   // the other buffer's strip is done two tiles on
        }
        if (!failed && stage(-1, 0, 0)) mbar_arrive(&sh.full[n & 1]);
        asm volatile("cp.async.wait_all;" ::: "memory");   // no copy outlives its thread
        return;
    }
    const int g = lane >> 2, t = lane & 3, wr = (wid >> 2) * 32, wc = (wid & 3) * 16;
    for (int n = 0;; ++n) {
        const int s = n & 1;
        const bool ok = mbar_wait_warp(&sh.full[s], (n >> 1) & 1, &sh.quit, limit);
        if (!ok && lane == 0) {
            atomicOr(err, 4);
            sh.quit = sh.leave = 1;
        }
        const WideShared::Work w = sh.tile[s];
        if (!ok || w.q < 0) {
            asm volatile("bar.sync 2, %0;" ::"n"(32 * kWideWarps) : "memory");
            return;
        }
        WideShared::Stage &st = sh.st[s];
        const int S = S_[w.q], f = f_[w.q], r0 = w.r0 + wr + g, c0 = w.c0 + wc + 2 * t;
        double *A = F + foff[w.q];
        const bool old = w.c0 != k, pivots = w.r0 == k + kPiv && w.c0 == w.r0 && w.r0 < S;
        double acc[4][2][2];
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) {
                double2 v = *reinterpret_cast<const double2 *>(
                    &st.C[wr + 8 * mi + g][wc + 8 * ni + 2 * t]);
                if (!old) v = make_double2(0.0, 0.0);
                acc[mi][ni][0] = -v.x;
                acc[mi][ni][1] = -v.y;
            }
        if (w.r0 + wr < f && w.c0 + wc < f) {
            const double(*sa)[kPiv + 4] = sh.A[w.a];
#pragma unroll 8
            for (int kk = 0; kk < kPiv; kk += 4) {
                double a[4], b[2];
#pragma unroll
                for (int ni = 0; ni < 2; ++ni) b[ni] = st.B[kk + t][wc + 8 * ni + g];
#pragma unroll
                for (int mi = 0; mi < 4; ++mi) a[mi] = sa[wr + 8 * mi + g][kk + t];
#pragma unroll
                for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                    for (int ni = 0; ni < 2; ++ni)
                        dmma_8x8x4(acc[mi][ni][0], acc[mi][ni][1], a[mi], b[ni]);
            }
        }
        __syncwarp();
        if (!pivots && lane == 0) mbar_arrive(&sh.empty[s]);
        const int wn = pivots ? min(kPiv, S - w.r0) : 0;   // the next block's pivots
        PivotSmem &ps = *reinterpret_cast<PivotSmem *>(&st);
        if (pivots) {
            asm volatile("bar.sync 2, %0;" ::"n"(32 * kWideWarps) : "memory");
            if (sh.leave) return;
        }
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) {
                const int r = r0 + 8 * mi, c = c0 + 8 * ni, rr = r - w.r0, cc = c - w.c0;
                const bool in = rr < wn && cc < wn;
                if (pivots) {
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        ps.M[rr * kLdX + cc + u] =
                            in ? -acc[mi][ni][u] : (rr == cc + u ? 1.0 : 0.0);
                }
                if (!in && r < f && c < f)
                    *reinterpret_cast<double2 *>(A + (long long)r * f + c) =
                        make_double2(-acc[mi][ni][0], -acc[mi][ni][1]);
            }
        if (!pivots) continue;
        asm volatile("bar.sync 2, %0;" ::"n"(32 * kWideWarps) : "memory");
        if (threadIdx.x < kInvThreads) {
            invert_block(ps, wn, flag);
            store_block(ps, wn, A + (long long)w.r0 * f + w.r0, f);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.empty[s]);
    }
}

// ------------------------------------------------------------------ leaves
// A front without children holds matrix entries only: A12 and A21 are sparse (a
// struct variable couples to a few pivots next to it) and A22 is zero.  So only
// A11 is eliminated densely, and H = A11^-1 A12, G = A21 A11^-1 and the Schur
// complement -G A12 are sums over those few entries: 2 S^3 flops and one write
// of the front instead of 2 S f^2 and a read and a write of it per step, and no
// zero fill and scatter before.
//
// Setup (k_leaf_lists, once per plan): each leaf's A12 entries by column and
// A21 entries by row, as (CSR entry, pivot index) in `list` at the leaf's range
// of assembly entries; ptr12[uoff + q + j] / ptr21[...] the first entry of
// struct variable j, j = 0 .. m.  stat[0]: the most A12 entries of a leaf;
// stat[1]: leaves with more than the setup's arrays hold.
constexpr int kLeafMaxS = 128;
constexpr int kLeafMaxEntries = 2048;   // A12 or A21 entries of a leaf

__global__ void __launch_bounds__(256) k_leaf_lists(const int *__restrict__ S_,
                                                    const int *__restrict__ f_,
                                                    const long long *__restrict__ foff,
                                                    const int *__restrict__ uoff,
                                                    const long long *__restrict__ aoff,
                                                    const int *__restrict__ csr,
                                                    const long long *__restrict__ pos, int2 *list,
                                                    long long *ptr12, long long *ptr21, int *stat)
{
    __shared__ int key[2][kLeafMaxEntries], id[2][kLeafMaxEntries], cnt[2];
    const int q = blockIdx.x, S = S_[q], f = f_[q], m = f - S;
    const long long a0 = aoff[q], a1 = aoff[q + 1];
    if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
    __syncthreads();
    for (long long e = a0 + threadIdx.x; e < a1; e += blockDim.x) {
        const int p = (int)(pos[e] - foff[q]), r = p / f, c = p - r * f;
        if (r < S && c < S) continue;
        const int h = r < S ? 0 : 1;   // A12, keyed by (column, row); A21 by (row, column)
        const int k = atomicAdd(&cnt[h], 1);
        if (k < kLeafMaxEntries) {
            key[h][k] = h == 0 ? c * f + r : p;
            id[h][k] = csr[e];
        }
    }
    __syncthreads();
    const int n0 = cnt[0], n1 = cnt[1];
    if (n0 > kLeafMaxEntries || n1 > kLeafMaxEntries) {
        if (threadIdx.x == 0) atomicAdd(&stat[1], 1);
        return;
    }
    if (threadIdx.x == 0) atomicMax(&stat[0], n0);
    // every entry's place by counting: the keys differ, so it is the same in
    // every run whatever order the entries came in
    for (int h = 0; h < 2; ++h) {
        const int n = h == 0 ? n0 : n1;
        const long long base = a0 + (h == 0 ? 0 : n0);
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            int rank = 0;
            for (int j = 0; j < n; ++j) rank += key[h][j] < key[h][i];
            list[base + rank] = make_int2(id[h][i], key[h][i] % f);
        }
        for (int j = threadIdx.x; j <= m; j += blockDim.x) {
            int before = 0;
            for (int i = 0; i < n; ++i) before += key[h][i] / f < S + j;
            (h == 0 ? ptr12 : ptr21)[uoff[q] + q + j] = base + before;
        }
    }
}

struct LeafMaps {
    const int *S, *f, *voff, *uoff, *vars, *csr, *row;
    const long long *foff, *aoff, *pos, *ptr12, *ptr21;
    const int2 *list;
};

// Leading dimension of a leaf's pivot block in shared memory: 2 modulo 16, so
// that a fragment read takes two wavefronts, the least for 256 bytes.
__host__ __device__ inline int leaf_ld(int S) { return (S + 13) / 16 * 16 + 2; }
inline size_t leaf_smem(int maxS, int maxf, int maxe, int gwarps)
{
    const int rows = (maxS + 7) / 8 * 8;
    return ((size_t)rows * leaf_ld(rows) + gwarps * (size_t)rows + maxe) * sizeof(double) +
           (size_t)(maxf + 1) * sizeof(int) + (size_t)maxe * sizeof(short);
}

// sum of x[c] v over a list's entries, four loads in flight
__device__ __forceinline__ double sparse_dot(const double *x, const short *c, const double *v,
                                             int b, int e)
{
    double s0 = 0.0, s1 = 0.0;
    for (; b < e; b += 4) {
        int k[4];
        double a[4], y[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            k[u] = b + u < e ? c[b + u] : 0;
            a[u] = b + u < e ? v[b + u] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) y[u] = b + u < e ? x[k[u]] : 0.0;
        s0 += y[0] * a[0] + y[2] * a[2];
        s1 += y[1] * a[1] + y[3] * a[3];
    }
    return s0 + s1;
}

// One CTA per leaf.  A11 in shared memory is inverted in FP64 by Gauss-Jordan
// blocks of 32 (invert32 by four warps, the products by all eight on the FP64
// tensor cores, a block row of eight rows per warp); then the sparse sums, one
// front row per warp.  maxrows, maxf, maxe: the level's largest pivot count
// (rounded up to 8), front and number of A12 entries; gwarps: the warps that have
// room for a row of G (fewer than eight where that lets two CTAs share an SM).
template <class T>
__global__ void __launch_bounds__(256, 2) k_leaf(const LeafMaps L, int maxrows, int maxf, int maxe,
                                                 int gwarps,
                                                 const double *__restrict__ val,
                                                 const double *__restrict__ rs, T *F, int *flag)
{
    extern __shared__ __align__(16) unsigned char leaf_raw[];
    __shared__ double col[2][kPanel][kHalf];
    __shared__ int piv[kHalf];
    const int q = blockIdx.x, S = L.S[q], f = L.f[q], vo = L.voff[q], m = f - S;
    const int n8 = (S + 7) / 8, ld = leaf_ld(8 * n8);
    double *M = reinterpret_cast<double *>(leaf_raw);
    double *grow = M + (size_t)maxrows * leaf_ld(maxrows);   // a row of G per warp
    double *ev = grow + gwarps * (size_t)maxrows;
    int *p12 = reinterpret_cast<int *>(ev + maxe);           // column j's entries [p12[j], p12[j+1])
    short *ec = reinterpret_cast<short *>(p12 + maxf + 1);   // an entry's pivot
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const long long a0 = L.aoff[q], a1 = L.aoff[q + 1], u0 = L.uoff[q] + q;
    for (int i = tid; i < 8 * n8 * ld; i += 256) M[i] = 0.0;
    // the A12 values (row scaled), in list order
    const long long e12 = L.ptr12[u0], e21 = L.ptr21[u0];
    for (int j = tid; j <= m; j += 256) p12[j] = (int)(L.ptr12[u0 + j] - e12);
    for (long long e = e12 + tid; e < e21; e += 256) {
        const int2 x = L.list[e];
        ev[e - e12] = val[x.x] * rs[L.vars[vo + x.y]];
        ec[e - e12] = (short)x.y;
    }
    __syncthreads();
    const long long fo = L.foff[q];
    for (long long e = a0 + tid; e < a1; e += 256) {
        const int p = (int)(L.pos[e] - fo), r = p / f, c = p - r * f;
        if (r < S && c < S) M[r * ld + c] = val[L.csr[e]] * rs[L.row[e]];
    }
    __syncthreads();
    bool bad = false;
#pragma unroll 1
    for (int k = 0; k < S; k += kHalf) {
        const int w = min(kHalf, S - k), b0 = k / 8, b1 = b0 + (w + 7) / 8;   // its 8-blocks
        if (tid < kInvThreads) bad |= invert32(M + k * ld + k, ld, w, col, piv);
        __syncthreads();
        // R = X A_KJ, a warp's 8-column blocks (two at most), in place
        double r[2][4][2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int nb = wid + 8 * u;
#pragma unroll
            for (int i = 0; i < 4; ++i) r[u][i][0] = r[u][i][1] = 0.0;
            if (nb >= n8 || (nb >= b0 && nb < b1)) continue;
#pragma unroll 2
            for (int k4 = 0; k4 < w; k4 += 4) {
                const double b = M[(k + k4 + t) * ld + 8 * nb + g];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (8 * i < w)
                        dmma_8x8x4(r[u][i][0], r[u][i][1], M[(k + 8 * i + g) * ld + k + k4 + t], b);
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int nb = wid + 8 * u;
            if (nb >= n8 || (nb >= b0 && nb < b1)) continue;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (8 * i < w)
                    *reinterpret_cast<double2 *>(&M[(k + 8 * i + g) * ld + 8 * nb + 2 * t]) =
                        make_double2(r[u][i][0], r[u][i][1]);
        }
        __syncthreads();
        // the other rows: A_IJ -= A_IK R, then A_IK = -A_IK X
        for (int mb = wid; mb < n8; mb += 8) {
            if (mb >= b0 && mb < b1) continue;
            double a[kHalf / 4];
#pragma unroll
            for (int k4 = 0; k4 < kHalf / 4; ++k4)
                a[k4] = 4 * k4 < w ? M[(8 * mb + g) * ld + k + 4 * k4 + t] : 0.0;
            __syncwarp();   // the row's A_IK is in registers
#pragma unroll 1
            for (int nb = 0; nb < n8; nb += 4) {
                double acc[4][2];
                double *d = &M[(8 * mb + g) * ld + 8 * nb + 2 * t];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const bool old = nb + u < n8 && !(nb + u >= b0 && nb + u < b1);
                    acc[u][0] = old ? -d[8 * u] : 0.0;
                    acc[u][1] = old ? -d[8 * u + 1] : 0.0;
                }
#pragma unroll
                for (int k4 = 0; k4 < kHalf / 4; ++k4)
                    if (4 * k4 < w) {
                        const double *b = &M[(k + 4 * k4 + t) * ld + 8 * nb + g];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (nb + u < n8) dmma_8x8x4(acc[u][0], acc[u][1], a[k4], b[8 * u]);
                    }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (nb + u < n8)
                        *reinterpret_cast<double2 *>(d + 8 * u) = make_double2(-acc[u][0], -acc[u][1]);
            }
        }
        __syncthreads();
    }
    if (bad && tid == 0) atomicOr(flag, 1);
    T *A = F + fo;
    // A11^-1 and H, a front row per warp
    for (int i = wid; i < S; i += 8) {
        const double *x = M + i * ld;
        T *d = A + (long long)i * f;
        for (int c = lane; c < S; c += 32) d[c] = (T)x[c];
        for (int j = lane; j < m; j += 32) d[S + j] = (T)sparse_dot(x, ec, ev, p12[j], p12[j + 1]);
    }
    // -G and -G A12: a row of A21 has few entries, the same for the whole warp
    if (wid >= gwarps) return;
    double *gr = grow + (size_t)wid * maxrows;
    for (int i = wid; i < m; i += gwarps) {
        T *d = A + (long long)(S + i) * f;
        const long long e0 = L.ptr21[u0 + i], e1 = L.ptr21[u0 + i + 1];
        const double s = rs[L.vars[vo + S + i]];
        double v[kLeafMaxS / 32] = {};
        for (long long e = e0; e < e1; ++e) {
            const int2 x = L.list[e];
            const double a = val[x.x] * s;
#pragma unroll
            for (int u = 0; u < kLeafMaxS / 32; ++u)
                if (lane + 32 * u < S) v[u] -= a * M[x.y * ld + lane + 32 * u];
        }
#pragma unroll
        for (int u = 0; u < kLeafMaxS / 32; ++u)
            if (lane + 32 * u < S) {
                gr[lane + 32 * u] = v[u];
                d[lane + 32 * u] = (T)v[u];
            }
        __syncwarp();
        for (int j = lane; j < m; j += 32) d[S + j] = (T)sparse_dot(gr, ec, ev, p12[j], p12[j + 1]);
        __syncwarp();
    }
}

// FP64 factors rounded to FP32 (the solve of the mixed form with FP64
// factorization).
__global__ void k_round_f32(const double *__restrict__ a, float *__restrict__ b, long long n)
{
    V2D_GRID_STRIDE(i, n) { b[i] = (float)a[i]; }
}

}  // namespace
}  // namespace v2d
