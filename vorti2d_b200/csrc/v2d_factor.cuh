// Numeric phase of the multifrontal factorization (v2d_mf.cu): batched dense
// kernels over the fronts of one tree level.
//
// Each front (S pivots of f variables, row-major f x f) is eliminated by
// blocked Gauss-Jordan steps of kPiv pivots.  A step on the pivots K = [k, e)
// of a front A does, in place,
//   X = A_KK^-1                          k_pivot_inverse (X replaces A_KK)
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
// Pivoting is partial over the rows of the pivot block, by implicit row
// exchanges inside X (no permutation leaves the block); the row scaling
// applied at assembly keeps the blocks well scaled, and the FP64 Krylov
// iteration around the factors absorbs the restriction.  X is computed in
// FP64 in both precisions: on a 181 x 181 Jacobian one FP32 solve then
// reduces the residual to 5e-6, against 2e-2 with an FP32 X and 9e-2 with
// FP32 LU factors and their explicit inverses (one and two GMRES iterations
// more).
#pragma once

#include "v2d_internal.cuh"

namespace v2d {
namespace {

constexpr int kPiv = 64;      // pivots per elimination step
constexpr int kTile = 64;     // output tile of the step's products
constexpr int kSlice = 32;    // inner columns per operand slice
// grids with one y index per front take at most this many fronts per launch
// (the grid's y dimension is limited to 65535)
constexpr int kMaxFrontsY = 65535;

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

// Every front's own matrix entries, row-scaled, into the zeroed fronts.
template <class T>
__global__ void k_scatter(long long n, const int *__restrict__ csr, const int *__restrict__ row,
                          const long long *__restrict__ pos, const double *__restrict__ val,
                          const double *__restrict__ rs, T *F)
{
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x)
        F[pos[e]] += (T)(val[csr[e]] * rs[row[e]]);
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

// Adds both children's contribution blocks to every front of a level: one
// warp per front row, each entry pulled from the children through the
// inverse maps (a fixed order of addition, no atomics, one pass over the
// front for both children).
constexpr int kExtendWarps = 8;

template <class T>
__global__ void __launch_bounds__(32 * kExtendWarps) k_extend_add(
    int q0, const int *__restrict__ S, const int *__restrict__ f,
    const long long *__restrict__ foff, const int *__restrict__ voff,
    const int *__restrict__ child0, const int *__restrict__ child1,
    const int *__restrict__ inv0, const int *__restrict__ inv1, T *F)
{
    const int q = q0 + blockIdx.y, fq = f[q], vo = voff[q];
    const int c0 = child0[q], c1 = child1[q];
    const int *m0 = inv0 + vo, *m1 = inv1 + vo;
    const int lane = threadIdx.x & 31;
    const T *A0 = nullptr, *A1 = nullptr;
    int f0 = 0, f1 = 0;
    if (c0 >= 0) {
        f0 = f[c0];
        A0 = F + foff[c0] + (long long)S[c0] * f0 + S[c0];
    }
    if (c1 >= 0) {
        f1 = f[c1];
        A1 = F + foff[c1] + (long long)S[c1] * f1 + S[c1];
    }
    T *A = F + foff[q];
    for (int a = blockIdx.x * kExtendWarps + (threadIdx.x >> 5); a < fq;
         a += gridDim.x * kExtendWarps) {
        const int r0 = c0 >= 0 ? m0[a] : -1, r1 = c1 >= 0 ? m1[a] : -1;
        if (r0 < 0 && r1 < 0) continue;
        const T *s0 = A0 + (long long)r0 * f0, *s1 = A1 + (long long)r1 * f1;
        T *d = A + (long long)a * fq;
        for (int b = lane; b < fq; b += 32) {
            const int j0 = r0 >= 0 ? m0[b] : -1, j1 = r1 >= 0 ? m1[b] : -1;
            if (j0 < 0 && j1 < 0) continue;
            T v = d[b];
            if (j0 >= 0) v += s0[j0];
            if (j1 >= 0) v += s1[j1];
            d[b] = v;
        }
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

// X = A_KK^-1 of one step's pivot block of every front (one CTA each), in
// place, in FP64.  The block sits in shared memory as 2 x 2 blocks of 32 and
// is inverted by block Gauss-Jordan: the 32 x 32 diagonal blocks one after
// the other in the registers of the CTA's four warps (invert32), the products
// between the blocks on the FP64 tensor cores.  The chain of pivot columns
// bounds it, not its 2 kPiv^3 flops: the code is kept short and rolled, since
// straight-line code that runs once waits for its own instructions.
constexpr int kInvThreads = 128;
constexpr int kHalf = kPiv / 2;
constexpr int kLdX = kPiv + 2;   // two wavefronts per fragment read, rows 16-byte aligned
constexpr int kPanel = 4;        // columns per panel of invert32, one per warp

// 1 / x to a few units in the last place: the hardware's approximation and
// two Newton steps (x = 0 and denormals: not finite; the caller looks at x).
__device__ __forceinline__ double reciprocal(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    y = fma(y, fma(-x, y, 1.0), y);
    return fma(y, fma(-x, y, 1.0), y);
}

// In-place inverse of the 32 x 32 block at M by four warps: lane = row,
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
// barrier per column instead of per panel 1.0e4.  Returns whether a pivot
// column was zero.
__device__ __forceinline__ bool invert32(double *M, double (*col)[kPanel][kHalf], int *piv)
{
    constexpr int R = kHalf / kPanel;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double a[R];
#pragma unroll
    for (int i = 0; i < R; ++i) a[i] = M[lane * kLdX + kPanel * i + w];
    bool bad = false, used = false;
    int step = 0;
    double scale = 0.0;
#pragma unroll 1
    for (int P = 0; P < R; ++P) {
        col[P & 1][w][lane] = a[0];
        __syncthreads();
        double pan[kPanel];
#pragma unroll
        for (int t = 0; t < kPanel; ++t) pan[t] = col[P & 1][t][lane];
#pragma unroll
        for (int t = 0; t < kPanel; ++t) {
            // the high word of |a| (its last five bits given up for the lane);
            // 0 for a row already used: one row at least is free
            const unsigned hi = ((unsigned)__double2hiint(pan[t]) << 1) & ~63u;
            const unsigned best =
                __reduce_max_sync(0xffffffffu, used ? 0u : hi | 32u | (unsigned)lane);
            const double rinv = reciprocal(pan[t]);
            const int p = best & 31;
            const bool me = lane == p;
            double inv = __shfl_sync(0xffffffffu, rinv, p);
            if (best < 64u) {
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
    __syncthreads();
#pragma unroll
    for (int i = 0; i < R; ++i) M[step * kLdX + piv[kPanel * i + w]] = a[i] * scale;
    return bad;
}

template <class T>
__global__ void __launch_bounds__(kInvThreads) k_pivot_inverse(int q0, int k,
                                                               const int *__restrict__ S_,
                                                               const int *__restrict__ f_,
                                                               const long long *__restrict__ foff,
                                                               T *F, int *flag)
{
    __shared__ __align__(16) double M[kPiv * kLdX];
    __shared__ double col[2][kPanel][kHalf];
    __shared__ int piv[kHalf];
    const int q = q0 + blockIdx.x;
    const int S = S_[q], f = f_[q];
    if (S <= k) return;
    const int w = min(kPiv, S - k), tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    T *A = F + foff[q] + (long long)k * f + k;
    // padded by the identity
    const int c0 = tid & (kPiv - 1);
#pragma unroll 16
    for (int r = tid / kPiv; r < kPiv; r += kInvThreads / kPiv)
        M[r * kLdX + c0] = (r < w && c0 < w) ? (double)A[(long long)r * f + c0]
                                             : (r == c0 ? 1.0 : 0.0);
    bool bad = false;
    const int nh = w > kHalf ? 2 : 1;
#pragma unroll 1
    for (int h = 0; h < nh; ++h) {
        // the step's block X, its row O, its column C and the rest Y
        double *X = M + h * (kHalf * kLdX + kHalf), *Y = M + (1 - h) * (kHalf * kLdX + kHalf);
        double *O = M + (h ? kHalf * kLdX : kHalf), *C = M + (h ? kHalf : kHalf * kLdX);
        __syncthreads();
        bad |= invert32(X, col, piv);
        __syncthreads();
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
            __syncthreads();
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                double *d = D + (8 * wid + g) * kLdX + 8 * n + 2 * t;
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    d[u] = i == 0 ? acc[n][u] : (i == 1 ? d[u] : 0.0) - acc[n][u];
            }
            __syncthreads();
        }
    }
    if (bad && tid == 0) atomicOr(flag, 1);
#pragma unroll 16
    for (int r = tid / kPiv; r < kPiv; r += kInvThreads / kPiv)
        if (r < w && c0 < w) A[(long long)r * f + c0] = (T)M[r * kLdX + c0];
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
    __device__ __forceinline__ void mac(const Smem &s)
    {
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
        const int wr = (w >> 2) * 32, wc = (w & 3) * 16;
#pragma unroll
        for (int k = 0; k < kSlice; k += 4) {
            double a[4], b[2];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi) a[mi] = s.A[wr + 8 * mi + g][k + t];
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) b[ni] = s.B[k + t][wc + 8 * ni + g];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                for (int ni = 0; ni < 2; ++ni)
                    dmma_8x8x4(acc[mi][ni][0], acc[mi][ni][1], a[mi], b[ni]);
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
    __device__ __forceinline__ void mac(const Smem &s)
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
        t.mac(sm[0]);
        cp_async_wait<0>();
        __syncthreads();
        t.mac(sm[1]);
    } else {
        cp_async_wait<0>();
        __syncthreads();
        t.mac(sm[0]);
    }
}

template <class T> constexpr size_t tile_smem_bytes() { return 2 * sizeof(typename Tile<T>::Smem); }

// R = X A_KJ of a step, in place, 64 columns per CTA (blocks [0, nt)); blocks
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
    const int q = q0 + blockIdx.y;
    const int S = S_[q], f = f_[q];
    if (S <= k) return;
    const int w = min(kPiv, S - k), e = k + w;
    T *A = F + foff[q];
    if ((int)blockIdx.x >= nt) {
        const int r0 = ((int)blockIdx.x - nt) * kTile;
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
    const int c0 = blockIdx.x * kTile;
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
// -C_I X in the pivot columns (R_K = X in place).
template <class T>
__global__ void __launch_bounds__(256, 3) k_update(int q0, int k, int nt, int v0,
                                                   const int *__restrict__ S_,
                                                   const int *__restrict__ f_,
                                                   const long long *__restrict__ foff,
                                                   const int *__restrict__ voff, T *F, const T *C)
{
    using P2 = typename Pair<T>::type;
    extern __shared__ __align__(16) unsigned char tile_raw[];
    const int q = q0 + blockIdx.y;
    const int S = S_[q], f = f_[q];
    if (S <= k) return;
    const int w = min(kPiv, S - k), e = k + w;
    const int r0 = (blockIdx.x / nt) * kTile, c0 = (blockIdx.x % nt) * kTile;
    if (r0 >= f || c0 >= f || (r0 >= k && min(r0 + kTile, f) <= e)) return;
    T *A = F + foff[q];
    const T *Cq = C + (long long)(voff[q] - v0) * kPiv;
    typename Tile<T>::Smem *sm = reinterpret_cast<typename Tile<T>::Smem *>(tile_raw);
    Tile<T> t;
    // the old entries, negated: loaded while the operands are on their way
    t.each([&](int rr, int cc, T (&v)[2]) {
        const int r = r0 + rr, c = c0 + cc;
        v[0] = v[1] = T(0);
        if (r < f && c < f && !(c >= k && c < e)) {
            const P2 o = *reinterpret_cast<const P2 *>(A + (long long)r * f + c);
            v[0] = -o.x;
            v[1] = -o.y;
        }
    });
    tile_product<T>(t, sm, Cq + (long long)r0 * kPiv, kPiv, min(kTile, f - r0),
                    A + (long long)k * f + c0, f, min(kTile, f - c0), w);
    t.each([&](int rr, int cc, T (&v)[2]) {
        const int r = r0 + rr, c = c0 + cc;
        if (r < f && c < f && !(r >= k && r < e)) {
            P2 o;
            o.x = -v[0];
            o.y = -v[1];
            *reinterpret_cast<P2 *>(A + (long long)r * f + c) = o;
        }
    });
}

// FP64 factors rounded to FP32 (the solve of the mixed form with FP64
// factorization).
__global__ void k_round_f32(const double *__restrict__ a, float *__restrict__ b, long long n)
{
    V2D_GRID_STRIDE(i, n) { b[i] = (float)a[i]; }
}

}  // namespace
}  // namespace v2d
