// Sparse direct factorization of the Newton system on the device: a
// multifrontal LU over a nested-dissection separator tree of the O-grid.
//
// It takes the place of the direct LU (MUMPS) of the reference's replicated
// solve (vorti2d/petsc_solver.py:55-61, 97-115): pure Newton (dtau = inf)
// systems of this discretisation defeat point / line block Jacobi and
// multigrid preconditioners, so every Newton iteration factors the current
// Jacobian and uses the factors as the right preconditioner of GMRES(m) (FP32
// factors inside FP64 defect correction in the mixed-precision form; FP64
// factors in the plain form).
//
// Symbolic phase (host, once per mesh and sparsity pattern):
//  * the separator tree is geometric: the root separator is the
//    circumferential row jmax/2, which splits the O-grid into an inner and an
//    outer annulus; each annulus is opened by its two seam columns into one
//    rectangle, and rectangles are split recursively by their middle column
//    or row (never rows 1 or jmax-2, whose boundary rows reach two rows away:
//    the Thom wall row, vorti2d_core.f90:322-339, and the outflow rows,
//    :254-269, :307-321) until they hold at most `leaf` nodes.  Every
//    separator thus spans at most one row or two half-columns, which keeps
//    the dense top fronts small;
//  * fronts are numbered level by level (level = height above the leaves), so
//    the fronts of one level, their dense storage and their assembly entries
//    are contiguous and each level is processed by a fixed set of batched
//    launches;
//  * struct(front) = (struct(children) U adj(separator)) minus the subtree,
//    over the symmetrised node graph of the CSR pattern; each CSR entry goes
//    to the front of whichever of its two nodes is eliminated first.
//
// Numeric phase (device, per Newton iteration): the row-scaled CSR values are
// scattered into the zeroed fronts; then, per level bottom-up, the children's
// contribution blocks are added and the fronts are eliminated by blocked
// Gauss-Jordan steps (v2d_factor.cuh), which leave A11^-1, G = A21 A11^-1
// (negated) and H = A11^-1 A12 in place and the Schur complement for the
// parent.
//
// Solve (device): forward per level bottom-up (gather t, contribution vector
// w - G t for the parent), backward top-down (x = A11^-1 t - H x_struct,
// scatter).  Every step is a row-parallel product split over CTAs, so the
// large top fronts spread over many SMs.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <type_traits>
#include <utility>
#include <vector>

#include "v2d_factor.cuh"
#include "v2d_internal.cuh"
#include "v2d_solve.cuh"

namespace v2d {

// rows per work item of the solve on levels with few fronts
constexpr int kSolveRowsHost = 8;
// the default work-item split aims at about this many items per level
constexpr int kItemsPerLevel = 600;

// Dependency counters of the plan's order check (host only; the kernels wait for
// the values themselves), per front q: forward items of q that wrote z rows (fz),
// the children's forward items that wrote contribution rows (fin), backward items
// of q (bx), gather items (fg, bg).
inline int ctr_fz(int q, int nf) { return q; }
inline int ctr_fin(int q, int nf) { return nf + q; }
inline int ctr_bx(int q, int nf) { return 2 * nf + q; }
inline int ctr_fg(int q, int nf) { return 3 * nf + q; }
inline int ctr_bg(int q, int nf) { return 4 * nf + q; }
constexpr int kCtrPerFront = 5;

// ================================================================ symbolic
namespace {

struct TreeNode {
    std::vector<int> sep;   // node ids (pointer order K = imax*j + i)
    int kid[2] = {-1, -1};
    int parent = -1;
};

struct TreeBuilder {
    int imax, jmax, leaf;
    std::vector<TreeNode> t;  // postorder

    int add(std::vector<int> &&sep, int a, int b)
    {
        TreeNode nd;
        nd.sep = std::move(sep);
        int q = 0;
        if (a >= 0) nd.kid[q++] = a;
        if (b >= 0) nd.kid[q++] = b;
        t.push_back(std::move(nd));
        const int id = (int)t.size() - 1;
        for (int c : t[id].kid)
            if (c >= 0) t[c].parent = id;
        return id;
    }
    std::vector<int> block(int i0, int i1, int j0, int j1) const
    {
        std::vector<int> v;
        for (int j = j0; j < j1; ++j)
            for (int i = i0; i < i1; ++i) v.push_back(j * imax + i);
        return v;
    }
    int col_cut(int i0, int i1, int j0, int j1)
    {
        const int c = (i0 + i1) / 2;
        int a = rect(i0, c, j0, j1);
        int b = rect(c + 1, i1, j0, j1);
        return add(block(c, c + 1, j0, j1), a, b);
    }
    // Rectangle [i0,i1) x [j0,j1) of the non-periodic part of the ring.
    int rect(int i0, int i1, int j0, int j1)
    {
        const int w = i1 - i0, h = j1 - j0;
        if (w <= 0 || h <= 0) return -1;
        if (w * h <= leaf) return add(block(i0, i1, j0, j1), -1, -1);
        if (w >= h && w >= 3) return col_cut(i0, i1, j0, j1);
        int best = -1;
        const int mid = (j0 + j1) / 2;
        for (int r = j0 + 1; r < j1 - 1; ++r) {
            if (r == 1 || r == jmax - 2) continue;
            if (best < 0 || std::abs(r - mid) < std::abs(best - mid)) best = r;
        }
        if (best < 0) {
            if (w >= 3) return col_cut(i0, i1, j0, j1);
            return add(block(i0, i1, j0, j1), -1, -1);
        }
        int a = rect(i0, i1, j0, best);
        int b = rect(i0, i1, best + 1, j1);
        return add(block(i0, i1, best, best + 1), a, b);
    }
    // Annulus rows [j0, j1): cutting the two seam columns leaves one
    // (non-periodic) rectangle [1, imax-1) x [j0, j1).
    int annulus(int j0, int j1)
    {
        if (j1 <= j0) return -1;
        int kid = rect(1, imax - 1, j0, j1);
        std::vector<int> sep;
        for (int c : {0, imax - 1})
            for (int j = j0; j < j1; ++j) sep.push_back(j * imax + c);
        return add(std::move(sep), kid, -1);
    }
    void build()
    {
        // Ring first: the root is the circumferential row jc, which splits the
        // O-grid into an inner and an outer annulus (each keeps the wall or the
        // far-field rows and their two-row reach); every separator then spans
        // at most one row or two half-columns.  Grids with too few rows for
        // that use the seam columns plus the middle column as the root.
        int jc = jmax / 2;
        if (jc == 1 || jc == jmax - 2) ++jc;
        if (jmax >= 8 && jc >= 2 && jc <= jmax - 4) {
            int a = annulus(0, jc);
            int b = annulus(jc + 1, jmax);
            std::vector<int> root;
            for (int i = 0; i < imax; ++i) root.push_back(jc * imax + i);
            add(std::move(root), a, b);
            return;
        }
        const int mid = imax / 2;
        int a = rect(1, mid, 0, jmax);
        int b = rect(mid + 1, imax - 1, 0, jmax);
        std::vector<int> root;
        for (int c : {0, mid, imax - 1})
            for (int j = 0; j < jmax; ++j) root.push_back(j * imax + c);
        add(std::move(root), a, b);
    }
};

// Node adjacency in CSR form: node v's neighbours are nb[off[v], off[v] + len[v]).
struct NodeGraph {
    std::vector<int> off, len, nb;
    struct Range {
        const int *b, *e;
        const int *begin() const { return b; }
        const int *end() const { return e; }
    };
    Range of(int v) const { return {nb.data() + off[v], nb.data() + off[v] + len[v]}; }
};

template <class T>
int upload_vec(T **d, const std::vector<T> &h)
{
    *d = nullptr;
    const size_t bytes = std::max<size_t>(1, h.size()) * sizeof(T);
    V2D_CUDA_TRY(cudaMalloc((void **)d, bytes));
    if (!h.empty()) V2D_CUDA_TRY(cudaMemcpy(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
    return V2D_OK;
}

}  // namespace

void mf_plan_destroy(MfPlan *p)
{
    if (!p) return;
    void *ptrs[] = {p->d_S, p->d_f, p->d_voff, p->d_uoff, p->d_child0, p->d_child1, p->d_parent,
                    p->d_foff, p->d_vars, p->d_cbmap, p->d_inv0, p->d_inv1, p->d_asm_csr,
                    p->d_asm_row, p->d_asm_pos, p->d_items, p->d_leaf_off, p->d_leaf12,
                    p->d_leaf21, p->d_leaf_list};
    for (void *q : ptrs)
        if (q) cudaFree(q);
    delete p;
}

// Work items of the solve.  Forward: per level bottom-up, per front, rows
// [0, f) -- whole fronts, or chunks of the level's rows-per-item count
// (item_rows, set by default from the level's size).  Backward: per level top-down, rows
// [0, S) in the same granularity.  Waits and done counters:
//   forward item of q   waits fin[q] = all children's items with contribution
//                       rows; done: fz[q] if it has z rows, fin[parent] if
//                       it has contribution rows
//   backward item of q  waits fz[q] = all of q's forward items with z rows,
//                       and bx[parent] = all of the parent's backward items
//                       (which waited for theirs: all ancestors' x);
//                       done: bx[q]
// On levels whose rows-per-item entry is negative, a front split into
// several items gets a gather item first in each sweep:
//   forward gather of q   waits fin[q]; done: fg[q]; q's forward items wait fg[q]
//   backward gather of q  waits bx[parent] (which implies that q's own
//                         contribution rows are done); done: bg[q]; q's
//                         backward items wait fz[q] and bg[q]
// The kernels run an item's rows with a gather of their own: gather items are
// places in the order only.
// The check: every wait's counter reaches exactly its target in all, and
// only through items earlier in the order; so the items an item reads have
// all finished before it starts, and a CTA that takes items in order only
// waits for items that running CTAs hold.
static int items_build(MfPlan *P)
{
    const int nf = P->nfront, nl = P->nlevel;
    std::vector<int> &it = P->h_items;
    it.clear();
    P->lvl_fwd.assign(nl + 1, 0);
    P->lvl_bwd.assign(nl + 1, 0);
    // rows per item of each level (0: whole fronts).  The default aims at
    // about kItemsPerLevel items per level: the level's rows over that
    // count, rounded down to a power of two in [kSolveRowsHost, 256]; whole
    // fronts where no front of the level is longer than that
    if ((int)P->item_rows.size() != nl) {
        P->item_rows.assign(nl, kSolveRowsHost);
        for (int L = 0; L < nl; ++L) {
            long long rows = 0;
            for (int q = P->lvl_off[L]; q < P->lvl_off[L + 1]; ++q) rows += P->f[q];
            int R = kSolveRowsHost;
            while (R < 256 && 2LL * R * kItemsPerLevel <= rows) R *= 2;
            P->item_rows[L] = P->lvl_maxf[L] <= R ? 0 : R;
        }
    }
    // rows per item; a negative entry -R splits fronts of more than R rows
    // into R-row items after one gather item per front (kind 2 forward, kind 3
    // backward)
    auto per = [&](int L) {
        const int r = P->item_rows[L];
        return r > 0 ? r : (r < 0 ? -r : INT_MAX);
    };
    auto gath_f = [&](int L, int q) { return P->item_rows[L] < 0 && P->f[q] > per(L); };
    auto gath_b = [&](int L, int q) {
        return P->item_rows[L] < 0 && P->S[q] > per(L) && P->f[q] > P->S[q];
    };
    int cur_level = 0;
    auto push = [&](int kind, int q, int rb, int re, int flag) {
        const int v[12] = {kind, q, rb, re, -1, 0, -1, 0, -1, -1, cur_level, flag};
        it.insert(it.end(), v, v + 12);
    };
    P->lvl_fwd_g.assign(nl, 0);
    P->lvl_bwd_g.assign(nl, 0);
    for (int L = 0; L < nl; ++L) {
        P->lvl_fwd[L] = (int)it.size() / 12;
        cur_level = L;
        const int R = per(L);
        for (int q = P->lvl_off[L]; q < P->lvl_off[L + 1]; ++q)
            if (gath_f(L, q)) {
                push(2, q, 0, P->f[q], 1);
                ++P->lvl_fwd_g[L];
            }
        for (int q = P->lvl_off[L]; q < P->lvl_off[L + 1]; ++q)
            for (int rb = 0; rb < P->f[q]; rb += std::min(R, P->f[q]))
                push(0, q, rb, (int)std::min<long long>((long long)rb + R, P->f[q]),
                     gath_f(L, q) ? 1 : 0);
    }
    P->lvl_fwd[nl] = (int)it.size() / 12;
    for (int L = nl - 1; L >= 0; --L) {
        P->lvl_bwd[L + 1] = (int)it.size() / 12;
        cur_level = L;
        const int R = (int)P->item_rows_b.size() == nl && P->item_rows[L] > 0 ? P->item_rows_b[L]
                                                                              : per(L);
        for (int q = P->lvl_off[L]; q < P->lvl_off[L + 1]; ++q)
            if (gath_b(L, q)) {
                push(3, q, 0, P->S[q], 1);
                ++P->lvl_bwd_g[L];
            }
        for (int q = P->lvl_off[L]; q < P->lvl_off[L + 1]; ++q)
            for (int rb = 0; rb < P->S[q]; rb += std::min(R, P->S[q]))
                push(1, q, rb, (int)std::min<long long>((long long)rb + R, P->S[q]),
                     gath_b(L, q) ? 1 : 0);
    }
    P->lvl_bwd[0] = (int)it.size() / 12;
    const int ni = (int)it.size() / 12;
    // totals per front (row items only; a gather item counts once into its
    // own counter)
    std::vector<int> nfz(nf, 0), nfin(nf, 0), nbx(nf, 0);
    for (int k = 0; k < ni; ++k) {
        const int *v = &it[12 * k];
        const int q = v[1];
        if (v[0] == 0) {
            if (v[2] < P->S[q]) ++nfz[q];
            if (v[3] > P->S[q] && P->parent[q] >= 0) ++nfin[P->parent[q]];
        } else if (v[0] == 1) {
            ++nbx[q];
        }
    }
    for (int k = 0; k < ni; ++k) {
        int *v = &it[12 * k];
        const int q = v[1], pa = P->parent[q];
        switch (v[0]) {
        case 0:   // forward rows: the front's gather item, or the children's rows
            if (v[11]) { v[4] = ctr_fg(q, nf); v[5] = 1; }
            else if (nfin[q] > 0) { v[4] = ctr_fin(q, nf); v[5] = nfin[q]; }
            if (v[2] < P->S[q]) v[8] = ctr_fz(q, nf);
            if (v[3] > P->S[q] && pa >= 0) v[9] = ctr_fin(pa, nf);
            break;
        case 2:   // forward gather: the children's rows
            if (nfin[q] > 0) { v[4] = ctr_fin(q, nf); v[5] = nfin[q]; }
            v[8] = ctr_fg(q, nf);
            break;
        case 1:   // backward rows: the front's z, and the gather item or the parent's x
            v[4] = ctr_fz(q, nf);
            v[5] = nfz[q];
            if (v[11]) { v[6] = ctr_bg(q, nf); v[7] = 1; }
            else if (pa >= 0) { v[6] = ctr_bx(pa, nf); v[7] = nbx[pa]; }
            v[8] = ctr_bx(q, nf);
            break;
        case 3:   // backward gather: the parent's x (hence every ancestor's)
            if (pa >= 0) { v[4] = ctr_bx(pa, nf); v[5] = nbx[pa]; }
            v[8] = ctr_bg(q, nf);
            break;
        }
    }
    // the check
    const int nc = kCtrPerFront * nf;
    std::vector<int> total(nc, 0), seen(nc, 0);
    bool ok = true;
    for (int q = 0; q < nf; ++q)
        ok = ok && P->S[q] > 0 && (P->f[q] == P->S[q] || P->parent[q] >= 0);
    for (int k = 0; k < ni && ok; ++k) {
        const int *v = &it[12 * k];
        const int q = v[1], kind = v[0];
        ok = ok && kind >= 0 && kind <= 3 && q >= 0 && q < nf && v[2] >= 0 && v[3] > v[2] &&
             v[3] <= ((kind == 0 || kind == 2) ? P->f[q] : P->S[q]) && (v[11] == 0 || v[11] == 1);
        if (ok && kind >= 2)   // a gather item covers its whole front, once
            ok = v[11] == 1 && v[2] == 0 && v[3] == (kind == 2 ? P->f[q] : P->S[q]) &&
                 (kind == 2 || P->parent[q] >= 0);
        for (int d : {v[8], v[9]}) {
            ok = ok && d >= -1 && d < nc;
            if (ok && d >= 0) ++total[d];
        }
    }
    for (int k = 0; k < ni && ok; ++k) {
        const int *v = &it[12 * k];
        const int q = v[1], pa = P->parent[q];
        for (int w : {0, 1}) {
            const int c = v[4 + 2 * w], t = v[5 + 2 * w];
            if (c < 0) continue;
            ok = ok && c < nc && t > 0 && total[c] == t && seen[c] == t;
        }
        // what each kind must have waited for, from the algorithm
        if (v[0] == 0)
            ok = ok && (v[11] ? v[4] == ctr_fg(q, nf) && v[5] == 1
                              : (nfin[q] == 0 || (v[4] == ctr_fin(q, nf) && v[5] == nfin[q])));
        else if (v[0] == 2)
            ok = ok && (nfin[q] == 0 || (v[4] == ctr_fin(q, nf) && v[5] == nfin[q]));
        else if (v[0] == 1)
            ok = ok && v[4] == ctr_fz(q, nf) && v[5] == nfz[q] &&
                 (v[11] ? v[6] == ctr_bg(q, nf) && v[7] == 1
                        : (pa < 0 || (v[6] == ctr_bx(pa, nf) && v[7] == nbx[pa])));
        else
            ok = ok && v[4] == ctr_bx(pa, nf) && v[5] == nbx[pa];
        for (int d : {v[8], v[9]})
            if (d >= 0) ++seen[d];
    }
    if (!ok) {
        set_error("mf_plan: solve work items failed their order check");
        it.clear();
        return V2D_EARG;
    }
    P->nitems = ni;
    P->nctr = nc;
    return V2D_OK;
}

int mf_plan_build(int imax, int jmax, int n, const int *h_rowptr, const int *h_colind,
                  int leaf, MfPlan **out)
{
    *out = nullptr;
    const int N = imax * jmax;
    V2D_ARG_CHECK(n == 2 * N, "mf_plan: system size %d != 2 * %d nodes", n, N);
    V2D_ARG_CHECK(imax >= 5 && jmax >= 4, "mf_plan: grid %d x %d too small", imax, jmax);
    // the CSR pattern: row pointers from 0, non-decreasing; columns in [0, n)
    V2D_ARG_CHECK(h_rowptr[0] == 0, "mf_plan: indptr[0] = %d, not 0", h_rowptr[0]);
    for (int r = 0; r < n; ++r)
        V2D_ARG_CHECK(h_rowptr[r + 1] >= h_rowptr[r], "mf_plan: indptr decreases at row %d", r);
    for (int p = 0; p < h_rowptr[n]; ++p)
        V2D_ARG_CHECK(h_colind[p] >= 0 && h_colind[p] < n,
                      "mf_plan: column index %d at entry %d outside [0, %d)", h_colind[p], p, n);
    TreeBuilder tb{imax, jmax, std::max(4, leaf), {}};
    tb.build();
    const int nf = (int)tb.t.size();
    // --- symmetrised node graph (CSR): the distinct other nodes of each
    // node's two rows, then every such edge in both directions
    NodeGraph adj;
    {
        std::vector<int> foff(N + 1, 0), fwd, mark(N, -1);
        fwd.reserve((size_t)h_rowptr[n] / 2 + 16);
        for (int a = 0; a < N; ++a) {
            for (int r : {a, N + a})
                for (int p = h_rowptr[r]; p < h_rowptr[r + 1]; ++p) {
                    const int c = h_colind[p], b = c < N ? c : c - N;
                    if (b != a && mark[b] != a) {
                        mark[b] = a;
                        fwd.push_back(b);
                    }
                }
            foff[a + 1] = (int)fwd.size();
        }
        adj.off.assign(N + 1, 0);
        for (int a = 0; a < N; ++a)
            for (int p = foff[a]; p < foff[a + 1]; ++p) {
                ++adj.off[a + 1];
                ++adj.off[fwd[p] + 1];
            }
        for (int a = 0; a < N; ++a) adj.off[a + 1] += adj.off[a];
        adj.nb.resize(adj.off[N]);
        std::vector<int> fill(adj.off.begin(), adj.off.end() - 1);
        for (int a = 0; a < N; ++a)
            for (int p = foff[a]; p < foff[a + 1]; ++p) {
                adj.nb[fill[a]++] = fwd[p];
                adj.nb[fill[fwd[p]]++] = a;
            }
        adj.len.resize(N);
        for (int a = 0; a < N; ++a) {
            int *b = adj.nb.data() + adj.off[a], *e = adj.nb.data() + adj.off[a + 1];
            std::sort(b, e);
            adj.len[a] = (int)(std::unique(b, e) - b);
        }
    }
    // --- elimination order (postorder of the tree)
    std::vector<int> elim(N, -1), owner(N, -1), last_elim(nf);
    int order = 0;
    for (int q = 0; q < nf; ++q) {
        for (int v : tb.t[q].sep) {
            if (elim[v] >= 0) {
                set_error("mf_plan: node %d in two separators", v);
                return V2D_EARG;
            }
            elim[v] = order++;
            owner[v] = q;
        }
        last_elim[q] = order - 1;
    }
    if (order != N) {
        set_error("mf_plan: tree covers %d of %d nodes", order, N);
        return V2D_EARG;
    }
    // --- struct sets
    std::vector<std::vector<int>> st(nf);
    std::vector<int> stamp(N, -1);
    for (int q = 0; q < nf; ++q) {
        std::vector<int> s;
        auto take = [&](int u) {
            if (elim[u] > last_elim[q] && stamp[u] != q) {
                stamp[u] = q;
                s.push_back(u);
            }
        };
        for (int c : tb.t[q].kid)
            if (c >= 0)
                for (int u : st[c]) take(u);
        for (int v : tb.t[q].sep)
            for (int u : adj.of(v)) take(u);
        std::sort(s.begin(), s.end(), [&](int a, int b) { return elim[a] < elim[b]; });
        st[q] = std::move(s);
    }
    // a separator may couple only into its own subtree or to ancestors
    std::vector<int> first_elim(nf);
    for (int q = 0; q < nf; ++q) {
        int fe = last_elim[q] - (int)tb.t[q].sep.size() + 1;
        for (int c : tb.t[q].kid)
            if (c >= 0) fe = std::min(fe, first_elim[c]);
        first_elim[q] = fe;
    }
    for (int q = 0; q < nf; ++q)
        for (int v : tb.t[q].sep)
            for (int u : adj.of(v))
                if (elim[u] < first_elim[q]) {
                    set_error("mf_plan: node %d couples to node %d of a sibling subtree", v, u);
                    return V2D_EARG;
                }
    // every struct node must belong to an ancestor (no coupling across subtrees)
    for (int q = 0; q < nf; ++q)
        for (int u : st[q]) {
            int a = tb.t[q].parent;
            while (a >= 0 && a != owner[u]) a = tb.t[a].parent;
            if (a < 0) {
                set_error("mf_plan: node %d couples across sibling subtrees", u);
                return V2D_EARG;
            }
        }
    // --- levels and level-major numbering
    std::vector<int> height(nf, 0);
    int nlevel = 0;
    for (int q = 0; q < nf; ++q) {
        int h = 0;
        for (int c : tb.t[q].kid)
            if (c >= 0) h = std::max(h, height[c] + 1);
        height[q] = h;
        nlevel = std::max(nlevel, h + 1);
    }
    std::vector<int> newid(nf), oldid;
    for (int L = 0; L < nlevel; ++L)
        for (int q = 0; q < nf; ++q)
            if (height[q] == L) {
                newid[q] = (int)oldid.size();
                oldid.push_back(q);
            }
    MfPlan *P = new MfPlan();
    P->N = N; P->n = n; P->nfront = nf; P->nlevel = nlevel;
    P->S.resize(nf); P->f.resize(nf); P->voff.resize(nf); P->uoff.resize(nf);
    P->child0.assign(nf, -1); P->child1.assign(nf, -1); P->parent.assign(nf, -1);
    P->foff.resize(nf);
    P->lvl_off.assign(nlevel + 1, 0);
    P->lvl_abeg.assign(nlevel, 0); P->lvl_aend.assign(nlevel, 0);
    P->lvl_maxS.assign(nlevel, 0); P->lvl_maxf.assign(nlevel, 0);
    std::vector<int> vars, cbmap;
    long long ftot = 0;
    int vtot = 0, utot = 0;
    for (int id = 0; id < nf; ++id) {
        const int q = oldid[id];
        const int s = (int)tb.t[q].sep.size(), m = (int)st[q].size();
        const int S = 2 * s, f = 2 * (s + m);
        P->S[id] = S; P->f[id] = f;
        P->voff[id] = vtot; vtot += f;
        P->uoff[id] = utot; utot += f - S;
        P->foff[id] = ftot; ftot += (long long)f * f;
        const int L = height[q];
        P->lvl_off[L + 1]++;
        P->lvl_maxS[L] = std::max(P->lvl_maxS[L], S);
        P->lvl_maxf[L] = std::max(P->lvl_maxf[L], f);
        if (tb.t[q].parent >= 0) P->parent[id] = newid[tb.t[q].parent];
        if (tb.t[q].kid[0] >= 0) P->child0[id] = newid[tb.t[q].kid[0]];
        if (tb.t[q].kid[1] >= 0) P->child1[id] = newid[tb.t[q].kid[1]];
        // front-local variables: node p -> vars 2p (psi, row/col p) and 2p+1 (ome, N+p)
        for (int u : tb.t[q].sep) { vars.push_back(u); vars.push_back(N + u); }
        for (int u : st[q]) { vars.push_back(u); vars.push_back(N + u); }
        P->maxS = std::max(P->maxS, S);
        P->maxf = std::max(P->maxf, f);
    }
    for (int L = 0; L < nlevel; ++L) P->lvl_off[L + 1] += P->lvl_off[L];
    // contribution-block maps: struct var of child -> local index in parent
    cbmap.assign(utot, -1);
    std::vector<int> loc(n, -1);
    for (int id = 0; id < nf; ++id) {
        const int pa = P->parent[id];
        if (pa < 0) continue;
        for (int t = 0; t < P->f[pa]; ++t) loc[vars[P->voff[pa] + t]] = t;
        for (int t = P->S[id]; t < P->f[id]; ++t) {
            const int li = loc[vars[P->voff[id] + t]];
            if (li < 0) {
                set_error("mf_plan: struct variable of front %d missing in its parent", id);
                mf_plan_destroy(P);
                return V2D_EARG;
            }
            cbmap[P->uoff[id] + t - P->S[id]] = li;
        }
        for (int t = 0; t < P->f[pa]; ++t) loc[vars[P->voff[pa] + t]] = -1;
    }
    // assembly entries grouped by front (level-major)
    std::vector<int> cnt(nf + 1, 0), entry_front(h_rowptr[n]);
    for (int r = 0; r < n; ++r)
        for (int p = h_rowptr[r]; p < h_rowptr[r + 1]; ++p) {
            const int c = h_colind[p];
            const int a = r < N ? r : r - N, b = c < N ? c : c - N;
            const int fr = newid[elim[a] < elim[b] ? owner[a] : owner[b]];
            entry_front[p] = fr;
            cnt[fr + 1]++;
        }
    for (int q = 0; q < nf; ++q) cnt[q + 1] += cnt[q];
    const long long nnz = h_rowptr[n];
    std::vector<int> asm_csr(nnz), asm_row(nnz);
    std::vector<long long> asm_pos(nnz);
    {
        // entries of each front in row order (a counting sort by front),
        // then each front's local positions from its variables' lookup
        std::vector<int> fill(cnt.begin(), cnt.end() - 1);
        for (int r = 0; r < n; ++r)
            for (int p = h_rowptr[r]; p < h_rowptr[r + 1]; ++p) {
                const int o = fill[entry_front[p]]++;
                asm_csr[o] = p;
                asm_row[o] = r;
            }
        for (int id = 0; id < nf; ++id) {
            const int f = P->f[id];
            for (int t = 0; t < f; ++t) loc[vars[P->voff[id] + t]] = t;
            for (int o = cnt[id]; o < cnt[id + 1]; ++o) {
                const int r = asm_row[o], c = h_colind[asm_csr[o]];
                const int lr = loc[r], lc = loc[c];
                if (lr < 0 || lc < 0) {
                    set_error("mf_plan: entry (%d, %d) outside its front", r, c);
                    mf_plan_destroy(P);
                    return V2D_EARG;
                }
                asm_pos[o] = P->foff[id] + (long long)lr * f + lc;
            }
            for (int t = 0; t < f; ++t) loc[vars[P->voff[id] + t]] = -1;
        }
    }
    for (int L = 0; L < nlevel; ++L) {
        P->lvl_abeg[L] = cnt[P->lvl_off[L]];
        P->lvl_aend[L] = cnt[P->lvl_off[L + 1]];
    }
    P->ftotal = ftot; P->vtotal = vtot; P->utotal = utot; P->nasm = nnz;
    double fl = 0.0;
    for (int id = 0; id < nf; ++id) {
        fl += 2.0 * P->S[id] * (double)P->f[id] * P->f[id];
        P->factor_flops += front_flops(P->S[id], P->f[id]);
        P->apply_entries += (long long)P->S[id] * (2LL * P->f[id] - P->S[id]);
    }
    P->flops = fl;
    // every index the kernels dereference stays inside its buffer
    bool ok = (long long)vars.size() == vtot && (long long)cbmap.size() == utot;
    for (int v : vars) ok = ok && v >= 0 && v < n;
    for (int id = 0; id < nf && ok; ++id) {
        ok = ok && P->S[id] > 0 && P->S[id] <= P->f[id] && P->S[id] % 2 == 0;
        const int pa = P->parent[id];
        if (pa >= 0)
            for (int t = 0; t < P->f[id] - P->S[id]; ++t) {
                const int li = cbmap[P->uoff[id] + t];
                ok = ok && li >= 0 && li < P->f[pa];
            }
        else
            ok = ok && P->f[id] == P->S[id];   // the root has no contribution block
        for (int c : {P->child0[id], P->child1[id]}) ok = ok && (c < 0 || (c < id && P->parent[c] == id));
    }
    for (long long e = 0; e < nnz && ok; ++e)
        ok = asm_pos[e] >= 0 && asm_pos[e] < ftot && asm_csr[e] >= 0 && asm_csr[e] < nnz &&
             asm_row[e] >= 0 && asm_row[e] < n;
    if (!ok) {
        set_error("mf_plan: internal index check failed (%d x %d grid)", imax, jmax);
        mf_plan_destroy(P);
        return V2D_EARG;
    }
    P->h_vars = std::move(vars);
    P->h_cbmap = std::move(cbmap);
    P->h_asm_csr = std::move(asm_csr);
    P->h_asm_row = std::move(asm_row);
    P->h_asm_pos = std::move(asm_pos);
    if (items_build(P) != V2D_OK) {
        mf_plan_destroy(P);
        return V2D_EARG;
    }
    *out = P;
    return V2D_OK;
}

// The work items with their fronts' scalars, as the kernels read them.
static std::vector<SolveItemDev> device_items(const MfPlan *P)
{
    std::vector<SolveItemDev> out(P->nitems);
    for (int k = 0; k < P->nitems; ++k) {
        const int *v = &P->h_items[12 * (size_t)k], q = v[1];
        auto cu = [&](int c) { return c >= 0 ? P->uoff[c] : -1; };
        out[k] = SolveItemDev{v[0], v[2], v[3], P->S[q], P->f[q], P->voff[q], P->uoff[q],
                              cu(P->child0[q]), P->foff[q], cu(P->child1[q])};
    }
    return out;
}

// The inverse contribution maps (k_assemble), from the uploaded arrays.
static int invert_cbmap(MfPlan *P)
{
    const size_t bytes = std::max<size_t>(1, P->vtotal) * sizeof(int);
    for (int **d : {&P->d_inv0, &P->d_inv1}) {
        V2D_CUDA_TRY(cudaMalloc((void **)d, bytes));
        V2D_CUDA_TRY(cudaMemset(*d, 0xff, bytes));
    }
    k_invert_cbmap<<<std::min(P->nfront, 32 * kSMs), 128>>>(
        P->nfront, P->d_S, P->d_f, P->d_voff, P->d_uoff, P->d_parent, P->d_child0, P->d_cbmap,
        P->d_inv0, P->d_inv1);
    V2D_CUDA_TRY(cudaGetLastError());
    V2D_CUDA_TRY(cudaStreamSynchronize(0));
    return V2D_OK;
}

// The leaves' entry lists (k_leaf_lists) from the uploaded arrays; leaf_smem
// stays 0, and the leaves are eliminated like other fronts, when one of them is
// too wide or has too many entries for the leaf kernel.
static int leaf_setup(MfPlan *P)
{
    const int nq = P->lvl_off[1], maxS = P->lvl_maxS[0];
    if (maxS > kLeafMaxS) return V2D_OK;
    const long long ne = P->lvl_aend[0];
    std::vector<long long> off(nq + 1, 0);
    int q = 0;
    for (long long e = 0; e < ne; ++e) {
        while (q + 1 < nq && P->h_asm_pos[e] >= P->foff[q + 1]) off[++q] = e;
    }
    while (q < nq) off[++q] = ne;
    const size_t np = (size_t)(nq < P->nfront ? P->uoff[nq] : P->utotal) + nq + 1;
    int *stat = nullptr, h[2] = {0, 0};
    V2D_TRY(upload_vec(&P->d_leaf_off, off));
    V2D_CUDA_TRY(cudaMalloc((void **)&P->d_leaf12, np * sizeof(long long)));
    V2D_CUDA_TRY(cudaMalloc((void **)&P->d_leaf21, np * sizeof(long long)));
    V2D_CUDA_TRY(cudaMalloc((void **)&P->d_leaf_list, std::max<size_t>(1, ne) * sizeof(int2)));
    V2D_CUDA_TRY(cudaMalloc((void **)&stat, sizeof(h)));
    cudaError_t e = cudaMemset(stat, 0, sizeof(h));
    if (e == cudaSuccess) {
        k_leaf_lists<<<nq, 256>>>(P->d_S, P->d_f, P->d_foff, P->d_uoff, P->d_leaf_off, P->d_asm_csr,
                                  P->d_asm_pos, P->d_leaf_list, P->d_leaf12, P->d_leaf21, stat);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(h, stat, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(stat);
    V2D_CUDA_TRY(e);
    // eight warps for the G rows, or fewer if then two CTAs fit on an SM
    constexpr size_t kPair = 228 * 1024 / 2 - 1024 - 2304;   // a CTA's half, less its static arrays
    int gw = 8;
    while (gw > 4 && leaf_smem(maxS, P->lvl_maxf[0], h[0], gw) > kPair) --gw;
    if (leaf_smem(maxS, P->lvl_maxf[0], h[0], gw) > kPair) gw = 8;
    const size_t bytes = leaf_smem(maxS, P->lvl_maxf[0], h[0], gw);
    if (h[1] == 0 && bytes <= 220 * 1024) {
        P->leaf_entries = h[0];
        P->leaf_warps = gw;
        P->leaf_smem = bytes;
    }
    return V2D_OK;
}

// The split a device solve starts with: about kItemsDevice items per level --
// one round of the dataflow solve's CTAs -- of 16 to 256 rows, and whole fronts
// where they are short and many.  Half the items of the plan's own default:
// an item's cost is its gather and its hand-over rather than its rows (181 x
// 181, FP32: 0.113 ms with this split, 0.138 ms with the plan's).  From 1024
// columns on the rows are the larger part: 8 rows at least, twice the forward
// items (half of them only hand z on).  Backward items are counted by the
// level's pivots, not its variables: with the forward items' rows a level of
// four fronts of 2048 kept 64 of 296 CTAs busy (FP64: 513 x 513 0.66 ms so,
// 0.58 with the backward count, 0.54 with both; 1025 x 1025 2.45, 2.01, 1.95).
static void device_item_rows(MfPlan *P)
{
    constexpr int kItemsDevice = 300, kWholeFronts = 64, kWholeMaxF = 256, kLongRows = 1024;
    P->item_rows.assign(P->nlevel, 0);
    P->item_rows_b.assign(P->nlevel, 0);
    for (int L = 0; L < P->nlevel; ++L) {
        const int nq = P->lvl_off[L + 1] - P->lvl_off[L], maxf = P->lvl_maxf[L];
        const bool wide = maxf >= kLongRows;
        long long rows = 0, pivots = 0;
        for (int q = P->lvl_off[L]; q < P->lvl_off[L + 1]; ++q) {
            rows += P->f[q];
            pivots += P->S[q];
        }
        int R = wide ? 8 : 16, Rb = R;
        while (R < 256 && (wide ? 4LL : 2LL) * R * kItemsDevice <= rows) R *= 2;
        while (Rb < R && 2LL * Rb * kItemsDevice <= pivots) Rb *= 2;
        const bool whole = maxf <= R || (nq >= kWholeFronts && maxf <= kWholeMaxF);
        P->item_rows[L] = whole ? 0 : R;
        P->item_rows_b[L] = Rb;
    }
}

// Device copies of a host plan's arrays; the host copies of the large index
// arrays are released.  On failure the plan is destroyed.
static int mf_plan_upload(MfPlan *P)
{
    device_item_rows(P);
    int st_up = items_build(P);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_S, P->S);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_f, P->f);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_voff, P->voff);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_uoff, P->uoff);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_child0, P->child0);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_child1, P->child1);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_parent, P->parent);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_foff, P->foff);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_vars, P->h_vars);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_cbmap, P->h_cbmap);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_asm_csr, P->h_asm_csr);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_asm_row, P->h_asm_row);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_asm_pos, P->h_asm_pos);
    if (st_up == V2D_OK) st_up = upload_vec(&P->d_items, device_items(P));
    if (st_up == V2D_OK) st_up = invert_cbmap(P);
    if (st_up == V2D_OK) st_up = leaf_setup(P);
    if (st_up != V2D_OK) {
        mf_plan_destroy(P);
        return st_up;
    }
    // host copies are not needed once uploaded
    std::vector<int>().swap(P->h_vars);
    std::vector<int>().swap(P->h_cbmap);
    std::vector<int>().swap(P->h_asm_csr);
    std::vector<int>().swap(P->h_asm_row);
    std::vector<long long>().swap(P->h_asm_pos);
    return V2D_OK;
}

int mf_plan_create(int imax, int jmax, int n, const int *h_rowptr, const int *h_colind,
                   int leaf, MfPlan **out)
{
    *out = nullptr;
    MfPlan *P = nullptr;
    V2D_TRY(mf_plan_build(imax, jmax, n, h_rowptr, h_colind, leaf, &P));
    V2D_TRY(mf_plan_upload(P));
    *out = P;
    return V2D_OK;
}

// New work-item granularity for the solve: rows[L] rows per item on level L
// (0: whole fronts; R > 0: R rows; R < 0: -R rows).  A level at its default
// count keeps the default's backward rows, whatever the others are set to; on
// another level the count holds for both sweeps.  Rebuilds and
// re-uploads the item table (its order is checked again); the device pointer
// changes, so solves captured in graphs before must be captured again
// (items_ver counts the tables).
int mf_plan_set_item_rows(MfPlan *P, const int *rows, int nlevels)
{
    V2D_ARG_CHECK(rows && nlevels == P->nlevel, "lu item rows: %d levels given, the plan has %d",
                  nlevels, P->nlevel);
    for (int L = 0; L < nlevels; ++L)
        V2D_ARG_CHECK(rows[L] >= -4096 && rows[L] <= 4096, "lu item rows: level %d: %d", L,
                      rows[L]);
    const std::vector<int> keep = P->item_rows, keep_b = P->item_rows_b;
    device_item_rows(P);
    for (int L = 0; L < nlevels; ++L)
        if (rows[L] != P->item_rows[L]) P->item_rows[L] = P->item_rows_b[L] = rows[L];
    if (items_build(P) != V2D_OK) {
        P->item_rows = keep;
        P->item_rows_b = keep_b;
        items_build(P);
        return V2D_EARG;
    }
    SolveItemDev *d = nullptr;
    V2D_TRY(upload_vec(&d, device_items(P)));
    if (P->d_items) cudaFree(P->d_items);
    P->d_items = d;
    ++P->items_ver;
    return V2D_OK;
}

// One plan for a block-diagonal system of several O-grid systems: the union
// of their front trees (a forest), fronts renumbered level by level across
// the parts, each part's variables, CSR entries and factor positions shifted
// by its offsets.  The factorization and the solve then treat every part in
// the same launches.  parts are host plans (mf_plan_build); row_off[k] and
// nnz_off[k] place part k's rows and CSR entries in the combined system of
// n rows.
int mf_plan_forest(const std::vector<MfPlan *> &parts, const std::vector<int> &row_off,
                   const std::vector<long long> &nnz_off, int n, MfPlan **out)
{
    *out = nullptr;
    const int np = (int)parts.size();
    V2D_ARG_CHECK(np > 0 && (int)row_off.size() == np && (int)nnz_off.size() == np,
                  "mf_plan_forest: %d parts, %zu row offsets, %zu entry offsets", np,
                  row_off.size(), nnz_off.size());
    int nl = 0;
    for (const MfPlan *Q : parts) {
        V2D_ARG_CHECK(Q && !Q->h_vars.empty(), "mf_plan_forest: a part without host arrays");
        nl = std::max(nl, Q->nlevel);
    }
    MfPlan *P = new MfPlan();
    P->n = n;
    P->nlevel = nl;
    // new front ids: level-major, parts in order within a level
    std::vector<std::vector<int>> nid(np);
    int nf = 0;
    P->lvl_off.assign(nl + 1, 0);
    for (int L = 0; L < nl; ++L) {
        P->lvl_off[L] = nf;
        for (int k = 0; k < np; ++k) {
            const MfPlan *Q = parts[k];
            if (nid[k].empty()) nid[k].assign(Q->nfront, -1);
            if (L >= Q->nlevel) continue;
            for (int q = Q->lvl_off[L]; q < Q->lvl_off[L + 1]; ++q) nid[k][q] = nf++;
        }
    }
    P->lvl_off[nl] = nf;
    P->nfront = nf;
    P->S.assign(nf, 0); P->f.assign(nf, 0); P->voff.assign(nf, 0); P->uoff.assign(nf, 0);
    P->child0.assign(nf, -1); P->child1.assign(nf, -1); P->parent.assign(nf, -1);
    P->foff.assign(nf, 0);
    std::vector<int> part_of(nf), old_of(nf);
    for (int k = 0; k < np; ++k)
        for (int q = 0; q < parts[k]->nfront; ++q) {
            part_of[nid[k][q]] = k;
            old_of[nid[k][q]] = q;
        }
    long long ftot = 0;
    int vtot = 0, utot = 0;
    for (int id = 0; id < nf; ++id) {
        const MfPlan *Q = parts[part_of[id]];
        const int q = old_of[id], k = part_of[id];
        P->S[id] = Q->S[q];
        P->f[id] = Q->f[q];
        P->voff[id] = vtot; vtot += Q->f[q];
        P->uoff[id] = utot; utot += Q->f[q] - Q->S[q];
        P->foff[id] = ftot; ftot += (long long)Q->f[q] * Q->f[q];
        if (Q->child0[q] >= 0) P->child0[id] = nid[k][Q->child0[q]];
        if (Q->child1[q] >= 0) P->child1[id] = nid[k][Q->child1[q]];
        if (Q->parent[q] >= 0) P->parent[id] = nid[k][Q->parent[q]];
        P->maxS = std::max(P->maxS, Q->S[q]);
        P->maxf = std::max(P->maxf, Q->f[q]);
        P->flops += 2.0 * Q->S[q] * (double)Q->f[q] * Q->f[q];
        P->factor_flops += front_flops(Q->S[q], Q->f[q]);
        P->apply_entries += (long long)Q->S[q] * (2LL * Q->f[q] - Q->S[q]);
    }
    P->ftotal = ftot; P->vtotal = vtot; P->utotal = utot;
    P->lvl_maxS.assign(nl, 0); P->lvl_maxf.assign(nl, 0);
    P->lvl_abeg.assign(nl, 0); P->lvl_aend.assign(nl, 0);
    for (int L = 0; L < nl; ++L) {
        const int a = P->lvl_off[L], b = P->lvl_off[L + 1];
        for (int id = a; id < b; ++id) {
            P->lvl_maxS[L] = std::max(P->lvl_maxS[L], P->S[id]);
            P->lvl_maxf[L] = std::max(P->lvl_maxf[L], P->f[id]);
        }
    }
    // front variables (shifted rows) and contribution maps (front-local)
    P->h_vars.resize(vtot);
    P->h_cbmap.resize(utot);
    for (int id = 0; id < nf; ++id) {
        const MfPlan *Q = parts[part_of[id]];
        const int q = old_of[id], ro = row_off[part_of[id]];
        for (int t = 0; t < Q->f[q]; ++t) P->h_vars[P->voff[id] + t] = Q->h_vars[Q->voff[q] + t] + ro;
        for (int t = 0; t < Q->f[q] - Q->S[q]; ++t)
            P->h_cbmap[P->uoff[id] + t] = Q->h_cbmap[Q->uoff[q] + t];
    }
    // assembly entries, level by level: each part's entries of the level with
    // shifted CSR entry, row and factor position (the front of an entry is
    // the one whose storage holds its position)
    long long nasm = 0;
    for (const MfPlan *Q : parts) nasm += Q->nasm;
    P->nasm = nasm;
    P->h_asm_csr.resize(nasm);
    P->h_asm_row.resize(nasm);
    P->h_asm_pos.resize(nasm);
    long long o = 0;
    for (int L = 0; L < nl; ++L) {
        P->lvl_abeg[L] = o;
        for (int k = 0; k < np; ++k) {
            const MfPlan *Q = parts[k];
            if (L >= Q->nlevel) continue;
            int q = Q->lvl_off[L];
            for (long long e = Q->lvl_abeg[L]; e < Q->lvl_aend[L]; ++e, ++o) {
                const long long pos = Q->h_asm_pos[e];
                while (q + 1 < Q->lvl_off[L + 1] && pos >= Q->foff[q + 1]) ++q;
                if (pos < Q->foff[q] || pos >= Q->foff[q] + (long long)Q->f[q] * Q->f[q]) {
                    set_error("mf_plan_forest: assembly entry outside its level's fronts");
                    mf_plan_destroy(P);
                    return V2D_EARG;
                }
                P->h_asm_csr[o] = (int)(Q->h_asm_csr[e] + nnz_off[k]);
                P->h_asm_row[o] = Q->h_asm_row[e] + row_off[k];
                P->h_asm_pos[o] = P->foff[nid[k][q]] + (pos - Q->foff[q]);
            }
        }
        P->lvl_aend[L] = o;
    }
    bool ok = o == nasm;
    for (int v : P->h_vars) ok = ok && v >= 0 && v < n;
    for (long long e = 0; e < nasm && ok; ++e)
        ok = P->h_asm_pos[e] >= 0 && P->h_asm_pos[e] < ftot && P->h_asm_row[e] >= 0 &&
             P->h_asm_row[e] < n && P->h_asm_csr[e] >= 0;
    if (!ok) {
        set_error("mf_plan_forest: index check failed");
        mf_plan_destroy(P);
        return V2D_EARG;
    }
    if (items_build(P) != V2D_OK) {
        mf_plan_destroy(P);
        return V2D_EARG;
    }
    V2D_TRY(mf_plan_upload(P));
    *out = P;
    return V2D_OK;
}

}  // namespace v2d

// Planning aid (no reference counterpart): runs only the host symbolic phase.
extern "C" int v2d_lu_plan_info(int imax, int jmax, const int *indptr, const int *indices,
                                int leaf, long long *out8)
{
    using namespace v2d;
    V2D_ARG_CHECK(indptr && indices && out8, "lu_plan_info: null pointer");
    MfPlan *P = nullptr;
    V2D_TRY(mf_plan_build(imax, jmax, 2 * imax * jmax, indptr, indices, leaf, &P));
    out8[0] = P->nfront;
    out8[1] = P->nlevel;
    out8[2] = P->maxS;
    out8[3] = P->maxf;
    out8[4] = P->ftotal;
    out8[5] = (long long)P->flops;
    out8[6] = P->vtotal;
    out8[7] = P->utotal;
    mf_plan_destroy(P);
    return V2D_OK;
}

extern "C" int v2d_lu_reciprocals(int n, const double *x, double *y)
{
    using namespace v2d;
    V2D_ARG_CHECK(n > 0, "lu_reciprocals: n = %d", n);
    V2D_ARG_CHECK(x && y, "lu_reciprocals: null pointer");
    DevBuf<double> d;
    V2D_TRY(d.alloc(2 * (size_t)n, 0));
    V2D_CUDA_TRY(cudaMemcpyAsync(d.p, x, n * sizeof(double), cudaMemcpyHostToDevice, 0));
    k_reciprocal<<<grid_for(n, 256), 256>>>(n, d.p, d.p + n);
    V2D_CUDA_TRY(cudaGetLastError());
    count_launches(1);
    V2D_CUDA_TRY(cudaMemcpyAsync(y, d.p + n, n * sizeof(double), cudaMemcpyDeviceToHost, 0));
    V2D_CUDA_TRY(cudaStreamSynchronize(0));
    return V2D_OK;
}

// Planning aid for the solve's work items (host only): info4 = {work items,
// counters, fronts, levels}; when cap_items >= items, items gets 12 ints per
// item (kind 0 forward / 1 backward, front, first row, end row, wait counter
// and target, second wait counter and target, two done counters, 0, 0; -1
// for none); when cap_fronts >= fronts, fronts3 gets S, f and the parent of
// each front.
extern "C" int v2d_lu_solve_plan(int imax, int jmax, const int *indptr, const int *indices,
                                 int leaf, int *info4, int *items, int cap_items, int *fronts3,
                                 int cap_fronts)
{
    return v2d_lu_solve_plan_split(imax, jmax, indptr, indices, leaf, nullptr, 0, info4, items,
                                   cap_items, fronts3, cap_fronts);
}

extern "C" int v2d_lu_solve_plan_split(int imax, int jmax, const int *indptr, const int *indices,
                                       int leaf, const int *rows, int nrows, int *info4,
                                       int *items, int cap_items, int *fronts3, int cap_fronts)
{
    using namespace v2d;
    V2D_ARG_CHECK(indptr && indices && info4, "lu_solve_plan: null pointer");
    MfPlan *P = nullptr;
    V2D_TRY(mf_plan_build(imax, jmax, 2 * imax * jmax, indptr, indices, leaf, &P));
    if (rows) {
        if (nrows != P->nlevel) {
            set_error("lu_solve_plan: %d rows-per-item entries, the plan has %d levels", nrows,
                      P->nlevel);
            mf_plan_destroy(P);
            return V2D_EARG;
        }
        P->item_rows.assign(rows, rows + nrows);
        const int st = items_build(P);
        if (st != V2D_OK) {
            mf_plan_destroy(P);
            return st;
        }
    }
    info4[0] = P->nitems;
    info4[1] = P->nctr;
    info4[2] = P->nfront;
    info4[3] = P->nlevel;
    if (items && cap_items >= P->nitems) std::copy(P->h_items.begin(), P->h_items.end(), items);
    if (fronts3 && cap_fronts >= P->nfront)
        for (int q = 0; q < P->nfront; ++q) {
            fronts3[3 * q] = P->S[q];
            fronts3[3 * q + 1] = P->f[q];
            fronts3[3 * q + 2] = P->parent[q];
        }
    mf_plan_destroy(P);
    return V2D_OK;
}

namespace v2d {

// ================================================================ numeric
namespace {

// ---------------------------------------------------------- transposed solve
// The transposed solve is the adjoint of the solve's steps taken in reverse
// order.  Bottom-up (adjoint of the backward sweep): the front gathers g on
// its fully summed variables plus its children's contributions (the same
// contribution-block maps as the forward sweep), forms ybar = A11^-T acc_FS
// (kept in zbuf) and passes acc_CB - H^T acc_FS up.  Top-down (adjoint of the
// forward sweep): the front takes its parent's adjoint right-hand side
// upd_bar on its contribution rows, t = ybar - G^T upd_bar, and writes
// lambda = rs .* t on its fully summed variables.  One CTA per front; the
// transposed products read the factor rows column-wise (one thread per
// column, coalesced across the warp).
template <class T>
__global__ void __launch_bounds__(kSolveThreads) k_tup_front(int q0, const MfDev D, const T *F,
                                                              const T *g, T *zbuf, T *upd)
{
    extern __shared__ unsigned char smem_raw[];
    T *acc = reinterpret_cast<T *>(smem_raw);   // f
    T *yb = acc + D.maxf;                         // S
    const int q = q0 + blockIdx.x;
    const int S = D.S[q], f = D.f[q], vo = D.voff[q], m = f - S;
    const T *A = F + D.foff[q];
    const int *vars = D.vars + vo;
    const int tid = threadIdx.x;
    for (int p = tid; p < f; p += blockDim.x) acc[p] = p < S ? g[vars[p]] : T(0);
    __syncthreads();
    for (int slot = 0; slot < 2; ++slot) {
        const int c = slot == 0 ? D.child0[q] : D.child1[q];
        if (c >= 0) {
            const int mc = D.f[c] - D.S[c];
            const int *map = D.cbmap + D.uoff[c];
            const T *u = upd + D.uoff[c];
            for (int e = tid; e < mc; e += blockDim.x) acc[map[e]] += u[e];
        }
        __syncthreads();
    }
    for (int j = tid; j < S; j += blockDim.x) {     // ybar = A11^-T acc_FS
        T v = T(0);
        for (int i = 0; i < S; ++i) v += A[(long long)i * f + j] * acc[i];
        yb[j] = v;
    }
    __syncthreads();
    for (int j = tid; j < S; j += blockDim.x) zbuf[vo + j] = yb[j];
    T *uo = upd + D.uoff[q];
    for (int k = tid; k < m; k += blockDim.x) {     // acc_CB - H^T acc_FS
        T v = T(0);
        for (int i = 0; i < S; ++i) v += A[(long long)i * f + S + k] * acc[i];
        uo[k] = acc[S + k] - v;
    }
}

template <class T>
__global__ void __launch_bounds__(kSolveThreads) k_tdown_front(int q0, const MfDev D, const T *F,
                                                               const double *__restrict__ rs,
                                                               const T *zbuf, T *wb, T *lam)
{
    extern __shared__ unsigned char smem_raw[];
    T *wbar = reinterpret_cast<T *>(smem_raw);  // f
    const int q = q0 + blockIdx.x;
    const int S = D.S[q], f = D.f[q], vo = D.voff[q], m = f - S;
    const T *A = F + D.foff[q];
    const int *vars = D.vars + vo;
    const int tid = threadIdx.x;
    const int pa = D.parent[q];
    for (int k = tid; k < m; k += blockDim.x) {     // upd_bar from the parent
        const T u = pa >= 0 ? wb[D.voff[pa] + D.cbmap[D.uoff[q] + k]] : T(0);
        wbar[S + k] = u;
    }
    __syncthreads();
    // t = ybar - G^T upd_bar: column i of the stored -G
    for (int i = tid; i < S; i += blockDim.x) {
        T t = zbuf[vo + i];
        for (int j = S; j < f; ++j) t += A[(long long)j * f + i] * wbar[j];
        wbar[i] = t;
    }
    __syncthreads();
    for (int p = tid; p < f; p += blockDim.x) wb[vo + p] = wbar[p];
    for (int p = tid; p < S; p += blockDim.x) lam[vars[p]] = (T)(rs[vars[p]] * (double)wbar[p]);
}

}  // namespace

// ------------------------------------------------------------ host drivers
// Shared memory of the transposed solve's launches, es bytes per entry: an f
// and an S vector going up, an f vector going down.
static size_t tup_smem(const MfPlan *P, size_t es) { return ((size_t)P->maxf + P->maxS) * es; }
static size_t tdown_smem(const MfPlan *P, size_t es) { return (size_t)P->maxf * es; }

// The dynamic shared memory limit of a kernel (cudaFuncSetAttribute) holds
// per function and device for the whole process, so every handle shares it:
// it is only ever raised, to the largest size any handle launches with.
// Setting it to one handle's smaller size would make the launches of a
// handle with larger fronts fail.  Until it is set, a launch may use the
// default 48 KB less the kernel's static shared memory.
static cudaError_t raise_dyn_smem(const void *fn, size_t bytes)
{
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, size_t> limit;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, fn);
    if (e != cudaSuccess) return e;
    const size_t room = fa.sharedSizeBytes < 48 * 1024 ? 48 * 1024 - fa.sharedSizeBytes : 0;
    std::lock_guard<std::mutex> lock(mu);
    size_t &cur = limit[{fn, dev}];
    if (bytes <= std::max(cur, room)) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) cur = bytes;
    return e;
}

// The split form's lower-level launches: threads that compute an item and
// resident CTAs per SM.
constexpr int kLowThreads = 128;
constexpr int kLowMinBlocks = 4;

// Shared memory of a dataflow launch whose largest front has maxf variables
// (es bytes each), `want` CTAs per SM at most: the vector, then kStages chunks
// of what is left of the SM's share.  A chunk below kMinChunk holds too few
// rows to stage (each CTA then takes a larger share, or reads its rows from
// global memory).
static FlowShape flow_shape(int maxf, size_t es, int want)
{
    constexpr int kMinChunk = 8192;
    FlowShape sh;
    sh.vbytes = (int)(((size_t)maxf * es + 127) / 128 * 128);
    for (int d = want; d >= 1; --d) {
        const int share = std::min(227 * 1024, 228 * 1024 / d - 1024) - (int)sizeof(FlowShared) - 256;
        sh.cbytes = std::max(0, (share - sh.vbytes) / kStages) / 128 * 128;
        if (sh.cbytes >= kMinChunk) break;
    }
    if (sh.cbytes < 1024) sh.cbytes = 0;
    sh.smem = (size_t)sh.vbytes + (size_t)kStages * sh.cbytes;
    return sh;
}

// The kernel of a form (0, 1; 2: the split form's lower levels) of the
// dataflow solve.
template <class T> static const void *flow_kernel(int form)
{
    return form == 0 ? (const void *)k_solve_flow<T, 2>
                     : form == 1 ? (const void *)k_solve_flow<T, 3>
                                 : (const void *)k_solve_flow<T, kLowMinBlocks, kLowThreads>;
}

// Sizes one form's launches for fronts of up to maxf variables; per_sm CTAs
// at most.
static int flow_setup(const MfFactor *M, int form, int maxf, int per_sm, FlowShape *out)
{
    const size_t es = M->fp32 ? sizeof(float) : sizeof(double);
    const void *fn = M->fp32 ? flow_kernel<float>(form) : flow_kernel<double>(form);
    FlowShape sh = flow_shape(maxf, es, per_sm);
    V2D_CUDA_TRY(raise_dyn_smem(fn, sh.smem));
    int dev = 0, nsm = 0, occ = 0;
    V2D_CUDA_TRY(cudaGetDevice(&dev));
    V2D_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    V2D_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &occ, fn, 32 + (form == 2 ? kLowThreads : kSolveThreads), sh.smem));
    sh.grid = nsm * std::min(occ, per_sm);
    *out = sh;
    return V2D_OK;
}

int mf_factor_create(const MfPlan *P, int fp32, int fact64, MfFactor **out)
{
    *out = nullptr;
    MfFactor *M = new MfFactor();
    M->fp32 = fp32;
    M->fact64 = fp32 && fact64 ? 1 : 0;
    M->limits = WaitLimits{kFlowSpins, kPipeSpins};
    const size_t es = fp32 ? sizeof(float) : sizeof(double);          // solve
    const size_t esf = fp32 && !M->fact64 ? sizeof(float) : sizeof(double);   // factorization
    cudaError_t e = cudaSuccess;
    auto grab = [&](void **p, size_t bytes) {
        if (e == cudaSuccess) e = cudaMalloc(p, std::max<size_t>(bytes, 16));
    };
    grab(&M->F, (size_t)P->ftotal * esf);
    if (M->fact64) grab(&M->F32, (size_t)P->ftotal * sizeof(float));
    // tickets, then upd, then z: one fill before each dataflow solve
    const size_t upd0 = 128, z0 = upd0 + ((size_t)P->utotal * es + 127) / 128 * 128;
    M->msg_bytes = z0 + (size_t)P->vtotal * es;
    grab(&M->msg, M->msg_bytes);
    if (e == cudaSuccess) {
        M->tickets = (int *)M->msg;
        M->upd = (char *)M->msg + upd0;
        M->z = (char *)M->msg + z0;
    }
    long long cols = 0;   // front variables of the largest level
    for (int L = 0; L < P->nlevel; ++L) {
        long long v = 0;
        for (int q = P->lvl_off[L]; q < P->lvl_off[L + 1]; ++q) v += P->f[q];
        cols = std::max(cols, v);
    }
    grab(&M->cols, (size_t)cols * kPiv * esf);
    grab(&M->wb, (size_t)P->vtotal * es);
    grab((void **)&M->rs, (size_t)P->n * sizeof(double));
    int steps = 0;   // of all levels: a tile counter for each
    for (int S : P->lvl_maxS) steps += (S + kPiv - 1) / kPiv;
    grab((void **)&M->flag, (1 + steps) * sizeof(int));
    M->steps = steps;
    grab((void **)&M->bar, sizeof(MfBarrier));
    if (e == cudaSuccess) e = cudaMemset(M->bar, 0, sizeof(MfBarrier));
    if (e != cudaSuccess) {
        set_error("mf_factor: allocation of %.1f MB failed: %s",
                  ((double)P->ftotal * (esf + (M->fact64 ? 4 : 0))) / 1e6, cudaGetErrorString(e));
        mf_factor_destroy(M);
        return V2D_ENOMEM;
    }
    // dynamic shared memory of the solve and factorization kernels (set once,
    // outside any stream capture)
    const size_t solve = (size_t)P->maxf * es;
    if (solve + P->maxS * es > 227 * 1024) {
        set_error("mf_factor: front of %d unknowns (separator %d) exceeds shared memory",
                  P->maxf, P->maxS);
        mf_factor_destroy(M);
        return V2D_EARG;
    }
    auto attr = [&](const void *fn, size_t bytes) {
        if (e == cudaSuccess) e = raise_dyn_smem(fn, bytes);
    };
    // the largest front accepted: two f vectors
    if (2 * P->maxf * es > 227 * 1024) {
        set_error("mf_factor: front of %d unknowns exceeds shared memory (transposed solve)",
                  P->maxf);
        mf_factor_destroy(M);
        return V2D_EARG;
    }
    if (fp32) {
        attr((const void *)k_solve_level<float>, solve);
        attr((const void *)k_tup_front<float>, tup_smem(P, es));
        attr((const void *)k_tdown_front<float>, tdown_smem(P, es));
    } else {
        attr((const void *)k_solve_level<double>, solve);
        attr((const void *)k_tup_front<double>, tup_smem(P, es));
        attr((const void *)k_tdown_front<double>, tdown_smem(P, es));
    }
    if (esf == sizeof(float)) {
        attr((const void *)k_leaf<float>, P->leaf_smem);
        attr((const void *)k_row_block<float>, tile_smem_bytes<float>());
        attr((const void *)k_update<float>, tile_smem_bytes<float>());
    } else {
        attr((const void *)k_leaf<double>, P->leaf_smem);
        attr((const void *)k_row_block<double>, tile_smem_bytes<double>());
        attr((const void *)k_update<double>, tile_smem_bytes<double>());
        attr((const void *)k_update_wide, sizeof(WideShared));
    }
    if (e != cudaSuccess) {
        set_error("mf_factor: %s", cudaGetErrorString(e));
        mf_factor_destroy(M);
        return V2D_ECUDA;
    }
    // dataflow solve: as many CTAs as can be resident at once, two (form 0) or
    // three (form 1) per SM
    for (int form = 0; form < 2; ++form) {
        const int st = flow_setup(M, form, P->maxf, 2 + form, &M->shape[form]);
        if (st != V2D_OK) {
            mf_factor_destroy(M);
            return st;
        }
    }
    if (M->shape[0].grid <= 0) {
        set_error("mf_factor: no CTA of the dataflow solve fits on an SM");
        mf_factor_destroy(M);
        return V2D_ECUDA;
    }
    cudaGetLastError();
    *out = M;
    return V2D_OK;
}

void mf_factor_destroy(MfFactor *M)
{
    if (!M) return;
    if (M->graph) cudaGraphExecDestroy(M->graph);
    void *ptrs[] = {M->F, M->F32, M->msg, M->cols, M->wb, M->rs, M->flag, M->bar};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    delete M;
}

MfDev mf_dev(const MfPlan *P, const MfFactor *M)
{
    MfDev D;
    D.S = P->d_S; D.f = P->d_f; D.voff = P->d_voff; D.uoff = P->d_uoff;
    D.child0 = P->d_child0; D.child1 = P->d_child1; D.parent = P->d_parent; D.foff = P->d_foff;
    D.vars = P->d_vars; D.cbmap = P->d_cbmap;
    D.inv0 = P->d_inv0; D.inv1 = P->d_inv1;
    D.maxS = P->maxS; D.maxf = P->maxf;
    return D;
}

template <class T>
static int factor_launches(const MfPlan *P, MfFactor *M, const int *rowptr, const double *val,
                           cudaStream_t s, cudaEvent_t *ev = nullptr, int *codes = nullptr,
                           int cap = 0, int *nev_out = nullptr)
{
    T *F = (T *)M->F, *C = (T *)M->cols;
    long long launches = 0;
    const size_t smem = tile_smem_bytes<T>();
    // with ev: an event is recorded after each kernel (kind * 1000 + level;
    // kinds 0 rowscale, 1 scatter, 2 assembly with the first pivot inverse,
    // 3 leaves, 4 row block, 6 update)
    int nev = 0;
    auto mark = [&](int code) -> int {
        const cudaError_t le = cudaGetLastError();
        if (le != cudaSuccess) {
            set_error("LU factor: launch of kind %d at level %d failed: %s", code / 1000,
                      code % 1000, cudaGetErrorString(le));
            return V2D_ECUDA;
        }
        if (!ev) return V2D_OK;
        if (nev >= cap) {
            set_error("LU factor timing: more than %d launches", cap);
            return V2D_EARG;
        }
        codes[nev] = code;
        V2D_CUDA_TRY(cudaEventRecord(ev[nev], s));
        ++nev;
        return V2D_OK;
    };
    int *ticket = M->flag + 1;
    V2D_CUDA_TRY(cudaMemsetAsync(ticket, 0, M->steps * sizeof(int), s));
    k_rowscale<<<grid_for(P->n, 256), 256, 0, s>>>(P->n, rowptr, val, M->rs);
    V2D_TRY(mark(0));
    ++launches;
    // the leaves by their own kernel; matrix entries into the other fronts
    const int first = P->leaf_smem > 0 ? 1 : 0;
    const long long f0 = first == 0 ? 0 : first < P->nlevel ? P->foff[P->lvl_off[1]] : P->ftotal;
    const long long e0 = first ? P->lvl_aend[0] : 0, ne = P->nasm - e0;
    if (f0 < P->ftotal)
        V2D_CUDA_TRY(cudaMemsetAsync(F + f0, 0, (size_t)(P->ftotal - f0) * sizeof(T), s));
    if (ne > 0) {
        constexpr int per_block = 256 * kScatterEntries;
        k_scatter<T><<<(int)((ne + per_block - 1) / per_block), 256, 0, s>>>(
            ne, P->d_asm_csr + e0, P->d_asm_row + e0, P->d_asm_pos + e0, val, M->rs, F);
        V2D_TRY(mark(1000));
        ++launches;
    }
    if (first) {
        const LeafMaps lm{P->d_S, P->d_f, P->d_voff, P->d_uoff, P->d_vars, P->d_asm_csr,
                          P->d_asm_row, P->d_foff, P->d_leaf_off, P->d_asm_pos, P->d_leaf12,
                          P->d_leaf21, P->d_leaf_list};
        k_leaf<T><<<P->lvl_off[1], 256, P->leaf_smem, s>>>(lm, (P->lvl_maxS[0] + 7) / 8 * 8,
                                                          P->lvl_maxf[0], P->leaf_entries, P->leaf_warps, val,
                                                          M->rs, F, M->flag);
        V2D_TRY(mark(3000));
        ++launches;
    }
    const AssemblyMaps maps{P->d_S, P->d_f, P->d_voff, P->d_child0, P->d_child1, P->d_inv0,
                            P->d_inv1, P->d_foff};
    for (int L = first; L < P->nlevel; ++L) {
        const int q0 = P->lvl_off[L], nq = P->lvl_off[L + 1] - q0;
        const int maxf = P->lvl_maxf[L], nt = (maxf + kTile - 1) / kTile, v0 = P->voff[q0];
        // the extend-add's blocks of a front: none on the leaves
        const int nc = (maxf + kExtCols - 1) / kExtCols;
        const int per =
            1 + (L > 0 ? nc * ((maxf + kExtRows * kExtWarps - 1) / (kExtRows * kExtWarps)) : 0);
        k_assemble<T><<<nq * per, 32 * kExtWarps, 0, s>>>(q0, per, nc, maps, F, M->flag);
        V2D_TRY(mark(2000 + L));
        ++launches;
        const long long tiles = (long long)nq * nt * nt;
        const int minS = *std::min_element(P->S.begin() + q0, P->S.begin() + q0 + nq);
        for (int k = 0; k < P->lvl_maxS[L]; k += kPiv) {
            k_row_block<T><<<nq * 2 * nt, 256, smem, s>>>(q0, k, nt, v0, P->d_S, P->d_f, P->d_foff,
                                                        P->d_voff, F, C);
            V2D_TRY(mark(4000 + L));
            // From four tiles per SM on the wide update's pipeline pays: at 800 tiles
            // 52 us against 55, at 2178 61 against 68, at 24000 0.53 ms against 0.64;
            // with one tile per SM the three CTAs of k_update are the faster ones
            // (15 against 19 us at 180 tiles).
            if (sizeof(T) == 8 && k + kPiv <= minS && tiles >= 4 * kSMs) {
                const int len = (int)std::max(1LL, std::min(8LL, tiles / (4 * kSMs)));
                k_update_wide<<<kSMs, 32 * kWideWarps + kWideProducers, sizeof(WideShared), s>>>(
                    q0, nq, k, nt, len, v0, P->d_S, P->d_f, P->d_foff, P->d_voff, (double *)F,
                    (const double *)C, ticket++, M->flag, M->limits.pipe, &M->bar->err);
            } else {
                k_update<T><<<nq * nt * nt, 256, smem, s>>>(q0, k, nt, v0, P->d_S, P->d_f,
                                                            P->d_foff, P->d_voff, F, C, M->flag);
            }
            V2D_TRY(mark(6000 + L));
            launches += 2;
        }
    }
    if (M->fact64) {   // FP64 factors rounded to FP32 for the solve
        k_round_f32<<<grid_for(P->ftotal, 256), 256, 0, s>>>((const double *)M->F,
                                                             (float *)M->F32, P->ftotal);
        V2D_TRY(mark(11000));
        ++launches;
    }
    V2D_CUDA_TRY(cudaGetLastError());
    if (nev_out) *nev_out = nev;
    if (!ev) M->launches_per_factor = launches;
    return V2D_OK;
}

int mf_factor(const MfPlan *P, MfFactor *M, const int *rowptr, const double *val, cudaStream_t s)
{
    if (!M->graph || M->graph_val != val || M->graph_rowptr != rowptr) {
        if (M->graph) cudaGraphExecDestroy(M->graph);
        M->graph = nullptr;
        cudaGraph_t g = nullptr;
        V2D_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        int st = M->fp32 && !M->fact64 ? factor_launches<float>(P, M, rowptr, val, s)
                                       : factor_launches<double>(P, M, rowptr, val, s);
        cudaError_t e = cudaStreamEndCapture(s, &g);
        if (st != V2D_OK) {
            if (g) cudaGraphDestroy(g);
            return st;
        }
        if (e != cudaSuccess) {
            set_error("mf_factor: graph capture failed: %s", cudaGetErrorString(e));
            return V2D_ECUDA;
        }
        e = cudaGraphInstantiate(&M->graph, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) {
            set_error("mf_factor: graph instantiate failed: %s", cudaGetErrorString(e));
            return V2D_ECUDA;
        }
        M->graph_val = val;
        M->graph_rowptr = rowptr;
    }
    V2D_CUDA_TRY(cudaMemsetAsync(M->flag, 0, sizeof(int), s));
    V2D_CUDA_TRY(cudaGraphLaunch(M->graph, s));
    count_launches(M->launches_per_factor);
    return V2D_OK;
}

// Error of the launch just issued, named (the solve is usually issued inside
// a stream capture, where a failed launch invalidates the capture and later
// calls report only that).
static int solve_launch(const char *what, int L)
{
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return V2D_OK;
    set_error("LU solve: launch of %s (level %d) failed: %s", what, L, cudaGetErrorString(e));
    return V2D_ECUDA;
}

// Launch codes of the solve's kernels for per-launch timing (kind * 1000 + level).
enum { kCodeFwdLevel = 0, kCodeBwdLevel = 1, kCodeFlow = 2 };

template <class T>
static int apply_launches(const MfPlan *P, const MfFactor *M, const T *b, T *x, const int *stop_a,
                          const int *stop_b, cudaStream_t s, long long *n_launches,
                          cudaEvent_t *ev = nullptr, int *codes = nullptr, int cap = 0,
                          unsigned long long *trace = nullptr)
{
    // with ev: an event is recorded after each launch (at most cap launches)
    int nev = 0;
    auto mark = [&](int code) -> int {
        if (!ev) return V2D_OK;
        if (nev >= cap) {
            set_error("LU solve timing: more than %d launches", cap);
            return V2D_EARG;
        }
        codes[nev] = code;
        V2D_CUDA_TRY(cudaEventRecord(ev[nev], s));
        ++nev;
        return V2D_OK;
    };
    const MfDev D = mf_dev(P, M);
    const T *F = (const T *)(M->fact64 ? M->F32 : M->F);
    T *z = (T *)M->z, *upd = (T *)M->upd;
    const SolveItemDev *items = P->d_items;
    const size_t smf = (size_t)P->maxf * sizeof(T);
    long long launches = 0;
    if (M->flow) {
        // every message unset (0xff bytes: a NaN no arithmetic gives), tickets -1
        V2D_CUDA_TRY(cudaMemsetAsync(M->msg, 0xff, M->msg_bytes, s));
        V2D_CUDA_TRY(cudaMemsetAsync(x, 0xff, (size_t)P->n * sizeof(T), s));
        const FlowShape &up = M->shape[M->flow_form], &lo = M->shape[2];
        auto upper = [&](int i0, int i1, int slot) {
            const int n = std::max(1, std::min(i1 - i0, up.grid));
            if (M->flow_form == 1)
                k_solve_flow<T, 3><<<n, kSolveThreads + 32, up.smem, s>>>(
                    D, F, b, M->rs, z, upd, x, items, i0, i1, up.vbytes, up.cbytes,
                    M->tickets, slot, M->bar, stop_a, stop_b, M->limits, trace);
            else
                k_solve_flow<T, 2><<<n, kSolveThreads + 32, up.smem, s>>>(
                    D, F, b, M->rs, z, upd, x, items, i0, i1, up.vbytes, up.cbytes,
                    M->tickets, slot, M->bar, stop_a, stop_b, M->limits, trace);
        };
        auto lower = [&](int i0, int i1, int slot) {
            k_solve_flow<T, kLowMinBlocks, kLowThreads>
                <<<std::max(1, std::min(i1 - i0, lo.grid)), kLowThreads + 32, lo.smem, s>>>(
                    D, F, b, M->rs, z, upd, x, items, i0, i1, lo.vbytes, lo.cbytes,
                    M->tickets, slot, M->bar, stop_a, stop_b, M->limits, trace);
        };
        const int Ls = M->split;
        if (Ls > 0 && Ls < P->nlevel && lo.grid > 0) {
            lower(P->lvl_fwd[0], P->lvl_fwd[Ls], 0);
            V2D_TRY(solve_launch("k_solve_flow (lower levels, forward)", 0));
            V2D_TRY(mark(kCodeFlow * 1000));
            upper(P->lvl_fwd[Ls], P->lvl_bwd[Ls], 1);
            V2D_TRY(solve_launch("k_solve_flow (upper levels)", 0));
            V2D_TRY(mark(kCodeFlow * 1000 + 1));
            lower(P->lvl_bwd[Ls], P->nitems, 2);
            V2D_TRY(solve_launch("k_solve_flow (lower levels, backward)", 0));
            V2D_TRY(mark(kCodeFlow * 1000 + 2));
            launches = 3;
        } else {
            upper(0, P->nitems, 0);
            V2D_TRY(solve_launch("k_solve_flow", 0));
            V2D_TRY(mark(kCodeFlow * 1000));
            launches = 1;
        }
    } else {
        // a level's gather items (first in its range) need no launch
        for (int L = 0; L < P->nlevel; ++L) {
            const int i0 = P->lvl_fwd[L] + P->lvl_fwd_g[L], n = P->lvl_fwd[L + 1] - i0;
            k_solve_level<T><<<n, kSolveThreads, smf, s>>>(D, F, b, M->rs, z, upd, x, items, i0,
                                                          stop_a, stop_b);
            V2D_TRY(solve_launch("k_solve_level (forward)", L));
            V2D_TRY(mark(kCodeFwdLevel * 1000 + L));
            ++launches;
        }
        for (int L = P->nlevel - 1; L >= 0; --L) {
            const int i0 = P->lvl_bwd[L + 1] + P->lvl_bwd_g[L], n = P->lvl_bwd[L] - i0;
            k_solve_level<T><<<n, kSolveThreads, smf, s>>>(D, F, b, M->rs, z, upd, x, items, i0,
                                                          stop_a, stop_b);
            V2D_TRY(solve_launch("k_solve_level (backward)", L));
            V2D_TRY(mark(kCodeBwdLevel * 1000 + L));
            ++launches;
        }
    }
    V2D_CUDA_TRY(cudaGetLastError());
    if (n_launches) *n_launches = ev ? nev : launches;
    return V2D_OK;
}

int mf_apply(const MfPlan *P, const MfFactor *M, const void *b, void *x, const int *stop_a,
             const int *stop_b, cudaStream_t s, long long *n_launches)
{
    if (M->fp32)
        return apply_launches<float>(P, M, (const float *)b, (float *)x, stop_a, stop_b, s,
                                     n_launches);
    return apply_launches<double>(P, M, (const double *)b, (double *)x, stop_a, stop_b, s,
                                  n_launches);
}

template <class T>
static int apply_transpose_launches(const MfPlan *P, MfFactor *M, const T *g, T *lam,
                                    cudaStream_t s, long long *launches)
{
    const MfDev D = mf_dev(P, M);
    const T *F = (const T *)(M->fact64 ? M->F32 : M->F);
    const size_t up = tup_smem(P, sizeof(T)), down = tdown_smem(P, sizeof(T));
    for (int L = 0; L < P->nlevel; ++L) {
        const int q0 = P->lvl_off[L], nq = P->lvl_off[L + 1] - q0;
        k_tup_front<T><<<nq, kSolveThreads, up, s>>>(q0, D, F, g, (T *)M->z, (T *)M->upd);
    }
    for (int L = P->nlevel - 1; L >= 0; --L) {
        const int q0 = P->lvl_off[L], nq = P->lvl_off[L + 1] - q0;
        k_tdown_front<T><<<nq, kSolveThreads, down, s>>>(q0, D, F, M->rs, (const T *)M->z,
                                                        (T *)M->wb, lam);
    }
    V2D_CUDA_TRY(cudaGetLastError());
    count_launches(2LL * P->nlevel);
    if (launches) *launches = 2LL * P->nlevel;
    return V2D_OK;
}

int mf_apply_transpose(const MfPlan *P, MfFactor *M, const void *g, void *lambda, cudaStream_t s,
                       long long *launches)
{
    if (M->fp32)
        return apply_transpose_launches<float>(P, M, (const float *)g, (float *)lambda, s,
                                               launches);
    return apply_transpose_launches<double>(P, M, (const double *)g, (double *)lambda, s,
                                            launches);
}

int mf_set_wait_limits(MfPlan *P, MfFactor *M, int gather, int pipe)
{
    M->limits.gather = gather < 0 ? kFlowSpins : std::min(gather, kFlowSpins);
    M->limits.pipe = pipe < 0 ? kPipeSpins : std::min(pipe, kPipeSpins);
    if (M->graph) V2D_CUDA_TRY(cudaGraphExecDestroy(M->graph));
    M->graph = nullptr;
    ++P->items_ver;
    return V2D_OK;
}

int mf_set_split(const MfPlan *P, MfFactor *M, int split)
{
    V2D_ARG_CHECK(split >= 0 && split < P->nlevel, "lu split: level %d (0 .. %d)", split,
                  P->nlevel - 1);
    if (split == 0) {
        M->split = 0;
        return V2D_OK;
    }
    int wcap = 0;
    for (int L = 0; L < split; ++L) wcap = std::max(wcap, P->lvl_maxf[L]);
    FlowShape sh;
    V2D_TRY(flow_setup(M, 2, wcap, kLowMinBlocks, &sh));
    V2D_ARG_CHECK(sh.grid > 0, "lu split: no CTA of the lower-level launch fits on an SM");
    M->shape[2] = sh;
    M->split = split;
    return V2D_OK;
}

int mf_time_apply(const MfPlan *P, const MfFactor *M, int reps, size_t flush_bytes, cudaStream_t s,
                  double *ms_avg)
{
    const size_t es = M->fp32 ? sizeof(float) : sizeof(double);
    DevBuf<char> buf;
    V2D_TRY(buf.alloc(2 * P->n * es + flush_bytes + 256, s));
    V2D_CUDA_TRY(cudaMemsetAsync(buf.p, 0, 2 * P->n * es, s));
    char *fl = buf.p + 2 * P->n * es;
    cudaEvent_t e0, e1;
    V2D_CUDA_TRY(cudaEventCreate(&e0));
    V2D_CUDA_TRY(cudaEventCreate(&e1));
    double total = 0.0;
    int st = V2D_OK;
    for (int r = 0; r < reps && st == V2D_OK; ++r) {
        if (flush_bytes) cudaMemsetAsync(fl, r & 0xff, flush_bytes, s);
        cudaEventRecord(e0, s);
        st = mf_apply(P, M, buf.p, buf.p + P->n * es, nullptr, nullptr, s, nullptr);
        cudaEventRecord(e1, s);
        if (cudaEventSynchronize(e1) != cudaSuccess) st = V2D_ECUDA;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        total += ms;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (st != V2D_OK) return st;
    V2D_TRY(mf_check_barrier(const_cast<MfFactor *>(M), s));   // a solve that gave up is no time
    *ms_avg = total / reps;
    return V2D_OK;
}

// Measurement aid: one dataflow solve of a zero vector with a per-item
// trace (ns of the global timer at the ticket, when the item's vector is
// gathered, after its rows): ticks[3 i + k] for the n items (n <= cap).
int mf_trace_apply(const MfPlan *P, const MfFactor *M, cudaStream_t s, unsigned long long *ticks,
                   int cap, int *n)
{
    V2D_ARG_CHECK(M->flow, "LU solve trace: needs the dataflow solve");
    V2D_ARG_CHECK(cap >= P->nitems, "LU solve trace: %d items, room for %d", P->nitems, cap);
    const size_t es = M->fp32 ? sizeof(float) : sizeof(double);
    DevBuf<char> buf;
    V2D_TRY(buf.alloc(2 * P->n * es + 3 * (size_t)P->nitems * sizeof(unsigned long long) + 256, s));
    V2D_CUDA_TRY(cudaMemsetAsync(buf.p, 0, 2 * P->n * es, s));
    unsigned long long *tr = (unsigned long long *)(buf.p + ((2 * P->n * es + 15) / 16) * 16);
    V2D_CUDA_TRY(cudaMemsetAsync(tr, 0, 3 * (size_t)P->nitems * sizeof(unsigned long long), s));
    int st = M->fp32 ? apply_launches<float>(P, M, (const float *)buf.p,
                                             (float *)(buf.p + P->n * es), nullptr, nullptr, s,
                                             nullptr, nullptr, nullptr, 0, tr)
                     : apply_launches<double>(P, M, (const double *)buf.p,
                                              (double *)(buf.p + P->n * es), nullptr, nullptr, s,
                                              nullptr, nullptr, nullptr, 0, tr);
    V2D_TRY(st);
    V2D_CUDA_TRY(cudaMemcpyAsync(ticks, tr, 3 * (size_t)P->nitems * sizeof(unsigned long long),
                                 cudaMemcpyDeviceToHost, s));
    V2D_CUDA_TRY(cudaStreamSynchronize(s));
    V2D_TRY(mf_check_barrier(const_cast<MfFactor *>(M), s));
    *n = P->nitems;
    return V2D_OK;
}

// Keeps the device busy for about `us` microseconds (bounded), so that the
// host can enqueue a whole solve before it starts and per-launch events then
// time the device, not the host's submission.
__global__ void k_delay(int us)
{
    for (int i = 0; i < us; ++i) __nanosleep(1000);
}

int mf_time_apply_launches(const MfPlan *P, const MfFactor *M, int reps, size_t flush_bytes,
                           cudaStream_t s, double *ms, int *codes, int cap, int *n)
{
    const size_t es = M->fp32 ? sizeof(float) : sizeof(double);
    DevBuf<char> buf;
    V2D_TRY(buf.alloc(2 * P->n * es + flush_bytes + 256, s));
    V2D_CUDA_TRY(cudaMemsetAsync(buf.p, 0, 2 * P->n * es, s));
    char *fl = buf.p + 2 * P->n * es;
    std::vector<cudaEvent_t> ev(cap + 1, nullptr);
    int st = V2D_OK;
    for (auto &e : ev)
        if (st == V2D_OK && cudaEventCreate(&e) != cudaSuccess) st = V2D_ECUDA;
    std::vector<double> acc(cap, 0.0);
    long long nl = 0;
    for (int r = 0; r < reps && st == V2D_OK; ++r) {
        if (flush_bytes) cudaMemsetAsync(fl, r & 0xff, flush_bytes, s);
        k_delay<<<1, 32, 0, s>>>(300);
        cudaEventRecord(ev[0], s);
        st = M->fp32 ? apply_launches<float>(P, M, (const float *)buf.p,
                                             (float *)(buf.p + P->n * es), nullptr, nullptr, s,
                                             &nl, ev.data() + 1, codes, cap)
                     : apply_launches<double>(P, M, (const double *)buf.p,
                                              (double *)(buf.p + P->n * es), nullptr, nullptr,
                                              s, &nl, ev.data() + 1, codes, cap);
        if (st == V2D_OK && cudaEventSynchronize(ev[nl]) != cudaSuccess) st = V2D_ECUDA;
        for (long long k = 0; k < nl && st == V2D_OK; ++k) {
            float t = 0.f;
            cudaEventElapsedTime(&t, ev[k], ev[k + 1]);
            acc[k] += t;
        }
    }
    for (auto &e : ev)
        if (e) cudaEventDestroy(e);
    if (st != V2D_OK) return st;
    V2D_TRY(mf_check_barrier(const_cast<MfFactor *>(M), s));
    for (long long k = 0; k < nl; ++k) ms[k] = acc[k] / reps;
    *n = (int)nl;
    return V2D_OK;
}

int mf_time_factor_launches(const MfPlan *P, MfFactor *M, const int *rowptr, const double *val,
                            int reps, cudaStream_t s, double *ms, int *codes, int cap, int *n)
{
    std::vector<cudaEvent_t> ev(cap + 1, nullptr);
    int st = V2D_OK;
    for (auto &e : ev)
        if (st == V2D_OK && cudaEventCreate(&e) != cudaSuccess) st = V2D_ECUDA;
    std::vector<double> acc(cap, 0.0);
    int nl = 0;
    for (int r = 0; r < reps && st == V2D_OK; ++r) {
        k_delay<<<1, 32, 0, s>>>(2000);
        cudaEventRecord(ev[0], s);
        st = M->fp32 && !M->fact64
                 ? factor_launches<float>(P, M, rowptr, val, s, ev.data() + 1, codes, cap, &nl)
                 : factor_launches<double>(P, M, rowptr, val, s, ev.data() + 1, codes, cap, &nl);
        if (st == V2D_OK && cudaEventSynchronize(ev[nl]) != cudaSuccess) st = V2D_ECUDA;
        for (int k = 0; k < nl && st == V2D_OK; ++k) {
            float t = 0.f;
            cudaEventElapsedTime(&t, ev[k], ev[k + 1]);
            acc[k] += t;
        }
    }
    for (auto &e : ev)
        if (e) cudaEventDestroy(e);
    if (st != V2D_OK) return st;
    V2D_TRY(mf_check_barrier(M, s));
    for (int k = 0; k < nl; ++k) ms[k] = acc[k] / reps;
    *n = nl;
    return V2D_OK;
}

const int *mf_error_word(const MfFactor *M) { return M->bar ? &M->bar->err : nullptr; }

int mf_check_barrier(MfFactor *M, cudaStream_t s)
{
    if (!M->bar) return V2D_OK;
    int err = 0;
    V2D_CUDA_TRY(cudaMemcpyAsync(&err, &M->bar->err, sizeof(int), cudaMemcpyDeviceToHost, s));
    V2D_CUDA_TRY(cudaStreamSynchronize(s));
    if (err) {
        V2D_CUDA_TRY(cudaMemsetAsync(M->bar, 0, sizeof(MfBarrier), s));
        set_error(err & 4 ? "LU factor: a wait of the wide update timed out"
                          : "LU solve: a dependency wait of the dataflow solve timed out");
        return V2D_ETIMEOUT;
    }
    return V2D_OK;
}

}  // namespace v2d
