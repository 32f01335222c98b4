// plan.cu -- flatten a host PLR tree into the device block table.
//
// The tree walk visits nodes in the order of DPLR's recursions
// (src/dplrpmv.c:166-173: ne, sw, then nw, se), records one LRDesc per
// low-rank block and one LeafDesc per dense leaf, assigns every factor
// array a 256-byte aligned slot in one FP64 pool, and builds the apply
// schedules for op N and op T.
#include "hoststage.cuh"

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <numeric>

namespace dg {

static thread_local std::string g_last_error;

void set_error(const char *fmt, ...)
{
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_last_error = buf;
}

int fail(int code, const char *fmt, ...)
{
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_last_error = buf;
    return code;
}

const char *last_error_c() { return g_last_error.c_str(); }

static long long align32(long long x) { return (x + 31) & ~31LL; }

// Structural checks performed by DPLR's recursions before they touch any
// output (src/dplrpmv.c:22-36, :116-130); here they run over the whole
// tree up front so that a malformed tree never produces partial output.
static int check_node(const DPlrMtx *A, int m, const char *fn, int depth)
{
    if (!A) return fail(DPLR_GPU_EINVAL, "%s: null node", fn);
    if (depth > 60) return fail(DPLR_GPU_EINVAL, "%s: tree too deep", fn);
    if (A->type != PLR_DMTX && A->type != PLR_HMTX)
        return fail(DPLR_GPU_EINVAL, "%s: invalid A type", fn);
    if (A->size != m) return fail(DPLR_GPU_EINVAL, "%s: invalid A size", fn);
    if (A->type == PLR_DMTX) {
        if (m > 0 && !A->dd.d) return fail(DPLR_GPU_EINVAL, "%s: dense leaf without data", fn);
        if ((long long)m * m > (1LL << 31))
            return fail(DPLR_GPU_EINVAL, "%s: dense leaf too large", fn);
        return 0;
    }
    if (m % 2 != 0) return fail(DPLR_GPU_EINVAL, "%s: H node of odd size %d", fn, m);
    int h = m / 2;
    const DPlrMtx *lr[2] = {A->dh.ne, A->dh.sw};
    for (const DPlrMtx *L : lr) {
        if (!L) return fail(DPLR_GPU_EINVAL, "%s: null low-rank block", fn);
        if (L->type != PLR_LRMTX) return fail(DPLR_GPU_EINVAL, "%s: invalid A type", fn);
        if (L->size != h) return fail(DPLR_GPU_EINVAL, "%s: invalid A size", fn);
        if (L->dlr.rank < 0 || L->dlr.rank > L->dlr.capacity)
            return fail(DPLR_GPU_EINVAL, "%s: rank %d outside [0, capacity %d]", fn,
                        L->dlr.rank, L->dlr.capacity);
        if (L->dlr.rank > 0 && (!L->dlr.u || !L->dlr.v || !L->dlr.sig))
            return fail(DPLR_GPU_EINVAL, "%s: low-rank block without data", fn);
    }
    int rc = check_node(A->dh.nw, h, fn, depth + 1);
    if (rc) return rc;
    return check_node(A->dh.se, h, fn, depth + 1);
}

int validate_tree(int m, const DPlrMtx *A, const char *fn)
{
    if (m < 0) return fail(DPLR_GPU_EINVAL, "%s: invalid matrix size %d", fn, m);
    return check_node(A, m, fn, 0);
}

// ------------------------------------------------------------- flattening
struct Builder {
    Plan *p;
    int walk(const DPlrMtx *A, int row0, int level)
    {
        if (A->type == PLR_DMTX) {
            LeafDesc L;
            L.d = p->pool_doubles;
            L.row0 = row0;
            L.b = A->size;
            p->pool_doubles += align32((long long)L.b * L.b);
            p->leaves.push_back(L);
            p->nnz += (long long)L.b * L.b;
            return ~(int)(p->leaves.size() - 1);
        }
        int idx = (int)p->nodes.size();
        p->nodes.push_back(HDesc{});
        int h = A->size / 2;
        p->levels = std::max(p->levels, level + 1);
        int ids[2];
        for (int s = 0; s < 2; ++s) {
            const DPlrMtx *B = s == 0 ? A->dh.ne : A->dh.sw;
            LRDesc d;
            d.n = h;
            d.rank = B->dlr.rank;
            d.row0 = s == 0 ? row0 : row0 + h;
            d.col0 = s == 0 ? row0 + h : row0;
            d.level = level;
            d.node = idx;
            d.is_ne = s == 0;
            d.u = p->pool_doubles;
            p->pool_doubles += align32((long long)h * d.rank);
            d.v = p->pool_doubles;
            p->pool_doubles += align32((long long)h * d.rank);
            d.sig = p->pool_doubles;
            p->pool_doubles += align32(d.rank);
            d.toff = p->total_rank;
            p->total_rank += d.rank;
            p->max_rank = std::max(p->max_rank, d.rank);
            p->nnz += 2LL * h * d.rank;          // U and V, as src/dplrnz.c:45 counts
            ids[s] = (int)p->lr.size();
            p->lr.push_back(d);
        }
        HDesc hd;
        hd.row0 = row0;
        hd.m = A->size;
        hd.level = level;
        hd.ne = ids[0];
        hd.sw = ids[1];
        hd.parent = -1;
        hd.nw = walk(A->dh.nw, row0, level + 1);
        hd.se = walk(A->dh.se, row0 + h, level + 1);
        if (hd.nw >= 0) p->nodes[hd.nw].parent = idx;
        if (hd.se >= 0) p->nodes[hd.se].parent = idx;
        p->nodes[idx] = hd;
        return idx;
    }
};

// Equal tiles per leaf: of at most 64 rows, 32 in trees of up to 2048 and 16 in
// trees of up to 1024, whose tiles of 64 rows would leave most SMs idle (one of 64
// rows and 6 columns is 12 us of one SM's FP64 in an N = 1024 product).  The rule
// looks at the tree and not at the plan, so that a matrix of a batch is summed as
// it is alone.  (Tiles of one height for the whole plan, a power of two dividing
// every leaf, left leaves of 50 rows with tiles of 2 and leaves of 75 with tiles
// of 1.)
void tile_starts(const Plan *p, std::vector<int> &starts, int rows)
{
    starts.clear();
    size_t tree = 0;
    for (const LeafDesc &L : p->leaves) {         // in row order
        while (tree + 1 < p->tree_row0.size() && p->tree_row0[tree + 1] <= L.row0) ++tree;
        const int m = (tree + 1 < p->tree_row0.size() ? p->tree_row0[tree + 1] : p->m) - p->tree_row0[tree];
        const int most = rows > 0 ? rows : m <= 1024 ? 16 : m <= 2048 ? 32 : 64;
        const int nt = (L.b + most - 1) / most;
        for (int k = 0; k < nt; ++k) starts.push_back(L.row0 + (int)((long long)k * L.b / nt));
    }
    starts.push_back(p->m);
}

std::pair<int, int> tile_range(const std::vector<int> &starts, int r0, int n)
{
    const auto lo = std::lower_bound(starts.begin(), starts.end(), r0);
    const auto hi = std::lower_bound(lo, starts.end(), r0 + n);
    return {(int)(lo - starts.begin()), (int)(hi - starts.begin())};
}

// Rows of a panel item of block L: the autotuner's, else 512 and less in small
// trees (by the tree, for the same reason).
int untuned_chunk_rows(const LRDesc &L)
{
    const long long m = (long long)L.n << (L.level + 1);
    return m <= 1024 ? 64 : m <= 4096 ? 128 : m <= 16384 ? 256 : kChunkRows;
}

int chunk_rows(const Plan *p, const LRDesc &L) { return p->chunk_tuned ? p->chunk_rows : untuned_chunk_rows(L); }

// Apply schedule for op N (trans = 0) or op T (trans = 1): panels contract
// V (U) with x over the block's input rows, tiles expand U (V) T_b over the
// block's output rows plus the leaf term.
// Output tiles (whole tiles in every leaf) and their terms: every
// low-rank block whose output rows cover the tile, then the leaf term.
// Blocks of H nodes shallower than lmin are left out: the schedule then
// applies the block-diagonal part of the matrix made of its subtrees at
// depth lmin (and the leaves above them).
void build_tiles(const Plan *p, int trans, const std::vector<int> &starts, std::vector<int2> &tiles,
                 std::vector<int> &begin, std::vector<TileTerm> &terms, int lmin)
{
    const int ntiles = (int)starts.size() - 1;
    std::vector<std::vector<TileTerm>> per(ntiles);
    // the leaf first: it needs no T, so an expand that runs ahead can begin with it
    for (const LeafDesc &L : p->leaves) {
        const auto rng = tile_range(starts, L.row0, L.b);
        for (int t = rng.first; t < rng.second; ++t) {
            const int t0 = starts[t];
            TileTerm tt;
            tt.b = 0;
            tt.lda = L.b;
            tt.K = L.b;
            tt.src = 1;
            tt.ldb = 0;
            tt.x_row0 = L.row0;
            if (!trans) {
                tt.a = L.d + (t0 - L.row0);
                tt.trans_a = 0;
            } else {
                tt.a = L.d + (long long)(t0 - L.row0) * L.b;
                tt.trans_a = 1;
            }
            per[t].push_back(tt);
        }
    }
    for (size_t b = 0; b < p->lr.size(); ++b) {
        const LRDesc &L = p->lr[b];
        if (L.rank == 0 || L.level < lmin) continue;
        int out0 = trans ? L.col0 : L.row0;
        long long base = trans ? L.v : L.u;
        const auto rng = tile_range(starts, out0, L.n);
        for (int t = rng.first; t < rng.second; ++t) {
            TileTerm tt;
            tt.a = base + (starts[t] - out0);
            tt.b = L.toff;
            tt.lda = L.n;
            tt.K = L.rank;
            tt.trans_a = 0;
            tt.src = 0;
            tt.ldb = L.rank;
            tt.x_row0 = 0;
            per[t].push_back(tt);
        }
    }
    tiles.clear();
    begin.clear();
    terms.clear();
    for (int t = 0; t < ntiles; ++t) {
        tiles.push_back(make_int2(starts[t], starts[t + 1] - starts[t]));
        begin.push_back((int)terms.size());
        terms.insert(terms.end(), per[t].begin(), per[t].end());
    }
    begin.push_back((int)terms.size());
}

void build_schedule(const Plan *p, int trans, Schedule &S, int lmin)
{
    S.items.clear();
    S.reduces.clear();
    S.max_nch = 0;
    long long poff = 0;
    for (size_t b = 0; b < p->lr.size(); ++b) {
        const LRDesc &L = p->lr[b];
        if (L.rank == 0 || L.n == 0 || L.level < lmin) continue;
        const int CH = chunk_rows(p, L);
        int nch = (L.n + CH - 1) / CH;
        for (int c = 0; c < nch; ++c) {
            PanelItem it;
            it.f = trans ? L.u : L.v;
            it.p = poff;
            it.in0 = trans ? L.row0 : L.col0;
            it.n = L.n;
            it.rank = L.rank;
            it.r0 = c * CH;
            it.len = std::min(CH, L.n - c * CH);
            it.chunk = c;
            S.items.push_back(it);
        }
        ReduceItem r;
        r.p = poff;
        r.t = L.toff;
        r.sig = L.sig;
        r.rank = L.rank;
        r.nch = nch;
        S.max_nch = std::max(S.max_nch, nch);
        S.reduces.push_back(r);
        poff += (long long)nch * L.rank;
    }
    S.partial_per_rhs = poff;
    S.t_per_rhs = p->total_rank;
    S.max_rank = p->max_rank;

    std::vector<int> starts;
    tile_starts(p, starts);
    build_tiles(p, trans, starts, S.tiles, S.tile_begin, S.terms, lmin);
}

int upload_schedule(Schedule &S, long long *bytes)
{
    TableBlock tb;
    add_schedule(S, tb);
    return tb.upload(&S.d_block, bytes);
}

// The live factor values of a host tree as pieces of the pool, in the same
// pre-order as Builder::walk (ascending offsets).
struct Uploader {
    Plan *p;
    std::vector<UploadPiece> pieces;
    size_t lr_i = 0, leaf_i = 0;
    int walk(const DPlrMtx *A)
    {
        if (A->type == PLR_DMTX) {
            const LeafDesc &L = p->leaves[leaf_i++];
            pieces.push_back({L.d, A->dd.d, (size_t)L.b * L.b});
            return 0;
        }
        for (int s = 0; s < 2; ++s) {
            const DPlrMtx *B = s == 0 ? A->dh.ne : A->dh.sw;
            const LRDesc &L = p->lr[lr_i++];
            if (B->dlr.rank != L.rank || B->size != L.n)
                return fail(DPLR_GPU_EINVAL, "plan refresh: structure or rank changed");
            size_t cnt = (size_t)L.n * L.rank;
            if (cnt) {
                pieces.push_back({L.u, B->dlr.u, cnt});
                pieces.push_back({L.v, B->dlr.v, cnt});
                pieces.push_back({L.sig, B->dlr.sig, (size_t)L.rank});
            }
        }
        int rc = walk(A->dh.nw);
        if (rc) return rc;
        return walk(A->dh.se);
    }
};

int plan_upload_values(Plan *p, const DPlrMtx *A, cudaStream_t st)
{
    if (p->ntrees != 1) return fail(DPLR_GPU_EINVAL, "plan refresh: batched plans are refreshed through the pool");
    if (!A || A->size != p->m) return fail(DPLR_GPU_EINVAL, "plan refresh: size mismatch");
    int rc = validate_tree(p->m, A, "dplr_gpu_plan_refresh");
    if (rc) return rc;
    Uploader up{p, {}};
    rc = up.walk(A);
    if (rc) return rc;
    if (up.lr_i != p->lr.size() || up.leaf_i != p->leaves.size())
        return fail(DPLR_GPU_EINVAL, "plan refresh: structure changed");
    if ((rc = stage_upload(p->pool, up.pieces, st))) return rc;
    if ((rc = pairs_refresh(p, st))) return rc;
    DG_CUDA(cudaStreamSynchronize(st));
    return 0;
}

// The block table with op N's schedule, and op T's schedule.
int upload_tables(Plan *p, long long *bytes)
{
    TableBlock tb;
    tb.add(p->lr, &p->d_lr);
    tb.add(p->leaves, &p->d_leaves);
    add_schedule(p->sched[0], tb);
    const int rc = tb.upload(&p->d_tables, bytes);
    return rc ? rc : upload_schedule(p->sched[1], bytes);
}

int plan_build(int m, const DPlrMtx *A, cudaStream_t st, Plan **out, bool values)
{
    return plan_build_forest(1, &m, &A, st, out, values);
}

// A forest of independent trees as one block-diagonal matrix: tree i owns
// rows [sum_{k<i} m_k, sum_{k<=i} m_k).  Blocks and leaves of all trees go
// into the same tables, so every phase covers all trees in one launch.
int plan_build_forest(int count, const int *ms, const DPlrMtx *const *As, cudaStream_t st, Plan **out, bool values)
{
    int rc;
    long long total = 0;
    for (int i = 0; i < count; ++i) {
        if ((rc = validate_tree(ms[i], As[i], count == 1 ? "dplr_gpu_plan_create" : "dplr_gpu_batch_create")))
            return rc;
        total += ms[i];
    }
    if (total > (1LL << 31) - 1) return fail(DPLR_GPU_EINVAL, "plan: %lld rows exceed the int range", total);
    Plan *p = new Plan();
    p->m = (int)total;
    p->ntrees = count;
    Builder b{p};
    int row0 = 0;
    for (int i = 0; i < count; ++i) {
        p->tree_row0.push_back(row0);
        b.walk(As[i], row0, 0);
        row0 += ms[i];
    }
    build_schedule(p, 0, p->sched[0]);
    build_schedule(p, 1, p->sched[1]);
    long long bytes = 0;
    size_t pool_bytes = (size_t)std::max<long long>(p->pool_doubles, 1) * sizeof(double);
    cudaError_t e = dev_malloc((void **)&p->pool, pool_bytes);
    if (e != cudaSuccess) {
        plan_free(p);
        return fail(DPLR_GPU_ENOMEM, "plan: cannot allocate %zu bytes of factor pool: %s",
                    pool_bytes, cudaGetErrorString(e));
    }
    bytes += (long long)pool_bytes;
    // the 256-byte alignment gaps between arrays are zero, so that two plans
    // of equal factors have equal pools
    if (cudaMemsetAsync(p->pool, 0, pool_bytes, st) != cudaSuccess) {
        plan_free(p);
        return fail(DPLR_GPU_ECUDA, "plan: cannot clear the factor pool");
    }
    if ((rc = upload_tables(p, &bytes))) {
        plan_free(p);
        return rc;
    }
    p->device_bytes = bytes;
    Uploader up{p, {}};
    for (int i = 0; i < count && values && !rc; ++i) rc = up.walk(As[i]);
    if (!rc) rc = stage_upload(p->pool, up.pieces, st);
    if (rc) {
        plan_free(p);
        return rc;
    }
    *out = p;
    return 0;
}

// Rebuild the apply schedules (after a change of the panel chunk length); those
// that were there stay on an error.
int plan_reschedule(Plan *p)
{
    long long bytes = 0;
    Schedule now[2];
    int rc = 0;
    for (int trans = 0; trans < 2 && !rc; ++trans) {
        build_schedule(p, trans, now[trans]);
        now[trans].nb_cap = p->nb_cap;
        rc = upload_schedule(now[trans], &bytes);
    }
    for (int trans = 0; trans < 2; ++trans) {
        if (!rc) std::swap(p->sched[trans], now[trans]);
        free_schedule(now[trans]);
    }
    return rc;
}

void free_schedule(Schedule &S)
{
    cudaFree(S.d_block);
    cudaFree(S.d_item_red);
    cudaFree(S.d_term_red);
    S.d_block = nullptr;
    S.d_item_red = S.d_term_red = nullptr;
    S.d_items = nullptr;
    S.d_reduces = nullptr;
    S.d_tiles = nullptr;
    S.d_tile_begin = nullptr;
    S.d_terms = nullptr;
    S.d_caps = nullptr;
}

void factor_free(Plan *p);   // factor.cu
void sliced_free(Plan *p);   // sliced.cu
void mixed_free(Plan *p);    // sliced.cu

void plan_free(Plan *p)
{
    if (!p) return;
    mixed_free(p);
    factor_free(p);
    sliced_free(p);
    pairs_free(p);
    cudaFree(p->pool);
    cudaFree(p->d_tables);
    cudaFree(p->d_tree_row0);
    free_schedule(p->sched[0]);
    free_schedule(p->sched[1]);
    cudaFree(p->work);
    cudaFree(p->xbuf);
    cudaFree(p->ybuf);
    if (p->tc_err_h) cudaFreeHost(p->tc_err_h);
    grad_free(p);
    cudaFree(p->gbuf);
    delete p;
}

int ensure_buffer(double **buf, size_t *have, size_t need)
{
    if (need <= *have && *buf) return 0;
    if (*buf) cudaFree(*buf);
    *buf = nullptr;
    *have = 0;
    size_t n = std::max<size_t>(need, 1);
    cudaError_t e = dev_malloc((void **)buf, n * sizeof(double));
    if (e != cudaSuccess)
        return fail(DPLR_GPU_ENOMEM, "cannot allocate %zu bytes of device scratch: %s",
                    n * sizeof(double), cudaGetErrorString(e));
    *have = n;
    return 0;
}

}  // namespace dg
