// Gauss-Seidel (FESolver::solveLinear, src/FESolver.cpp:561-601) on the sparse J
// = K - diag(FP): the whole solve, sweeps and residual checks, in one launch of
// one thread-block cluster.
//
// A sweep visits the rows in order, and row u needs this sweep's values of its
// lower-numbered neighbours and the last sweep's of the others.  With level(u) =
// 1 + the highest level of u's lower neighbours, the rows of a level are
// independent, and sweep s + 1 can follow sweep s at a distance of D = 1 + the
// largest level difference between neighbours (4 on a Kuhn mesh numbered by
// coordinate): at step w every row with level(u) + D s = w, for any sweep s, is
// updated at once, so S sweeps of L levels take L + D (S - 1) steps instead of
// L S.  The iterates are those of the row-by-row order up to rounding.
//
// Every thread owns one row, with its matrix entries in registers; a CTA owns a
// run of consecutive rows, so that on a mesh numbered by coordinate only the
// rows at its ends have neighbours elsewhere.  x lies in every CTA's shared
// memory, a CTA's rows ordered so that rows updated at the same steps are
// neighbours (a warp's gathers then fall into few banks).  A new value goes to
// the CTAs that need it with st.async, which also counts it on the receiver's
// mbarrier of the step: a CTA goes on when its own rows are done (a block
// barrier) and the bytes due have come.  With them comes a token from each CTA
// it exchanges values with: nobody is more than one step ahead of a CTA it
// sends to, also past steps at which that one has no rows, so two mbarriers in
// turn are enough; and a CTA's values and token of a step leave after it has
// read what it needs, so no value is overwritten before its last read.
// A step is bound by latency: one row's gathers and sum, the remote stores and
// the barrier; 0.29 us in one CTA, 0.52 us in a cluster.  A Gauss-Seidel step of
// 1,859 unknowns (126 sweeps) took 4.2 ms with dense sweeps over 64-row blocks
// and takes 0.43 ms.
#include <algorithm>
#include <cmath>
#include <exception>

#include "mp_alloc.h"
#include "mp_internal.h"

namespace mp {

namespace {

constexpr int GS_ENTRIES = 14;         // off-diagonal entries of a row: a Kuhn node's neighbours
constexpr int GS_MAX_CLUSTER = 8;      // portable cluster size
constexpr unsigned GS_SPIN_LIMIT = 1u << 22;

struct GsArgs {
    // by position, [P] = [CTAs][threads]
    const int *row;                    // equation, -1: padding
    const int *level;
    const unsigned char *to;           // bit r: CTA r needs the row's values
    const unsigned short *col;         // [GS_ENTRIES][P] positions of the row's neighbours (own position: none)
    const int *slot;                   // [GS_ENTRIES + 1][P] slots of K's values; the last: the diagonal's
    const int *phase;                  // [P / 32] steps the warp is active at, modulo D (-1: never)
    const int *due;                    // [CTAs][levels] values it gets from rows at levels l, l - D, l - 2 D, ...
    const int *near;                   // [CTAs] bit r: it exchanges values with CTA r
    const double *kval, *FP, *b;
    double *y;
    double *out;                       // [0] sweeps done, [1] last ||b - J y||^2, [2] converged, [3] a wait gave up
    int n, levels, distance, max_sweeps;
    double tol;                        // on sqrt(||b - J y||^2) / n
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_size() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned sm_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned in_cta(unsigned a, unsigned rank) {
    unsigned q;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(q) : "r"(a), "r"(rank));
    return q;
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1) k_gs_cluster(GsArgs a) {
    extern __shared__ __align__(16) double x[];        // [P]
    __shared__ double part[THREADS / 32], total[GS_MAX_CLUSTER];
    __shared__ double token[GS_MAX_CLUSTER];
    __shared__ unsigned long long come[2];
    const unsigned rank = cluster_rank(), size = cluster_size();
    const int t = threadIdx.x, lane = t & 31, P = (int)size * THREADS, p = (int)rank * THREADS + t;
    const bool row = a.row[p] >= 0;
    const int level = row ? a.level[p] : 1 << 30, phase = a.phase[p >> 5];
    const unsigned to = row ? a.to[p] : 0, near = a.near[rank];
    const bool tokens = t < (int)size && (near >> t & 1);   // this thread sends CTA t its token
    double v[GS_ENTRIES], inv = 0.0, b = 0.0;
    constexpr bool WIDE = THREADS <= 512;              // registers for whole offsets; else two positions in one
    unsigned c[WIDE ? GS_ENTRIES : GS_ENTRIES / 2];
#pragma unroll
    for (int k = 0; k < GS_ENTRIES; k++) v[k] = 0.0;
#pragma unroll
    for (int k = 0; k < (WIDE ? GS_ENTRIES : GS_ENTRIES / 2); k++) c[k] = 0;
    bool keep = false;                                 // |J_uu| < 1e-12: the row keeps its value
    if (row) {
        const int u = a.row[p];
#pragma unroll
        for (int k = 0; k < GS_ENTRIES; k++) {
            const unsigned q = a.col[k * P + p];
            if (WIDE) c[k] = q * (unsigned)sizeof(double);
            else c[k / 2] |= q << (16 * (k & 1));
            if ((int)q != p) v[k] = a.kval[a.slot[k * P + p]];
        }
        const double diag = a.kval[a.slot[GS_ENTRIES * P + p]] - a.FP[u];
        b = a.b[u];
        keep = fabs(diag) < 1e-12;
        inv = 1.0 / diag;
    }
    if (t == 0) {
        for (int k = 0; k < 2; k++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sm_addr(come + k)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int q = t; q < P; q += THREADS) {
        const int w = a.row[q];
        x[q] = w >= 0 ? a.y[w] : 0.0;
    }
    cluster_sync();
    auto row_sum = [&] {
        double s[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < GS_ENTRIES; k++) {
            const unsigned o = WIDE ? c[k] : (c[k / 2] >> (16 * (k & 1)) & 0xFFFFu) * (unsigned)sizeof(double);
            s[k % 3] = fma(v[k], *reinterpret_cast<const double *>(reinterpret_cast<const char *>(x) + o), s[k % 3]);
        }
        return (s[0] + s[1]) + s[2];
    };
    // the bytes that come at step w: values and tokens
    auto incoming = [&](int w, int turn, int S) {
        int hi = min(w, a.levels - 1);
        hi -= (hi - turn + a.distance) % a.distance;
        const int lo = w - a.distance * S;
        const int *o = a.due + rank * a.levels;
        return 8u * (unsigned)((hi >= 0 ? o[hi] : 0) - (lo >= 0 ? o[min(lo, hi)] : 0) + __popc(near));
    };
    auto send = [&](unsigned at, double value, unsigned bar, unsigned r) {
        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(in_cta(at, r)),
                     "l"(__double_as_longlong(value)), "r"(in_cta(bar, r))
                     : "memory");
    };
    int done = 0;
    unsigned step = 0;                                 // of all sweeps so far: mbarrier and parity
    double r2 = 0.0;
    bool converged = false, ok = true;
    // the reference checks the residual after sweeps 1, 26, 51, ...
    while (done < a.max_sweeps) {
        const int S = done == 0 ? 1 : min(25, a.max_sweeps - done);
        const int steps = a.levels + a.distance * (S - 1);
        int turn = 0;                                  // step modulo distance
        unsigned bytes = near && t == 0 ? incoming(0, 0, S) : 0;
        int w = 0;
        for (; w < steps && ok; w++, step++) {
            const unsigned bar = sm_addr(come + (step & 1));
            if (near && t == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
            // level + distance * s = w for a sweep s of this batch
            if (phase == turn && w >= level && w < level + a.distance * S) {
                double xn = (b - row_sum()) * inv;
                if (keep) xn = x[p];
                x[p] = xn;
                for (unsigned m = to; m; m &= m - 1) send(sm_addr(x + p), xn, bar, __ffs(m) - 1);
            }
            if (tokens) send(sm_addr(token + rank), 0.0, bar, t);
            turn = turn + 1 == a.distance ? 0 : turn + 1;
            if (near && t == 0 && w + 1 < steps) bytes = incoming(w + 1, turn, S);
            __syncthreads();
            for (unsigned i = 0; near; i++) {
                unsigned got;
                asm volatile(
                    "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                    "selp.u32 %0, 1, 0, p;\n\t}"
                    : "=r"(got)
                    : "r"(bar), "r"((step >> 1) & 1)
                    : "memory");
                if (got) break;
                if (i > GS_SPIN_LIMIT) {               // a warp's lanes poll as one, and give up as one
                    ok = false;
                    break;
                }
            }
        }
        // After a wait that gave up: no arming, sending or waiting any more, so that a phase that
        // never ends gets no second arrival and the other CTAs' waits give up too; the host is
        // told.  (1,859 unknowns, 126 sweeps: 432.3 us before, 433.8 so, within the noise.)
        for (; w < steps; w++) __syncthreads();
        done += S;
        if ((done - 1) % 25) break;                    // the sweep limit came before the next check
        double r = 0.0;
        if (row) {
            const double diag = a.kval[a.slot[GS_ENTRIES * P + p]] - a.FP[a.row[p]];
            r = b - fma(diag, x[p], row_sum());
        }
        r *= r;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        if (lane == 0) part[t >> 5] = r;
        __syncthreads();
        if (t < (int)size) {
            double s = 0.0;
            for (int k = 0; k < THREADS / 32; k++) s += part[k];
            asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(in_cta(sm_addr(total + rank), t)), "d"(s) : "memory");
        }
        cluster_sync();
        r2 = 0.0;
        for (unsigned k = 0; k < size; k++) r2 += total[k];
        cluster_sync();                                // before the next check overwrites the sums
        if (sqrt(r2) / a.n < a.tol) {
            converged = true;
            break;
        }
    }
    if (row) a.y[a.row[p]] = x[p];
    if (!ok) a.out[3] = 1.0;
    if (rank == 0 && t == 0) {
        a.out[0] = done;
        a.out[1] = r2;
        a.out[2] = converged;
    }
    cluster_sync();                                    // no CTA leaves while others may still write to it
    if (!ok)
        for (int i = 0; i < 100; i++) __nanosleep(1000);   // values not waited for may still be on their way
}

struct GsState {
    bool usable = false;
    void *blob = nullptr;
    GsArgs a{};
    double *out = nullptr, *out_host = nullptr;
    int threads = 512, cluster = 1;
};

}  // namespace

void gs_free(mp_ctx *ctx) {
    GsState *s = static_cast<GsState *>(ctx->gs);
    if (!s) return;
    if (s->blob) cudaFree(s->blob);
    if (s->out) cudaFree(s->out);
    if (s->out_host) cudaFreeHost(s->out_host);
    delete s;
    ctx->gs = nullptr;
}

static int gs_plan(mp_ctx *ctx, bool *usable) {
    GsState *s = static_cast<GsState *>(ctx->gs);
    if (!s) {
        s = new GsState();
        ctx->gs = s;
        const int n = ctx->neq;
        bool fits = false;
        int rc = fe_pattern_fits(ctx, &fits);
        if (rc) return rc;
        const std::vector<long long> &ptr = ctx->csr_ptr;
        const std::vector<int> &col = ctx->csr_col;
        if (ptr.empty() || n > 1024 * GS_MAX_CLUSTER) fits = false;
        for (int u = 0; u < n && fits; u++) fits = ptr[u + 1] - ptr[u] <= GS_ENTRIES + 1;
        if (!fits) return MP_OK;
        std::vector<int> level(n, 0);
        int levels = 0, distance = 1;
        for (int u = 0; u < n; u++) {
            for (long long k = ptr[u]; k < ptr[u + 1] && col[k] < u; k++) level[u] = std::max(level[u], level[col[k]] + 1);
            levels = std::max(levels, level[u] + 1);
        }
        for (int u = 0; u < n; u++)
            for (long long k = ptr[u]; k < ptr[u + 1] && col[k] < u; k++)
                distance = std::max(distance, level[u] - level[col[k]] + 1);
        // a CTA's run of rows: by level modulo distance, each class padded to whole warps, then by
        // level and number.  Small CTAs have the quicker block barrier and registers to spare.
        std::vector<int> row, phase, place(n);
        int threads = 512, cluster = 1;
        for (bool done = false; !done;) {
            done = true;
            row.assign((size_t)threads * cluster, -1);
            phase.assign(row.size() / 32, -1);
            std::vector<std::vector<int>> at(distance);
            for (int r = 0; r < cluster && done; r++) {
                const int u0 = (int)((long long)n * r / cluster), u1 = (int)((long long)n * (r + 1) / cluster);
                for (auto &c : at) c.clear();
                for (int u = u0; u < u1; u++) at[level[u] % distance].push_back(u);
                int o = r * threads;
                for (int c = 0; c < distance && done; c++) {
                    std::stable_sort(at[c].begin(), at[c].end(), [&](int i, int j) { return level[i] < level[j]; });
                    if (o + (((int)at[c].size() + 31) & ~31) > (r + 1) * threads) done = false;
                    for (size_t k = 0; k < at[c].size() && done; k++) {
                        phase[o >> 5] = c;
                        place[at[c][k]] = o;
                        row[o++] = at[c][k];
                    }
                    o = (o + 31) & ~31;
                }
            }
            if (!done) {
                cluster *= 2;
                if (cluster > GS_MAX_CLUSTER && threads == 512) {
                    threads = 1024;
                    cluster = GS_MAX_CLUSTER / 2;
                }
                if (cluster > GS_MAX_CLUSTER) return MP_OK;
            }
        }
        // 26 sweeps take 2 levels + 24 distance steps of 0.18 us in one CTA, 0.48 in a cluster of
        // 512 threads a CTA, 0.68 of 1,024, and 40 us; dense sweeps 140 us and 0.43 us a row.  Numbers
        // far from the coordinates' order make many levels and large distances: 144 rows numbered at
        // random 294 us here, 232 dense; 567 rows 453 and 396, at random within slabs 640 and 395; but
        // 1,859 rows at random 500 and 931.  By coordinate 60 to 214 us here, 163 to 3,970 dense.
        const double step = cluster == 1 ? 0.18 : threads == 512 ? 0.48 : 0.68;
        if (40 + (2.0 * levels + 24.0 * distance) * step > 140 + 0.43 * n) return MP_OK;
        const int P = (int)row.size();
        // who needs whose values
        std::vector<unsigned char> to(P, 0);
        std::vector<int> near(cluster, 0), due((size_t)cluster * levels, 0);
        for (int u = 0; u < n; u++) {
            const int own = place[u] / threads;
            for (long long k = ptr[u]; k < ptr[u + 1]; k++) {
                const int r = place[col[k]] / threads;
                if (r != own) to[place[u]] |= (unsigned char)(1u << r);
            }
            near[own] |= to[place[u]];
            for (int r = 0; r < cluster; r++)
                if (to[place[u]] >> r & 1) due[(size_t)r * levels + level[u]]++;
        }
        for (int r = 0; r < cluster; r++)
            for (int l = distance; l < levels; l++) due[(size_t)r * levels + l] += due[(size_t)r * levels + l - distance];
        std::vector<int> lev(P, 0), slot((GS_ENTRIES + 1) * (size_t)P, 0);
        std::vector<unsigned short> cc(GS_ENTRIES * (size_t)P);
        for (int p = 0; p < P; p++) {
            const int u = row[p];
            for (int k = 0; k < GS_ENTRIES; k++) cc[(size_t)k * P + p] = (unsigned short)p;
            if (u < 0) continue;
            lev[p] = level[u];
            int k = 0;
            for (long long q = ptr[u]; q < ptr[u + 1]; q++) {
                if (col[q] == u) {
                    slot[(size_t)GS_ENTRIES * P + p] = (int)ctx->csr_slot[q];
                } else {
                    cc[(size_t)k * P + p] = (unsigned short)place[col[q]];
                    slot[(size_t)k * P + p] = (int)ctx->csr_slot[q];
                    k++;
                }
            }
        }
        size_t off[8], end = 0;
        const size_t bytes[8] = {sizeof(int) * row.size(), sizeof(int) * lev.size(), sizeof(int) * slot.size(),
                                 sizeof(int) * phase.size(), sizeof(unsigned short) * cc.size(),
                                 sizeof(int) * due.size(), sizeof(int) * near.size(), to.size()};
        const void *src[8] = {row.data(), lev.data(), slot.data(), phase.data(), cc.data(), due.data(), near.data(),
                              to.data()};
        for (int k = 0; k < 8; k++) {
            off[k] = end;
            end = (end + bytes[k] + 255) & ~size_t(255);
        }
        if (!allocate_all({{&s->blob, end}, {(void **)&s->out, sizeof(double) * 4}}, device_room, cudaFree)) {
            gs_free(ctx);
            return MP_OK;
        }
        char *base = static_cast<char *>(s->blob);
        for (int k = 0; k < 8; k++) MP_CUDA(ctx, upload(ctx, base + off[k], src[k], bytes[k]));
        MP_CUDA(ctx, cudaHostAlloc(&s->out_host, sizeof(double) * 4, 0));
        const int most = (int)sizeof(double) * 1024 * GS_MAX_CLUSTER;
        MP_CUDA(ctx, cudaFuncSetAttribute(k_gs_cluster<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        MP_CUDA(ctx, cudaFuncSetAttribute(k_gs_cluster<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        s->a.row = reinterpret_cast<const int *>(base + off[0]);
        s->a.level = reinterpret_cast<const int *>(base + off[1]);
        s->a.slot = reinterpret_cast<const int *>(base + off[2]);
        s->a.phase = reinterpret_cast<const int *>(base + off[3]);
        s->a.col = reinterpret_cast<const unsigned short *>(base + off[4]);
        s->a.due = reinterpret_cast<const int *>(base + off[5]);
        s->a.near = reinterpret_cast<const int *>(base + off[6]);
        s->a.to = reinterpret_cast<const unsigned char *>(base + off[7]);
        MP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        s->a.n = n;
        s->a.levels = levels;
        s->a.distance = distance;
        s->cluster = cluster;
        s->threads = threads;
        s->usable = true;
    }
    *usable = s->usable;
    return MP_OK;
}

// Plans the solve on its first use after mp_fe_setup.  *usable: every row fits
// a thread and all rows one cluster of at most 8 CTAs, K has the mesh's
// pattern, and the rows' numbering makes this the faster way.  Where the device or the host is too full for the plan, the dense
// sweeps take the call and the next call asks again.
int gs_prepare(mp_ctx *ctx, bool *usable) {
    *usable = false;
    try {
        return gs_plan(ctx, usable);
    } catch (const std::exception &) {
        gs_free(ctx);
        return MP_OK;
    }
}

// Sweeps J y = G from the current y; FP is J's diagonal term.  *stop: a device word
// that is not zero when the solve failed.
int gs_enqueue(mp_ctx *ctx, double tol, const unsigned **stop) {
    GsState *s = static_cast<GsState *>(ctx->gs);
    GsArgs a = s->a;
    a.kval = ctx->sp_val;
    a.FP = ctx->FP;
    a.b = ctx->G;
    a.y = ctx->y;
    a.out = s->out;
    a.max_sweeps = ctx->gs_max_sweeps;
    a.tol = tol;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(s->cluster);
    cfg.blockDim = dim3(s->threads);
    cfg.dynamicSmemBytes = sizeof(double) * (size_t)s->threads * s->cluster;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = s->cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const int mk = kt_begin(ctx, MP_KT_TRSV, 0);
    MP_CUDA(ctx, cudaMemsetAsync(s->out, 0, sizeof(double) * 4, ctx->stream));
    MP_CUDA(ctx, cudaLaunchKernelEx(&cfg, s->threads == 512 ? k_gs_cluster<512> : k_gs_cluster<1024>, a));
    ++ctx->launches;
    kt_end(ctx, mk);
    MP_CUDA(ctx, cudaMemcpyAsync(s->out_host, s->out, sizeof(double) * 4, cudaMemcpyDeviceToHost, ctx->stream));
    if (stop) *stop = reinterpret_cast<const unsigned *>(s->out + 3) + 1;  // the high word of 1.0
    return MP_OK;
}

// The solve's results, after the stream has been waited for.
int gs_finish(mp_ctx *ctx, mp_newton_stats *st) {
    GsState *s = static_cast<GsState *>(ctx->gs);
    if (s->out_host[3] != 0.0) return fail(ctx, MP_ERR_TIMEOUT, "a bounded wait in the Gauss-Seidel sweep gave up");
    if (st) {
        const bool converged = s->out_host[2] != 0.0;
        st->linear_iterations = converged ? (int)s->out_host[0] - 1 : ctx->gs_max_sweeps;
        st->linear_residual = std::sqrt(s->out_host[1]) / ctx->neq;
        if (!converged) st->linear_failures++;
    }
    return MP_OK;
}

}  // namespace mp
