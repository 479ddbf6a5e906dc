// The Newton step around its linear solve, for the sparse solvers: one kernel
// forms F1, G and FP of a step, one checks a direct solve's residual, one
// applies the update -- with the decision between them on the device, so that
// a step is enqueued whole and read back once.  Before, a step was a dozen
// launches and four round trips to the host: 0.11 ms of the 0.23 ms that a
// step of 567 unknowns took, 0.14 of 0.46 ms with Gauss-Seidel.
#include <cmath>
#include <cstring>

#include "mp_internal.h"

namespace mp {

namespace {

constexpr int STEP_THREADS = 128;
constexpr int CHECK_TEAM = 16;  // lanes that share one row

// Words of ctx->scal (8 doubles) that a step uses.
enum { S_Y2 = 0, S_R2 = 1, S_OF2 = 2, S_GO = 5, S_FLAGS = 6, S_TICKET = 7 };

// value of lane k of the team, k < TEAM
template <int TEAM>
__device__ __forceinline__ double team_get(double v, int k) {
    return TEAM == 1 ? v : __shfl_sync(0xffffffffu, v, k, TEAM);
}
// largest v of the warp
__device__ __forceinline__ int warp_most(int v) { return __reduce_max_sync(0xffffffffu, v); }

struct TermArgs {
    const int *node;                   // [neq] equation -> node
    const int *eq_ptr, *eq_tet;
    const unsigned char *eq_a;
    const double *detJ, *den, *d, *F0;
    const int *sp_len, *sp_col;
    const long long *sp_ptr;
    const double *sp_val;
    double *F1, *G, *FP, *y;
    double *scal;
    unsigned *clear;                   // words to zero for the kernels that follow (nullable)
    int clear_words, neq, clear_y;
    double qe_eps0, mqe_eps0, n0, phi0, kTe, inv_kTe;
    double Na[4][8];
};

// For each equation A, in the reference's order of operations (the sums of
// k_node_terms, k_eq_gather and k_residual_sparse, bit for bit):
//   F1 += sum over its tets of its load, FP = the same of the Boltzmann term's
//   derivative, G = K d - F0 - F1          (src/FESolver.cpp:333-335, 367-431, 488-526)
// A team of lanes forms the terms of as many tets or columns at once, and then all
// add them up in order: one thread's chain of loads per tet was
// the latency of a small mesh's step.
template <int TEAM>
__global__ void __launch_bounds__(STEP_THREADS) k_newton_terms(TermArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 8) a.scal[i] = 0.0;
    if (i < a.clear_words) a.clear[i] = 0;
    const int lane = threadIdx.x & (TEAM - 1);
    const bool in = i / TEAM < a.neq;
    const int A = in ? i / TEAM : a.neq - 1;           // whole warps take part in the shuffles
    const double dA = a.d[A];
    const double ex = exp(__ddiv_rn(__dsub_rn(dA, a.phi0), a.kTe));
    const double f = __dmul_rn(a.qe_eps0, __dadd_rn(a.den[a.node[A]], __dmul_rn(a.n0, ex)));
    const double fp = __dmul_rn(__dmul_rn(__dmul_rn(a.mqe_eps0, a.n0), ex), a.inv_kTe);
    double F1 = a.F1[A], FP = 0.0;
    const int k0 = a.eq_ptr[A], k1 = a.eq_ptr[A + 1];
    int most = warp_most(k1 - k0);
    for (int base = 0; base < most; base += TEAM) {
        const int k = k0 + base + lane;
        double u = 0.0, v = 0.0;
        if (k < k1) {
            const double dj = a.detJ[a.eq_tet[k]];
            const int q = a.eq_a[k];
#pragma unroll
            for (int p = 0; p < 8; p++) {
                u = __dadd_rn(u, __dmul_rn(__dmul_rn(f, a.Na[q][p]), dj));
                v = __dadd_rn(v, __dmul_rn(__dmul_rn(fp, a.Na[q][p]), dj));
            }
            u = __dmul_rn(u, 1.0 / 8.0);
            v = __dmul_rn(v, 1.0 / 8.0);
        }
#pragma unroll
        for (int j = 0; j < TEAM; j++) {
            const double uj = team_get<TEAM>(u, j), vj = team_get<TEAM>(v, j);
            if (k0 + base + j < k1) {
                F1 = __dadd_rn(F1, uj);
                FP = __dadd_rn(FP, vj);
            }
        }
    }
    const long long row = a.sp_ptr[A >> 5] + (A & 31);
    const int len = a.sp_len[A];
    most = warp_most(len);
    double s = 0.0;
    for (int base = 0; base < most; base += TEAM) {
        const int k = base + lane;
        const double v = k < len ? __dmul_rn(a.sp_val[row + 32ll * k], a.d[a.sp_col[row + 32ll * k]]) : 0.0;
#pragma unroll
        for (int j = 0; j < TEAM; j++) {
            const double vj = team_get<TEAM>(v, j);
            if (base + j < len) s = __dadd_rn(s, vj);
        }
    }
    if (in && lane == 0) {
        a.F1[A] = F1;
        a.FP[A] = FP;
        a.G[A] = __dsub_rn(__dsub_rn(s, a.F0[A]), F1);
        if (a.clear_y) a.y[A] = 0.0;
    }
}

struct CheckArgs {
    const int *sp_len, *sp_col;
    const long long *sp_ptr;
    const double *sp_val, *FP, *y, *b;
    double *r, *scal;
    const unsigned long long *flags;
    unsigned long long bad;            // flag bits that refuse the solution
    int neq;
    double rtol;
    bool terms;                        // relative to r's terms, not to b
};

// r = b - (K y - FP .* y), its norm and b's, or that of the terms r is the sum of, |b| + |K| |y|
// + |FP| |y|; the last block decides whether the solution is taken (S_GO = 0): the first norm
// <= rtol times the second and none of the bad flags.
template <int TEAM>
__global__ void __launch_bounds__(STEP_THREADS) k_newton_check(CheckArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & (TEAM - 1);
    const int P = i / TEAM;
    double s = 0.0, t = 0.0, rr = 0.0, oo = 0.0;
    if (P < a.neq) {
        const long long row = a.sp_ptr[P >> 5] + (P & 31);
        const int len = a.sp_len[P];
        for (int k = lane; k < len; k += TEAM) {
            const double v = a.sp_val[row + 32ll * k], x = a.y[a.sp_col[row + 32ll * k]];
            s = fma(v, x, s);
            t = fma(fabs(v), fabs(x), t);
        }
    }
#pragma unroll
    for (int o = TEAM / 2; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    if (P < a.neq && lane == 0) {
        const double fy = a.FP[P] * a.y[P], v = a.b[P] - (s - fy);
        a.r[P] = v;
        rr = v * v;
        const double of = a.terms ? t + fabs(fy) + fabs(a.b[P]) : a.b[P];
        oo = of * of;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        rr += __shfl_xor_sync(0xffffffffu, rr, o);
        oo += __shfl_xor_sync(0xffffffffu, oo, o);
    }
    __shared__ double part[2][STEP_THREADS / 32];
    if ((threadIdx.x & 31) == 0) {
        part[0][threadIdx.x >> 5] = rr;
        part[1][threadIdx.x >> 5] = oo;
    }
    __syncthreads();
    if (threadIdx.x) return;
    for (int w = 1; w < STEP_THREADS / 32; w++) {
        rr += part[0][w];
        oo += part[1][w];
    }
    atomicAdd(a.scal + S_R2, rr);
    atomicAdd(a.scal + S_OF2, oo);
    __threadfence();
    unsigned *ticket = reinterpret_cast<unsigned *>(a.scal + S_TICKET);
    if (atomicAdd(ticket, 1u) + 1 < gridDim.x) return;
    __threadfence();
    *ticket = 0;
    const double r2 = __ldcg(a.scal + S_R2), of2 = __ldcg(a.scal + S_OF2);
    const unsigned long long fl = *reinterpret_cast<const volatile unsigned long long *>(a.flags) & a.bad;
    *reinterpret_cast<unsigned long long *>(a.scal + S_FLAGS) = fl;
    *reinterpret_cast<unsigned *>(a.scal + S_GO) = sqrt(r2) <= a.rtol * sqrt(of2) && !fl ? 0u : 1u;
}

// d -= y with sum y^2, and uh = g + d (src/FESolver.cpp:341-349, 610-618), unless *stop
__global__ void __launch_bounds__(256) k_newton_update(int n_nodes, const int *__restrict__ ID, const double *__restrict__ g,
                                                       const double *__restrict__ y, const unsigned *stop, double *d,
                                                       double *uh, double *sum) {
    if (stop && *stop) return;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    double s = 0.0;
    if (n < n_nodes) {
        const int A = ID[n];
        double u = g[n];
        if (A >= 0) {
            const double v = y[A], x = __dsub_rn(d[A], v);
            d[A] = x;
            u = __dadd_rn(u, x);
            s = v * v;
        }
        uh[n] = u;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0 && s != 0.0) atomicAdd(sum, s);
}

}  // namespace

int newton_terms(mp_ctx *ctx, const double *den, bool clear_y, unsigned *clear, int clear_words) {
    TermArgs a;
    a.node = ctx->eq_node;
    a.eq_ptr = ctx->eq_ptr;
    a.eq_tet = ctx->eq_tet;
    a.eq_a = ctx->eq_a;
    a.detJ = ctx->detJ;
    a.den = den;
    a.d = ctx->d;
    a.F0 = ctx->F0;
    a.sp_len = ctx->sp_len;
    a.sp_col = ctx->sp_col;
    a.sp_ptr = ctx->sp_ptr;
    a.sp_val = ctx->sp_val;
    a.F1 = ctx->F1;
    a.G = ctx->G;
    a.FP = ctx->FP;
    a.y = ctx->y;
    a.scal = ctx->scal;
    a.clear = clear;
    a.clear_words = clear_words;
    a.neq = ctx->neq;
    a.clear_y = clear_y;
    a.qe_eps0 = QE / EPS0;
    a.mqe_eps0 = -QE / EPS0;
    a.n0 = ctx->n0;
    a.phi0 = ctx->phi0;
    a.kTe = ctx->kTe;
    a.inv_kTe = 1.0 / ctx->kTe;
    const Quadrature q = make_quadrature();
    for (int k = 0; k < 4; k++)
        for (int p = 0; p < 8; p++) a.Na[k][p] = q.Na[k][p];
    // eight lanes an equation where latency counts, four where the lanes' own adding up
    // does: 8, 4, 2, 1 lanes made a step of 8,379 unknowns 484, 491, 492, 495 us, and one of
    // 89,276 (conjugate gradients cut short) 133, 117, 123, 125 us
    const int team = ctx->neq < 16384 ? 8 : 4;
    const unsigned blocks = (unsigned)(((long long)ctx->neq * team + STEP_THREADS - 1) / STEP_THREADS);
    if (team == 8) k_newton_terms<8><<<blocks, STEP_THREADS, 0, ctx->stream>>>(a), ++ctx->launches;
    else k_newton_terms<4><<<blocks, STEP_THREADS, 0, ctx->stream>>>(a), ++ctx->launches;
    MP_CUDA(ctx, cudaGetLastError());
    return MP_OK;
}

int newton_check(mp_ctx *ctx, double rtol, bool terms, unsigned long long bad_flags) {
    CheckArgs a;
    a.sp_len = ctx->sp_len;
    a.sp_col = ctx->sp_col;
    a.sp_ptr = ctx->sp_ptr;
    a.sp_val = ctx->sp_val;
    a.FP = ctx->FP;
    a.y = ctx->y;
    a.b = ctx->G;
    a.r = ctx->work;
    a.scal = ctx->scal;
    a.flags = ctx->counters + C_FLAGS;
    a.bad = bad_flags;
    a.neq = ctx->neq;
    a.rtol = rtol;
    a.terms = terms;
    const unsigned blocks = (unsigned)(((long long)ctx->neq * CHECK_TEAM + STEP_THREADS - 1) / STEP_THREADS);
    k_newton_check<CHECK_TEAM><<<blocks, STEP_THREADS, 0, ctx->stream>>>(a), ++ctx->launches;
    MP_CUDA(ctx, cudaGetLastError());
    return MP_OK;
}

const unsigned *newton_go(mp_ctx *ctx) { return reinterpret_cast<const unsigned *>(ctx->scal + S_GO); }

int newton_update(mp_ctx *ctx, const unsigned *stop) {
    k_newton_update<<<(ctx->n_nodes + 255) / 256, 256, 0, ctx->stream>>>(ctx->n_nodes, ctx->ID, ctx->g, ctx->y, stop,
                                                                        ctx->d, ctx->uh, ctx->scal + S_Y2),
        ++ctx->launches;
    MP_CUDA(ctx, cudaGetLastError());
    MP_CUDA(ctx, cudaMemcpyAsync(ctx->scal_host, ctx->scal, sizeof(double) * 8, cudaMemcpyDeviceToHost, ctx->stream));
    return MP_OK;
}

// What a step left, after the stream has been waited for.
void newton_read(mp_ctx *ctx, NewtonState *s) {
    s->l2 = std::sqrt(ctx->scal_host[S_Y2]) / ctx->neq;
    s->rn = std::sqrt(ctx->scal_host[S_R2]);
    s->of = std::sqrt(ctx->scal_host[S_OF2]);
    unsigned go;
    std::memcpy(&go, ctx->scal_host + S_GO, sizeof(go));
    s->taken = go == 0;
    std::memcpy(&s->flags, ctx->scal_host + S_FLAGS, sizeof(s->flags));
}

}  // namespace mp
