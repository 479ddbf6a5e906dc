// Sparse direct solve of J y = G, J = K - diag(FP): L D L^T without pivoting on
// 64 x 64 tiles in a nested-dissection order (mp_nd_plan.cpp), in FP64.
//
// k_nd_factor is one launch: CTAs take the plan's tasks in order by an atomic
// ticket and a task forms one tile, all its products first (left-looking), so
// every entry is one sum in a fixed order and the factor is the same from run
// to run.  A tile is announced by its flag word; a task waits only for tiles
// of tasks before it in the order, whose CTAs already run, so no co-residency
// is assumed.
//   warp 16 (one lane) producer: takes the ticket, waits for the flags of a
//                      product's two tiles and copies them (cp.async.bulk) into
//                      one of two shared-memory stages, ahead of the others;
//   warps 0-15         C -= A D B^T on the FP64 tensor cores (mma.sync m8n8k4),
//                      then the tile's end: off the diagonal L = C L_jj^-T D_j^-1;
//                      on it the 64 x 64 factor, its inverse, and the forward
//                      substitution of the right-hand side.
//   warp 17 (one lane) publisher: releases a finished tile's flag, so that only
//                      it waits for the tile's stores.
// Measured (B200, Newton step of the Lapack method, dense LDL^T before -> now): 567
// unknowns 0.70 -> 0.15 ms, 8,379 15.5 -> 0.46 ms, 32,244 (mixed form) 41.3 ->
// 1.29 ms.  The chain of diagonal blocks, 15 us a block (64 x 64 factor 8.4,
// products through the tile before it 3, hand-over between SMs 2; with 8 working
// warps instead of 16, 17.7 us), bounds the small meshes and the upper levels of
// the large ones; the FP64 tensor cores' rate (64 multiply-adds a cycle and SM) and
// the tasks' own latency the lower levels.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <exception>

#include "mp_alloc.h"
#include "mp_internal.h"
#include "mp_nd.h"
#include "mp_recip.cuh"

namespace mp {

namespace {

constexpr int T = ND_TILE;
constexpr int TT = T * T;
constexpr int STAGES = 2;
constexpr int WORK = 512;              // threads of warps 0-15
constexpr int THREADS = WORK + 64;     // and the producer's and the publisher's warp
constexpr int PUBS = 4;
constexpr unsigned POLL_LIMIT = 1u << 22;
constexpr int ZD = 3 * T;              // a tile column's z, D and 1/D

struct NdArgs {
    const NdTask *task;
    const NdItem *item;
    const int *perm, *ent_src;
    const unsigned short *ent_at;
    const double *kval, *FP, *b;
    double *tile, *zd, *x;             // x: the solution by column, emptied here
    unsigned *flag;                    // [ntile] epoch of the tile's last forming
    unsigned *ctl;                     // ticket, abort
    unsigned long long *flags;
    int ntask, ntile, ncol;
    unsigned epoch;
};

struct Smem {
    double stage[STAGES][2][TT];
    double zd[STAGES][ZD];
    double c[TT];                      // the tile being finished
    double inv[TT];                    // a diagonal block's inverse
    double invt[7 * 7 * 64];           // its first 56 rows and columns, transposed
    double tt[7 * 64];                 // 8 rows of L times the inverse's rows above, transposed
    double r[T], d[T], dinv[T];
    double z7[8][8];                   // by inverse block: the last 8 rows of z
    NdTask task[STAGES];
    NdItem item[STAGES];
    int last[STAGES];                  // 1: the task's last item, 2: no more tasks
    int pub[PUBS][2];                  // tiles to announce (-1: none), -2 first: the end
    unsigned long long full[STAGES], empty[STAGES], pub_full[PUBS], pub_empty[PUBS];
    int abort;
};
static_assert(sizeof(Smem) <= 227 * 1024, "shared memory of a CTA");

__device__ __forceinline__ unsigned sa(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(unsigned long long *b, unsigned n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sa(b)), "r"(n) : "memory");
}
__device__ __forceinline__ bool bar_try(unsigned long long *b, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(sa(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bar_arrive(unsigned long long *b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sa(b)) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned long long *b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sa(b)), "r"(bytes) : "memory");
}
// Bounded wait; false when it gave up or the CTA's abort flag is up.
__device__ __forceinline__ bool bar_wait(unsigned long long *b, unsigned parity, volatile int *abort) {
    for (unsigned i = 0;; i++) {
        if (bar_try(b, parity)) return true;
        if ((i & 63) == 63 && *abort) return false;
        if (i > POLL_LIMIT) {
            *abort = 1;
            return false;
        }
    }
}
// Untiled bulk copy; both addresses and the size are multiples of 16 bytes.
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sa(dst)),
                 "l"(src), "r"(bytes), "r"(sa(bar))
                 : "memory");
}
// orders the generic-proxy writes that the flags waited for announced before
// this thread's next bulk copies
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned *p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Stops every CTA at its next wait and reports the timeout.
__device__ __forceinline__ void give_up(unsigned *ctl_abort, unsigned long long *flags) {
    atomicExch(ctl_abort, 1u);
    atomicOr(flags, FLAG_LOOKBACK_TIMEOUT);
}
// Bounded wait for *f == epoch; false when it gave up (every CTA then stops) or
// another CTA's did.
__device__ bool poll(const unsigned *f, unsigned epoch, unsigned *ctl_abort, unsigned long long *flags) {
    for (unsigned i = 0;; i++) {
        if (ld_acquire(f) == epoch) return true;
        if ((i & 63) == 63 && *(volatile unsigned *)ctl_abort) return false;
        if (i > POLL_LIMIT) {
            give_up(ctl_abort, flags);
            return false;
        }
    }
}
// A column's solution, or z, that is not formed yet: a NaN (a value that happens to
// carry its bits is written as the canonical NaN), so that the values themselves are
// the flag and a step of a triangular solve is one trip through L2.
constexpr unsigned long long EMPTY = 0xFFFFFFFFFFFFFFFFull;
__device__ __forceinline__ unsigned long long ld_relaxed64(const double *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_value(double *p, double x) {
    unsigned long long v = (unsigned long long)__double_as_longlong(x);
    if (v == EMPTY) v = 0x7FF8000000000000ull;
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Bounded wait until v[0], v[STEP], ..., v[(N - 1) STEP] are formed, all lanes of a warp alike.
template <int N, int STEP>
__device__ bool poll_values(const double *v, double (&x)[N], unsigned *ctl_abort, unsigned long long *flags) {
    for (unsigned i = 0;; i++) {
        bool ready = true;
#pragma unroll
        for (int k = 0; k < N; k++) {
            const unsigned long long b = ld_relaxed64(v + STEP * k);
            x[k] = __longlong_as_double((long long)b);
            ready &= b != EMPTY;
        }
        if (__all_sync(0xffffffffu, ready)) return true;
        if ((i & 63) == 63 && __any_sync(0xffffffffu, *(volatile unsigned *)ctl_abort)) return false;
        if (i > POLL_LIMIT) {
            give_up(ctl_abort, flags);
            return false;
        }
    }
}
// barrier of the first N threads, and the same with a vote
template <int N = WORK>
__device__ __forceinline__ void sync_work() { asm volatile("barrier.cta.sync 1, %0;" ::"n"(N) : "memory"); }
template <int N = WORK>
__device__ __forceinline__ bool all_work(bool p) {
    unsigned r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, 2, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((unsigned)p), "n"(N)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// An 8 x 8 accumulator block (lane 4r + q holds columns 2q, 2q + 1 of row r) to
// and from its stored order (lane 4r + q holds columns q, q + 4), one 16-byte
// access a lane: lanes q and q ^ 2 swap one value.
__device__ __forceinline__ double2 to_stored(const double (&c)[2], int lane) {
    const bool low = (lane & 3) < 2;
    const double got = __shfl_xor_sync(0xffffffffu, low ? c[1] : c[0], 2);
    return low ? make_double2(c[0], got) : make_double2(got, c[1]);
}
__device__ __forceinline__ int stored_lane(int lane) {
    const int q = lane & 3;  // q = 0, 1 store columns 0, 2 (and 4, 6); q = 2, 3 store 1, 3 (and 5, 7)
    return (lane & ~3) + (q < 2 ? 2 * q : 2 * q - 3);
}
__device__ __forceinline__ void store_block(double *blk, const double (&c)[2], int lane) {
    const double2 v = to_stored(c, lane);
    *reinterpret_cast<double2 *>(blk + 2 * stored_lane(lane)) = v;
}
__device__ __forceinline__ void load_block(const double *blk, double (&c)[2], int lane) {
    const double2 v = *reinterpret_cast<const double2 *>(blk + 2 * stored_lane(lane));
    const bool low = (lane & 3) < 2;
    const double got = __shfl_xor_sync(0xffffffffu, low ? v.y : v.x, 2);
    c[0] = low ? v.x : got;
    c[1] = low ? got : v.y;
}
// position in a tile of 56 rows (the same order as nd_at)
__device__ __forceinline__ int at56(int r, int c) {
    return (c >> 3) * 448 + (r >> 3) * 64 + ((r & 7) * 4 + (c & 3)) * 2 + ((c >> 2) & 1);
}
__device__ __forceinline__ double2 frag(const double *blk, int lane) {
    return *reinterpret_cast<const double2 *>(blk + 2 * lane);
}

// A warp's 8 x 8 blocks of a tile: rows h, h + 4 (h = warp / 4) and two columns,
// {q, q + 4} or, for odd h, {3 - q, 7 - q} (q = warp % 4, the SM quarter it runs
// on), so that every quarter gets its share of a tile's leading rows and columns
// (a part's last tile is rarely full) and of a triangular product.
struct TileBlocks {
    int h, c0;
    __device__ __forceinline__ int row(int i) const { return h + 4 * i; }
    __device__ __forceinline__ int col(int j) const { return c0 + 4 * j; }
    __device__ __forceinline__ int at(int i, int j) const { return col(j) * 512 + row(i) * 64; }
};

// One block column k of acc += A B^T for NI of the warp's rows and NJ of its
// columns (J0 on), B scaled by d[].  No branches between the products: mma.sync
// under a branch the compiler cannot prove uniform costs it a re-convergence.
template <bool SCALE, int NI, int J0, int NJ>
__device__ __forceinline__ void gemm_step(double (&acc)[2][2][2], const double *A, const double *B, const double *d,
                                          int k, const TileBlocks &tb, int lane) {
    double2 a[NI], b[2];
#pragma unroll
    for (int i = 0; i < NI; i++) a[i] = frag(A + k * 512 + tb.row(i) * 64, lane);
#pragma unroll
    for (int j = J0; j < J0 + NJ; j++) b[j] = frag(B + k * 512 + tb.col(j) * 64, lane);
    if (SCALE) {
        const double d0 = d[8 * k + (lane & 3)], d1 = d[8 * k + 4 + (lane & 3)];
#pragma unroll
        for (int j = J0; j < J0 + NJ; j++) {
            b[j].x *= d0;
            b[j].y *= d1;
        }
    }
#pragma unroll
    for (int i = 0; i < NI; i++)
#pragma unroll
        for (int j = J0; j < J0 + NJ; j++) dmma(acc[i][j], a[i].x, b[j].x);
#pragma unroll
    for (int i = 0; i < NI; i++)
#pragma unroll
        for (int j = J0; j < J0 + NJ; j++) dmma(acc[i][j], a[i].y, b[j].y);
}
template <bool SCALE, int NI>
__device__ __forceinline__ void gemm_rows(double (&acc)[2][2][2], const double *A, const double *B, const double *d,
                                          int kb, bool two, const TileBlocks &tb, int lane) {
    if (SCALE) {
        if (two) {
#pragma unroll 1
            for (int k = 0; k < kb; k++) gemm_step<SCALE, NI, 0, 2>(acc, A, B, d, k, tb, lane);
        } else {
#pragma unroll 1
            for (int k = 0; k < kb; k++) gemm_step<SCALE, NI, 0, 1>(acc, A, B, d, k, tb, lane);
        }
    } else {
        // B lower triangular: block column k meets its block rows from k on
        const int k0 = min(kb, tb.col(0) + 1), k1 = min(kb, tb.col(1) + 1);
        if (two) {
#pragma unroll 1
            for (int k = 0; k < k0; k++) gemm_step<SCALE, NI, 0, 2>(acc, A, B, d, k, tb, lane);
#pragma unroll 1
            for (int k = k0; k < k1; k++) gemm_step<SCALE, NI, 1, 1>(acc, A, B, d, k, tb, lane);
        } else {
#pragma unroll 1
            for (int k = 0; k < k0; k++) gemm_step<SCALE, NI, 0, 1>(acc, A, B, d, k, tb, lane);
        }
    }
}
// acc += A B^T over kb blocks of 8 columns, for the tile's first mb x nb blocks.
// SCALE: B's columns scaled by d[]; else B is lower triangular.
template <bool SCALE>
__device__ __forceinline__ void gemm_tile(double (&acc)[2][2][2], const double *A, const double *B, const double *d,
                                          int kb, int mb, int nb, const TileBlocks &tb, int lane) {
    const bool two = tb.col(1) < nb;
    if (tb.col(0) >= nb || tb.row(0) >= mb) return;
    if (tb.row(1) < mb) gemm_rows<SCALE, 2>(acc, A, B, d, kb, two, tb, lane);
    else gemm_rows<SCALE, 1>(acc, A, B, d, kb, two, tb, lane);
}

// The 36 lower 8 x 8 blocks of a diagonal tile over 16 warps: the first to warp
// 0, which starts the factorization with it, up to three neighbours of a row to
// each of the others.
struct DiagBlocks {
    int row, c0, n;
    __device__ __forceinline__ int at(int i) const { return (c0 + i) * 512 + row * 64; }
};
__device__ __forceinline__ DiagBlocks diag_blocks(int warp) {
    // hexadecimal digit w (from the right): warp w's row, first column, blocks
    constexpr unsigned long long ROW = 0x0123344556667770ull, COL = 0x0002030305306300ull, NUM = 0x0232223332232331ull;
    return DiagBlocks{(int)(ROW >> 4 * warp & 15), (int)(COL >> 4 * warp & 15), (int)(NUM >> 4 * warp & 15)};
}
template <int N>
__device__ __forceinline__ void gemm_diag_n(double (&acc)[3][2], const double *A, const double *d, int kb,
                                            const DiagBlocks &db, int lane) {
    double odd[N][2];
#pragma unroll
    for (int i = 0; i < N; i++) odd[i][0] = odd[i][1] = 0.0;
#pragma unroll 2
    for (int k = 0; k < kb; k++) {
        double2 a = frag(A + k * 512 + db.row * 64, lane), b[N];
        a.x *= d[8 * k + (lane & 3)];
        a.y *= d[8 * k + 4 + (lane & 3)];
#pragma unroll
        for (int i = 0; i < N; i++) b[i] = frag(A + k * 512 + (db.c0 + i) * 64, lane);
#pragma unroll
        for (int i = 0; i < N; i++) {
            dmma(acc[i], a.x, b[i].x);
            dmma(odd[i], a.y, b[i].y);
        }
    }
#pragma unroll
    for (int i = 0; i < N; i++) {
        acc[i][0] += odd[i][0];
        acc[i][1] += odd[i][1];
    }
}
// acc += A D A^T on the lower blocks, for the tile's first mb block rows.
__device__ __forceinline__ void gemm_diag(double (&acc)[3][2], const double *A, const double *d, int kb, int mb,
                                          const DiagBlocks &db, int lane) {
    if (db.row >= mb) return;
    if (db.n == 3) gemm_diag_n<3>(acc, A, d, kb, db, lane);
    else if (db.n == 2) gemm_diag_n<2>(acc, A, d, kb, db, lane);
    else if (db.n == 1) gemm_diag_n<1>(acc, A, d, kb, db, lane);
}

// Row block w of A times v (first kb blocks of 8 columns): lane's partial sum
// for row 8w + lane / 4.
__device__ __forceinline__ double row_dot(const double *A, const double *v, int kb, int w, int lane) {
    double s0 = 0.0, s1 = 0.0;
#pragma unroll 2
    for (int k = 0; k < kb; k++) {
        const double2 a = frag(A + k * 512 + w * 64, lane);
        s0 = fma(a.x, v[8 * k + (lane & 3)], s0);
        s1 = fma(a.y, v[8 * k + 4 + (lane & 3)], s1);
    }
    return s0 + s1;
}
__device__ __forceinline__ double sum_quad(double s) {
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    return s;
}

// L D L^T of the 8 x 8 diagonal block s of sm.c in one warp, and the inverse of
// its L: lane 4r + q holds columns q and q + 4 of row r, of the whole symmetric
// block, so a pivot row is at hand in its own lanes' registers.  Two pivots a
// step through the inverse of their 2 x 2 block P = [p g; g c], so the chain
// holds one reciprocal per two pivots: row r's multipliers are (a_rk, a_r,k+1)
// P^-1.  What turns the blocks into single pivots comes after the last pair.
__device__ __forceinline__ void factor8(Smem &sm, int s, int lane, unsigned long long *flags) {
    const unsigned FULL = 0xffffffffu;
    const int r = lane >> 2, q = lane & 3;
    const double *blk = sm.c + s * 512 + s * 64;
    double a[2], m[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int c = q + 4 * i;
        a[i] = blk[nd_at(max(r, c), min(r, c))];
        m[i] = c == r ? 1.0 : 0.0;
    }
    double pr = 1.0, gr = 0.0, cr = 1.0;  // the 2 x 2 block of this row's pair
    bool sound = true;
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
        const int i = k >> 2, q0 = k & 3;
        const double p = __shfl_sync(FULL, a[i], 4 * k + q0);
        const double g = __shfl_sync(FULL, a[i], 4 * k + 4 + q0);
        const double c = __shfl_sync(FULL, a[i], 4 * k + 4 + q0 + 1);
        if ((r & 6) == k) {
            pr = p;
            gr = g;
            cr = c;
        }
        if (k == 6) break;  // the last rows are done
        const double u = __shfl_sync(FULL, a[i], (lane & ~3) | q0);
        const double v = __shfl_sync(FULL, a[i], (lane & ~3) | (q0 + 1));
        const double det = fma(p, c, -(g * g));
        sound &= invertible(det);
        double rd = reciprocal(det);
        if (r <= k + 1) rd = 0.0;
        const double w0 = fma(g, v, -(c * u)) * rd, w1 = fma(g, u, -(p * v)) * rd;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            if (4 * j + 3 > k + 1) {  // some lane's column is past the pivots
                const double x0 = __shfl_sync(FULL, a[j], 4 * k + q), x1 = __shfl_sync(FULL, a[j], 4 * k + 4 + q);
                a[j] = fma(w1, x1, fma(w0, x0, a[j]));
            }
            if (4 * j <= k + 1) {
                const double x0 = __shfl_sync(FULL, m[j], 4 * k + q), x1 = __shfl_sync(FULL, m[j], 4 * k + 4 + q);
                m[j] = fma(w1, x1, fma(w0, x0, m[j]));
            }
        }
    }
    // within each pair: L_k+1,k = g / p, the second pivot c - g^2 / p
    const double l = gr * reciprocal(pr);
    double dr = pr;
    {
        const double m0 = __shfl_sync(FULL, m[0], lane & ~4), m1 = __shfl_sync(FULL, m[1], lane & ~4);
        if (r & 1) {
            dr = fma(-l, gr, cr);
            m[0] = fma(-l, m0, m[0]);
            m[1] = fma(-l, m1, m[1]);
        }
    }
    // pr is the pivot of the pair's first row
    if (!sound || !invertible(dr)) atomicOr(flags, FLAG_SINGULAR);
    if (q > r) m[0] = 0.0;
    if (q + 4 > r) m[1] = 0.0;
    *reinterpret_cast<double2 *>(sm.inv + s * 512 + s * 64 + 2 * lane) = make_double2(m[0], m[1]);
    if (s < 7) {
        sm.invt[at56(8 * s + q, 8 * s + r)] = m[0];
        sm.invt[at56(8 * s + q + 4, 8 * s + r)] = m[1];
    }
    if (q == 0) {
        sm.d[8 * s + r] = dr;
        sm.dinv[8 * s + r] = reciprocal(dr);
    }
}

// Row block rb of L's block column s: A Linv8^T D^-1.
__device__ __forceinline__ void panel_block(Smem &sm, int s, int rb, int lane) {
    double *p = sm.c + s * 512 + rb * 64;
    const double2 a = frag(p, lane), b = frag(sm.inv + s * 512 + s * 64, lane);
    double w[2] = {0.0, 0.0}, w1[2] = {0.0, 0.0};
    dmma(w, a.x, b.x);
    dmma(w1, a.y, b.y);
    w[0] = (w[0] + w1[0]) * sm.dinv[8 * s + 2 * (lane & 3)];
    w[1] = (w[1] + w1[1]) * sm.dinv[8 * s + 2 * (lane & 3) + 1];
    __syncwarp();
    store_block(p, w, lane);
}

// Blocks u0, u0 + 15, ... (N of them, below `count`) of the lower triangle that
// starts at block `first` -= L D L^T of block column s; a block's number is
// its row's first, i (i + 1) / 2, plus its column.  All loads before the products.
template <int N>
__device__ __forceinline__ void trail_blocks(Smem &sm, int s, int first, int u0, int count, int lane) {
    double acc[N][2], acc2[N][2];
    double2 x[N], y[N];
    int at[N];
    const double d0 = -sm.d[8 * s + (lane & 3)], d1 = -sm.d[8 * s + 4 + (lane & 3)];
#pragma unroll
    for (int n = 0; n < N; n++) {
        const int u = u0 + 15 * n < count ? u0 + 15 * n : 0;
        const int i = (u >= 1) + (u >= 3) + (u >= 6) + (u >= 10) + (u >= 15) + (u >= 21), o = u - i * (i + 1) / 2;
        at[n] = (first + o) * 512 + (first + i) * 64;
        x[n] = frag(sm.c + s * 512 + (first + i) * 64, lane);
        y[n] = frag(sm.c + s * 512 + (first + o) * 64, lane);
        load_block(sm.c + at[n], acc[n], lane);
        acc2[n][0] = acc2[n][1] = 0.0;
    }
#pragma unroll
    for (int n = 0; n < N; n++) {
        dmma(acc[n], x[n].x, y[n].x * d0);
        dmma(acc2[n], x[n].y, y[n].y * d1);
    }
#pragma unroll
    for (int n = 0; n < N; n++) {
        acc[n][0] += acc2[n][0];
        acc[n][1] += acc2[n][1];
        const double2 v = to_stored(acc[n], lane);
        if (u0 + 15 * n < count) *reinterpret_cast<double2 *>(sm.c + at[n] + 2 * stored_lane(lane)) = v;
    }
}

// L D L^T of the 64 x 64 block in sm.c (lower part), warps 0-15: its inverse
// (sm.inv, and in global memory at g), sm.d, sm.dinv, and z = L^-1 r (at gz; D and
// 1/D beside it; gx is emptied; `release` is arrived at after the first step).  Eight columns a
// step.  Warp 0 runs the chain: it factors the 8 x 8 block, then forms the L rows
// and updates the block that the next step factors, while the other warps do the
// step's remaining rows and blocks and the inverse's next block row.  Latency-
// bound, 2,000 clocks a step: the 8 x 8 block 1,150, the L rows 190, the update
// 190, the rest barriers and the other warps' products (8 warps: 2,500 clocks).
__device__ void factor64(Smem &sm, int warp, int lane, double *g, double *gz, double *gx, unsigned long long *release,
                         unsigned long long *flags) {
    auto z_rows = [&](int w) {
        const double zr = sum_quad(row_dot(sm.inv, sm.r, 8, w, lane));
        if ((lane & 3) == 0) gz[8 * w + (lane >> 2)] = zr;
    };
#pragma unroll 1
    for (int s = 0; s < 8; s++) {
        if (warp == 0) {
            factor8(sm, s, lane, flags);
        } else if (s > 0) {
            // the rest of step s - 1's update, then tt = (L_s,0..s-1 Linv_0..s-1)^T
            const int n = 8 - s, count = n * (n + 1) / 2;  // block 0 is warp 0's
            if (count > 16) trail_blocks<2>(sm, s - 1, s, warp, count, lane);
            else if (warp < count) trail_blocks<1>(sm, s - 1, s, warp, count, lane);
            if (warp == 8) z_rows(s - 1);  // which has no part in the next
            if (15 - warp < s) {
                const int cb = 15 - warp;
                double acc[2] = {0.0, 0.0}, acc2[2] = {0.0, 0.0};
#pragma unroll 1
                for (int k = cb; k < s; k++) {
                    const double2 x = frag(sm.c + k * 512 + s * 64, lane);
                    const double2 y = frag(sm.invt + k * 448 + cb * 64, lane);
                    dmma(acc, x.x, y.x);
                    dmma(acc2, x.y, y.y);
                }
#pragma unroll
                for (int e = 0; e < 2; e++) sm.tt[at56(8 * cb + 2 * (lane & 3) + e, lane >> 2)] = acc[e] + acc2[e];
            }
        }
        sync_work();
        if (s == 0 && release && lane == 0) bar_arrive(release);
        if (warp == 0 && s < 7) {
            panel_block(sm, s, s + 1, lane);
            asm volatile("barrier.cta.arrive 3, %0;" ::"n"(WORK) : "memory");
            __syncwarp();
            trail_blocks<1>(sm, s, s + 1, 0, 1, lane);
            __syncwarp();
            continue;
        }
        if (warp > 0 && warp + s + 1 < 8) panel_block(sm, s, warp + s + 1, lane);
        // the inverse's block row s: -Linv8 (L_s Linv)
        if (warp == 1)
            *reinterpret_cast<double2 *>(g + s * 512 + s * 64 + 2 * lane) = frag(sm.inv + s * 512 + s * 64, lane);
        if (const int cb = 15 - warp; cb < s) {
            double acc[2] = {0.0, 0.0}, acc2[2] = {0.0, 0.0};
            const double2 x = frag(sm.inv + s * 512 + s * 64, lane), y = frag(sm.tt + cb * 64, lane);
            dmma(acc, -x.x, y.x);
            dmma(acc2, -x.y, y.y);
            acc[0] += acc2[0];
            acc[1] += acc2[1];
            store_block(sm.inv + cb * 512 + s * 64, acc, lane);
            store_block(g + cb * 512 + s * 64, acc, lane);
            if (s == 7) {
                const double v = sum_quad(fma(acc[0], sm.r[8 * cb + 2 * (lane & 3)], acc[1] * sm.r[8 * cb + 2 * (lane & 3) + 1]));
                if ((lane & 3) == 0) sm.z7[cb][lane >> 2] = v;
            }
            if (s < 7) {
#pragma unroll
                for (int e = 0; e < 2; e++) sm.invt[at56(8 * cb + 2 * (lane & 3) + e, 8 * s + (lane >> 2))] = acc[e];
            }
        }
        if (s < 7) asm volatile("barrier.cta.sync 3, %0;" ::"n"(WORK) : "memory");
    }
    if (warp == 0) {
        const double2 x = frag(sm.inv + 7 * 512 + 7 * 64, lane);
        const double v = sum_quad(fma(x.x, sm.r[56 + (lane & 3)], x.y * sm.r[60 + (lane & 3)]));
        if ((lane & 3) == 0) sm.z7[7][lane >> 2] = v;
    }
    sync_work();
    if (warp == 0) {
        if (lane < 8) {
            double v = 0.0;
#pragma unroll
            for (int k = 0; k < 8; k++) v += sm.z7[k][lane];
            gz[56 + lane] = v;
        }
    } else if (warp < 5) {
        const int i = 32 * (warp - 1) + lane;
        gz[T + i] = i < T ? sm.d[i] : sm.dinv[i - T];
    } else if (warp < 7) {
        gx[32 * (warp - 5) + lane] = __longlong_as_double((long long)EMPTY);
    }
}

__global__ void __launch_bounds__(THREADS, 1) k_nd_factor(NdArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    if (t == 0) {
        for (int s = 0; s < STAGES; s++) {
            bar_init(&sm.full[s], 1);
            bar_init(&sm.empty[s], WORK / 32);
        }
        for (int s = 0; s < PUBS; s++) {
            bar_init(&sm.pub_full[s], WORK / 32);
            bar_init(&sm.pub_empty[s], 1);
        }
        sm.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == WORK / 32 + 1) {
        // publisher: releases tiles' flags once all warps have written them, so that only
        // this warp waits for the stores
        if (lane) return;
        for (unsigned it = 0;; it++) {
            const int s = it % PUBS;
            if (!bar_wait(&sm.pub_full[s], (it / PUBS) & 1, &sm.abort)) return;
            const int p = sm.pub[s][0], q = sm.pub[s][1];
            if (p == -2) return;
            st_release(a.flag + p, a.epoch);
            if (q >= 0) st_release(a.flag + q, a.epoch);
            bar_arrive(&sm.pub_empty[s]);
        }
    }
    if (warp == WORK / 32) {
        if (lane) return;
        unsigned it = 0;
        bool ok = true;
        while (ok) {
            const unsigned tk = atomicAdd(a.ctl, 1u);
            const bool end = tk >= (unsigned)a.ntask;
            NdTask task{};
            if (!end) task = a.task[tk];
            else task.item1 = 1;
            for (int q = task.item0; q < task.item1; q++, it++) {
                const int s = it % STAGES;
                if (it >= STAGES && !bar_wait(&sm.empty[s], (it / STAGES - 1) & 1, &sm.abort)) {
                    ok = false;
                    break;
                }
                NdItem im{-1, ND_BEGIN, 0, 0};
                if (!end) im = a.item[q];
                if (im.a >= 0 && !(poll(a.flag + im.a, a.epoch, a.ctl + 1, a.flags) &&
                                   (im.b < 0 || poll(a.flag + im.b, a.epoch, a.ctl + 1, a.flags)))) {
                    ok = false;
                    break;
                }
                sm.task[s] = task;
                sm.item[s] = im;
                sm.last[s] = end ? 2 : q + 1 == task.item1;
                if (im.a < 0) {
                    bar_arrive(&sm.full[s]);
                    continue;
                }
                const unsigned bytes = (unsigned)im.kblocks * 512 * sizeof(double);
                fence_async();
                bar_expect(&sm.full[s], bytes * (im.b >= 0 ? 2 : 1) + ZD * (unsigned)sizeof(double));
                bulk_copy(sm.stage[s][0], a.tile + (size_t)im.a * TT, bytes, &sm.full[s]);
                if (im.b >= 0) bulk_copy(sm.stage[s][1], a.tile + (size_t)im.b * TT, bytes, &sm.full[s]);
                bulk_copy(sm.zd[s], a.zd + (size_t)im.col * ZD, ZD * sizeof(double), &sm.full[s]);
            }
            if (end) break;
        }
        if (!ok) {
            // stop the other warps, and let this CTA's copies land before it ends
            sm.abort = 1;
            for (unsigned j = it > STAGES ? it - STAGES : 0; j < it; j++)
                for (unsigned i = 0; i < POLL_LIMIT && !bar_try(&sm.full[j % STAGES], (j / STAGES) & 1); i++) {}
        }
        return;
    }

    TileBlocks tb;
    tb.h = warp >> 2;
    tb.c0 = tb.h & 1 ? 3 - (warp & 3) : warp & 3;
    const DiagBlocks db = diag_blocks(warp);
    const int rw = warp - 8;           // warps 8-15: the row block of the right-hand side they sum
    unsigned pubs = 0;
    // hands tiles p and q (-1: none) to the publisher; every work warp calls it after its writes
    auto publish = [&](int p, int q) {
        const int s = pubs % PUBS;
        bool ok = pubs < PUBS || bar_wait(&sm.pub_empty[s], (pubs / PUBS - 1) & 1, &sm.abort);
        if (t == 0 && ok) {
            sm.pub[s][0] = p;
            sm.pub[s][1] = q;
        }
        __syncwarp();
        if (lane == 0) bar_arrive(&sm.pub_full[s]);
        pubs++;
    };
    double accx[2][2][2], accd[3][2], rs = 0.0;
    for (unsigned it = 0;; it++) {
        const int s = it % STAGES;
        if (!all_work(bar_wait(&sm.full[s], (it / STAGES) & 1, &sm.abort))) {
            if (t == 0) give_up(a.ctl + 1, a.flags);
            return;
        }
        if (sm.last[s] == 2) return publish(-2, -1);
        const NdItem im = sm.item[s];
        const NdTask &task = sm.task[s];
        const int J = task.col, out = task.tile, xout = task.xtile, partial = task.partial;
        const bool diag = task.row == J, last = sm.last[s] != 0;
        // blocks of 8 rows in use: of the tile's rows, its columns, and the fused tile's columns
        const int mb = task.rblocks, nb = task.cblocks, pb = task.pblocks;
        const double *A = sm.stage[s][0], *B = sm.stage[s][1], *z = sm.zd[s], *D = z + T, *Di = z + 2 * T;
        if (im.b == ND_BEGIN) {
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) accx[i][j][0] = accx[i][j][1] = 0.0;
#pragma unroll
            for (int i = 0; i < 3; i++) accd[i][0] = accd[i][1] = 0.0;
            rs = 0.0;
            if (!partial) {
                // J's entries, now: the loads would be on the chain later.  They go through sm.c
                // (the off-diagonal tile) and sm.inv (the diagonal one) into the sums.
                const int x0 = diag ? task.xent0 : task.ent0, x1 = diag ? task.xent1 : task.ent1;
                const bool entries = x1 > x0;
#pragma unroll 1
                for (int i = t; i < TT / 2; i += WORK) {
                    if (entries) reinterpret_cast<double2 *>(sm.c)[i] = make_double2(0.0, 0.0);
                    if (diag) reinterpret_cast<double2 *>(sm.inv)[i] = make_double2(0.0, 0.0);
                }
                if (entries || diag) sync_work();
#pragma unroll 1
                for (int e = x0 + t; e < x1; e += WORK) sm.c[a.ent_at[e]] = a.kval[a.ent_src[e]];
                if (diag) {
#pragma unroll 1
                    for (int e = task.ent0 + t; e < task.ent1; e += WORK) sm.inv[a.ent_at[e]] = a.kval[a.ent_src[e]];
                    sync_work();
                    if (t < T) {
                        const int u = a.perm[J * T + t];
                        sm.inv[nd_at(t, t)] = u >= 0 ? sm.inv[nd_at(t, t)] - a.FP[u] : 1.0;
                        sm.r[t] = u >= 0 ? a.b[u] : 0.0;
                    }
                }
                if (entries || diag) sync_work();
                if (entries) {
#pragma unroll
                    for (int i = 0; i < 2; i++)
#pragma unroll
                        for (int j = 0; j < 2; j++) {
                            load_block(sm.c + tb.at(i, j), accx[i][j], lane);
                            accx[i][j][0] = -accx[i][j][0];
                            accx[i][j][1] = -accx[i][j][1];
                        }
                }
                if (diag) {
#pragma unroll
                    for (int i = 0; i < 3; i++)
                        if (i < db.n) {
                            load_block(sm.inv + db.at(i), accd[i], lane);
                            accd[i][0] = -accd[i][0];
                            accd[i][1] = -accd[i][1];
                        }
                }
            }
        } else if (im.b == ND_ADD || im.b == ND_ADDX) {
            if (diag && im.b == ND_ADD) {
#pragma unroll
                for (int i = 0; i < 3; i++)
                    if (i < db.n) {
                        double v[2];
                        load_block(A + db.at(i), v, lane);
                        accd[i][0] += v[0];
                        accd[i][1] += v[1];
                    }
                if (rw >= 0 && (lane & 3) == 0) rs += z[8 * rw + (lane >> 2)];
            } else {
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        double v[2];
                        load_block(A + tb.at(i, j), v, lane);
                        accx[i][j][0] += v[0];
                        accx[i][j][1] += v[1];
                    }
            }
        } else if (im.b != ND_INV) {
            if (im.b >= 0) gemm_tile<true>(accx, A, B, D, im.kblocks, diag ? nb : mb, diag ? pb : nb, tb, lane);
            if (diag) {
                gemm_diag(accd, A, D, im.kblocks, nb, db, lane);
                if (rw >= 0) rs += row_dot(A, z, im.kblocks, rw, lane);
            }
        } else {
            // the tile so far, C = K - products, then L = C Linv^T D^-1
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const double v[2] = {-accx[i][j][0], -accx[i][j][1]};
                    store_block(sm.c + tb.at(i, j), v, lane);
                    accx[i][j][0] = accx[i][j][1] = 0.0;
                }
            sync_work();
            gemm_tile<false>(accx, sm.c, A, nullptr, im.kblocks, diag ? nb : mb, im.kblocks, tb, lane);
            const int to = diag ? xout : out;
            double *g = a.tile + (size_t)to * TT, *l = sm.stage[s][1];  // (no second operand came)
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const int cb = tb.col(j);
                    accx[i][j][0] *= Di[8 * cb + 2 * (lane & 3)];
                    accx[i][j][1] *= Di[8 * cb + 2 * (lane & 3) + 1];
                    if (diag) store_block(l + tb.at(i, j), accx[i][j], lane);
                    store_block(g + tb.at(i, j), accx[i][j], lane);
                }
            publish(to, -1);
            if (diag) {
                // the last products of the diagonal block; warp 0 has the first block's only and goes
                // on to factor it while the others finish theirs
                sync_work();
                gemm_diag(accd, l, D, im.kblocks, nb, db, lane);
#pragma unroll
                for (int i = 0; i < 3; i++)
                    if (i < db.n) {
                        const double v[2] = {-accd[i][0], -accd[i][1]};
                        store_block(sm.c + db.at(i), v, lane);
                    }
                if (rw >= 0) {
                    rs = sum_quad(rs + row_dot(l, z, im.kblocks, rw, lane));
                    if ((lane & 3) == 0) sm.r[8 * rw + (lane >> 2)] -= rs;
                }
            }
        }
        __syncwarp();
        const bool fused = diag && im.b == ND_INV;  // the stage is still read: factor64 releases it
        if (!fused && lane == 0) bar_arrive(&sm.empty[s]);
        if (!last) continue;
        if (partial) {
            // the sums as they are
            if (diag) {
                double *g = a.tile + (size_t)out * TT;
#pragma unroll
                for (int i = 0; i < 3; i++)
                    if (i < db.n) store_block(g + db.at(i), accd[i], lane);
                rs = sum_quad(rs);
                if (rw >= 0 && (lane & 3) == 0) a.zd[(size_t)(a.ncol + out - a.ntile) * ZD + 8 * rw + (lane >> 2)] = rs;
            }
            const int to = diag ? xout : out;
            if (to >= 0) {
                double *g = a.tile + (size_t)to * TT;
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int j = 0; j < 2; j++) store_block(g + tb.at(i, j), accx[i][j], lane);
            }
            publish(out, diag ? to : -1);
            continue;
        }
        if (!diag) continue;
        // the diagonal block: factor, inverse, z = Linv (b - products)
        if (!fused) {
#pragma unroll
            for (int i = 0; i < 3; i++)
                if (i < db.n) {
                    const double v[2] = {-accd[i][0], -accd[i][1]};
                    store_block(sm.c + db.at(i), v, lane);
                }
            rs = sum_quad(rs);
            if (rw >= 0 && (lane & 3) == 0) sm.r[8 * rw + (lane >> 2)] -= rs;
            sync_work();
        }
        factor64(sm, warp, lane, a.tile + (size_t)out * TT, a.zd + (size_t)J * ZD, a.x + (size_t)J * T, fused ? &sm.empty[s] : nullptr,
                 a.flags);
        publish(out, -1);
    }
}

// ---- triangular solves with the stored factor ------------------------------------------

constexpr int SOLVE_STAGES = 6;
constexpr int SOLVE_WORK = 256;           // threads of warps 0-7
constexpr int SOLVE_THREADS = SOLVE_WORK + 32;  // and the producer's warp

struct SolveArgs {
    const int *ptr, *tiles;            // per column: the tiles it takes, in order (null tiles: tile ids ptr + 1 ..)
    const int *other;                  // tile -> the column whose values it multiplies
    const int *diag;                   // column -> its inverse's tile
    const int *perm;
    const double *tile, *b;
    double *zd, *x;                    // z (forward result), x [ncol][64]
    double *y;                         // solution by unknown
    unsigned *ctl;
    unsigned long long *flags;
    int ncol, add;
};

struct SolveSmem {
    double stage[SOLVE_STAGES][TT];
    double v[T];
    int col[SOLVE_STAGES], other[SOLVE_STAGES], last[SOLVE_STAGES];
    unsigned long long full[SOLVE_STAGES], empty[SOLVE_STAGES];
    int abort;
};

// Forward: z_J = Linv_J (b_J - sum_K L_JK z_K).  Backward: x_J = Linv_J^T (D_J^-1
// z_J - sum_I L_IJ^T x_I), which also adds to or sets y.  A column is a task,
// taken by ticket in the elimination order or its reverse; the producer
// streams the column's tiles, which do not depend on the solve, ahead of the
// values the others wait for.  Latency-bound: a chain of columns.  The values
// themselves are polled (no flag and no fence on the way), and what a column's end
// needs besides is read when the column starts: backward 16.6 -> 11.7 us at 567
// unknowns, 58 -> 40 at 8,379, 137 -> 90 at 32,244; forward 128 -> 103.  A launch
// empties what the next one fills: a factor or a forward solve x, a backward
// solve z.
template <bool BACK>
__global__ void __launch_bounds__(SOLVE_THREADS, 1) k_nd_solve(SolveArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SolveSmem &sm = *reinterpret_cast<SolveSmem *>(smem_raw);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    if (t == 0) {
        for (int s = 0; s < SOLVE_STAGES; s++) {
            bar_init(&sm.full[s], 1);
            bar_init(&sm.empty[s], SOLVE_WORK / 32);
        }
        sm.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp == SOLVE_WORK / 32) {
        if (lane) return;
        unsigned it = 0;
        bool ok = true;
        while (ok) {
            const unsigned tk = atomicAdd(a.ctl, 1u);
            const bool end = tk >= (unsigned)a.ncol;
            const int J = end ? -1 : BACK ? a.ncol - 1 - (int)tk : (int)tk;
            const int p0 = end ? 0 : a.ptr[J] + (BACK ? 1 : 0), p1 = end ? 0 : a.ptr[J + 1];
            // the column's tiles, then its inverse; backward the rows nearest the root first
            for (int p = p0; p <= p1; p++, it++) {
                const int s = it % SOLVE_STAGES;
                if (it >= SOLVE_STAGES && !bar_wait(&sm.empty[s], (it / SOLVE_STAGES - 1) & 1, &sm.abort)) {
                    ok = false;
                    break;
                }
                const int tl = end ? -1 : p == p1 ? a.diag[J] : BACK ? p1 - 1 - (p - p0) : a.tiles[p];
                sm.col[s] = J;
                sm.last[s] = p == p1;
                sm.other[s] = tl < 0 ? 0 : a.other[tl];
                if (end) {
                    bar_arrive(&sm.full[s]);
                    break;
                }
                bar_expect(&sm.full[s], TT * sizeof(double));
                bulk_copy(sm.stage[s], a.tile + (size_t)tl * TT, TT * sizeof(double), &sm.full[s]);
            }
            if (end) break;
        }
        if (!ok) {
            sm.abort = 1;
            for (unsigned j = it > SOLVE_STAGES ? it - SOLVE_STAGES : 0; j < it; j++)
                for (unsigned i = 0; i < POLL_LIMIT && !bar_try(&sm.full[j % SOLVE_STAGES], (j / SOLVE_STAGES) & 1); i++) {}
        }
        return;
    }
    // forward: warp w holds rows 8w .. 8w + 7, backward columns
    double s0 = 0.0, s1 = 0.0, rhs0 = 0.0, rhs1 = 0.0;
    int at = -1, u0 = -1, u1 = -1;            // the column under way; its lane's unknowns
    for (unsigned it = 0;; it++) {
        const int s = it % SOLVE_STAGES;
        bool ok = bar_wait(&sm.full[s], (it / SOLVE_STAGES) & 1, &sm.abort);
        const int J = sm.col[s], last = sm.last[s];
        if (ok && J >= 0 && J != at) {
            // what the column's end needs and does not depend on the others
            at = J;
            if (BACK && lane < 4) {
                const double *z = a.zd + (size_t)J * ZD + 8 * warp + lane;
                rhs0 = __ldcg(z) * __ldcg(z + 2 * T);
                rhs1 = __ldcg(z + 4) * __ldcg(z + 2 * T + 4);
                u0 = a.perm[J * T + 8 * warp + lane];
                u1 = a.perm[J * T + 8 * warp + lane + 4];
            }
            if (!BACK && (lane & 3) == 0) {
                u0 = a.perm[J * T + 8 * warp + (lane >> 2)];
                rhs0 = u0 >= 0 ? a.b[u0] : 0.0;
            }
        }
        if (ok && J >= 0 && !last) {
            const int o = sm.other[s];
            double x[BACK ? 8 : 16];
            if constexpr (BACK) ok = poll_values<8, 8>(a.x + (size_t)o * T + (lane >> 2), x, a.ctl + 1, a.flags);
            else ok = poll_values<16, 4>(a.zd + (size_t)o * ZD + (lane & 3), x, a.ctl + 1, a.flags);
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const double2 l = frag(sm.stage[s] + (BACK ? warp * 512 + k * 64 : k * 512 + warp * 64), lane);
                if constexpr (BACK) {
                    s0 = fma(l.x, x[k], s0);
                    s1 = fma(l.y, x[k], s1);
                } else {
                    s0 = fma(l.x, x[2 * k], s0);
                    s1 = fma(l.y, x[2 * k + 1], s1);
                }
            }
            __syncwarp();
            if (lane == 0) bar_arrive(&sm.empty[s]);
            if (ok) continue;
            sm.abort = 1;
        }
        if (!all_work<SOLVE_WORK>(ok)) {
            if (t == 0) give_up(a.ctl + 1, a.flags);
            return;
        }
        if (J < 0) return;
        // all of the column's tiles are in: the right-hand side, then the inverse
        if (BACK) {
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                s0 += __shfl_xor_sync(0xffffffffu, s0, o);
                s1 += __shfl_xor_sync(0xffffffffu, s1, o);
            }
            if (lane < 4) {
                sm.v[8 * warp + lane] = rhs0 - s0;
                sm.v[8 * warp + lane + 4] = rhs1 - s1;
            }
        } else {
            s0 = sum_quad(s0 + s1);
            if ((lane & 3) == 0) {
                sm.v[8 * warp + (lane >> 2)] = u0 >= 0 ? rhs0 - s0 : 0.0;
            }
        }
        sync_work<SOLVE_WORK>();
        if (BACK) {
            s0 = s1 = 0.0;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const double2 l = frag(sm.stage[s] + warp * 512 + k * 64, lane);
                s0 = fma(l.x, sm.v[8 * k + (lane >> 2)], s0);
                s1 = fma(l.y, sm.v[8 * k + (lane >> 2)], s1);
            }
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                s0 += __shfl_xor_sync(0xffffffffu, s0, o);
                s1 += __shfl_xor_sync(0xffffffffu, s1, o);
            }
            if (lane < 4) {
                st_value(a.x + (size_t)J * T + 8 * warp + lane, s0);
                st_value(a.x + (size_t)J * T + 8 * warp + lane + 4, s1);
                double *z = a.zd + (size_t)J * ZD + 8 * warp + lane;  // for the next forward solve
                z[0] = z[4] = __longlong_as_double((long long)EMPTY);
                if (u0 >= 0) a.y[u0] = a.add ? a.y[u0] + s0 : s0;
                if (u1 >= 0) a.y[u1] = a.add ? a.y[u1] + s1 : s1;
            }
        } else {
            const double zr = sum_quad(row_dot(sm.stage[s], sm.v, warp + 1, warp, lane));
            if ((lane & 3) == 0) {
                st_value(a.zd + (size_t)J * ZD + 8 * warp + (lane >> 2), zr);
                a.x[(size_t)J * T + 8 * warp + (lane >> 2)] = __longlong_as_double((long long)EMPTY);
            }
        }
        s0 = s1 = 0.0;
        sync_work<SOLVE_WORK>();
        if (lane == 0) bar_arrive(&sm.empty[s]);
    }
}

struct NdState {
    bool planned = false;              // the plan exists
    bool usable = false;               // and is on the device, with the factor's memory
    NdPlan plan;                       // (its long host lists are dropped once on the device)
    void *blob = nullptr;              // the plan's arrays
    const NdTask *task = nullptr;
    const NdItem *item = nullptr;
    const int *perm = nullptr, *ent_src = nullptr, *tile_ptr = nullptr, *tile_row = nullptr,
              *tile_col = nullptr, *row_ptr = nullptr, *row_tile = nullptr;
    const unsigned short *ent_at = nullptr;
    int ntask = 0;
    double *tile = nullptr, *zd = nullptr, *x = nullptr;
    unsigned *flag = nullptr;          // tiles (and scratch ones)
    size_t words = 0;
    unsigned *ctl = nullptr;           // [3][2] ticket and abort word of a factor, a forward and a backward launch
    unsigned epoch = 0;
};

NdState *state_of(mp_ctx *ctx) { return static_cast<NdState *>(ctx->nd); }

}  // namespace

static void nd_release(NdState *s) {
    void **p[] = {&s->blob, (void **)&s->tile, (void **)&s->zd, (void **)&s->x, (void **)&s->flag, (void **)&s->ctl};
    for (void **q : p) {
        if (*q) cudaFree(*q);
        *q = nullptr;
    }
    s->usable = false;
}

void nd_free(mp_ctx *ctx) {
    NdState *s = state_of(ctx);
    if (!s) return;
    nd_release(s);
    delete s;
    ctx->nd = nullptr;
}

// Which factorization is the faster one, by estimates measured on a B200 (us):
// a sparse one costs its chain of diagonal blocks and its products over the
// SMs; the dense ones a step per 64 columns and n^3/3 flops.
static bool nd_faster(long long products, int chain, int n, int sms, bool mixed) {
    const double nd = 14.0 * chain + 3.0 * (double)products / sms;
    const double steps = n / 64.0, flops = (double)n * n * n / 3.0;
    const double dense = mixed ? 30.0 * steps + flops / (n >= MP_MIXED_FP16_FROM ? 600e6 : 200e6)
                               : 40.0 * steps + flops / 25e6;
    return nd < dense;
}

// Puts the plan on the device, with the factor's memory (the largest part first).
// Where that cannot be had, the state stays unusable and takes none.
static int nd_place(mp_ctx *ctx, NdState *s) {
    NdPlan &p = s->plan;
    size_t off = 0;
    auto place = [&](size_t bytes) {
        const size_t o = off;
        off = (off + bytes + 255) & ~size_t(255);
        return o;
    };
#define ND_ARRAYS(X) X(task) X(item) X(perm) X(ent_src) X(ent_at) X(tile_ptr) X(tile_row) X(tile_col) X(row_ptr) X(row_tile)
    std::vector<unsigned char> host;
#define X(a) const size_t o_##a = place(p.a.size() * sizeof(p.a[0]));
    ND_ARRAYS(X)
#undef X
    host.resize(off + 256);
#define X(a) if (!p.a.empty()) std::memcpy(host.data() + o_##a, p.a.data(), p.a.size() * sizeof(p.a[0]));
    ND_ARRAYS(X)
#undef X
    s->words = (size_t)p.ntile + p.nscratch;
    if (!allocate_all({{(void **)&s->tile, sizeof(double) * s->words * TT},
                       {&s->blob, host.size()},
                       {(void **)&s->zd, sizeof(double) * (size_t)(p.ncol + p.nscratch) * ZD},
                       {(void **)&s->x, sizeof(double) * (size_t)p.ncol * T},
                       {(void **)&s->flag, sizeof(unsigned) * s->words},
                       {(void **)&s->ctl, sizeof(unsigned) * 8}},
                      device_room, cudaFree))
        return MP_OK;
    MP_CUDA(ctx, upload(ctx, s->blob, host.data(), host.size()));
#define X(a) s->a = reinterpret_cast<decltype(s->a)>(static_cast<unsigned char *>(s->blob) + o_##a);
    ND_ARRAYS(X)
#undef X
#undef ND_ARRAYS
    s->ntask = (int)p.task.size();
    // the blocks above an inverse's diagonal stay zero
    MP_CUDA(ctx, cudaMemsetAsync(s->tile, 0, sizeof(double) * (size_t)p.ntile * TT, ctx->stream));
    MP_CUDA(ctx, cudaMemsetAsync(s->flag, 0, sizeof(unsigned) * s->words, ctx->stream));
    MP_CUDA(ctx, cudaFuncSetAttribute(k_nd_factor, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem)));
    MP_CUDA(ctx, cudaFuncSetAttribute(k_nd_solve<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(SolveSmem)));
    MP_CUDA(ctx, cudaFuncSetAttribute(k_nd_solve<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(SolveSmem)));
    MP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    p.task.clear();
    p.task.shrink_to_fit();
    p.item.clear();
    p.item.shrink_to_fit();
    s->epoch = 0;
    s->usable = true;
    return MP_OK;
}

static int nd_plan_and_place(mp_ctx *ctx, bool mixed, bool *usable) {
    NdState *s = state_of(ctx);
    int rc;
    if (!s) {
        s = new NdState();
        ctx->nd = s;
        const int n = ctx->neq;
        bool fits = false;
        if ((rc = fe_pattern_fits(ctx, &fits))) return rc;
        if (fits && !ctx->csr_ptr.empty()) {
            std::vector<double> pos(3 * (size_t)n, 0.0), npos(3 * (size_t)ctx->n_nodes);
            std::vector<int> ID(ctx->n_nodes);
            MP_CUDA(ctx, cudaMemcpy(npos.data(), ctx->node_pos, sizeof(double) * npos.size(), cudaMemcpyDeviceToHost));
            MP_CUDA(ctx, cudaMemcpy(ID.data(), ctx->ID, sizeof(int) * ID.size(), cudaMemcpyDeviceToHost));
            for (int k = 0; k < ctx->n_nodes; k++)
                if (ID[k] >= 0)
                    for (int d = 0; d < 3; d++) pos[3 * (size_t)ID[k] + d] = npos[3 * (size_t)k + d];
            const double blocks = n / 64.0 + 1;
            const long long most = (long long)(blocks * blocks * blocks / 6 + 100);
            s->planned = nd_build_plan(n, ctx->csr_ptr, ctx->csr_col, ctx->csr_slot, pos, most, s->plan);
        }
    }
    if (!s->planned || !nd_faster(s->plan.products, s->plan.chain, ctx->neq, ctx->sm_count, mixed)) return MP_OK;
    if (!s->usable && (rc = nd_place(ctx, s))) {
        nd_release(s);
        return rc;
    }
    *usable = s->usable;
    return MP_OK;
}

// Builds the plan on the first direct solve after mp_fe_setup, and places it when
// it is first the faster way.  *usable: the sparse factorization applies (K has the
// mesh's pattern and is symmetric), is expected to be faster than the dense one
// and has its memory.  Where the device or the host is too full for it, the dense
// one takes the call and the next call asks again.
int nd_prepare(mp_ctx *ctx, bool mixed, bool *usable) {
    *usable = false;
    try {
        return nd_plan_and_place(ctx, mixed, usable);
    } catch (const std::exception &) {
        nd_free(ctx);
        return MP_OK;
    }
}

static int nd_launch_solve(mp_ctx *ctx, NdState *s, bool back, const double *b, double *y, bool add) {
    const NdPlan &p = s->plan;
    SolveArgs a;
    a.ptr = back ? s->tile_ptr : s->row_ptr;
    a.tiles = s->row_tile;
    a.other = back ? s->tile_row : s->tile_col;
    a.diag = s->tile_ptr;
    a.perm = s->perm;
    a.tile = s->tile;
    a.b = b;
    a.zd = s->zd;
    a.x = s->x;
    a.y = y;
    a.ctl = s->ctl + (back ? 4 : 2);
    a.flags = ctx->counters + C_FLAGS;
    a.ncol = p.ncol;
    a.add = add;
    const int grid = std::min(ctx->sm_count, p.ncol);
    const int mk = kt_begin(ctx, MP_KT_TRSV, 0);
    if (back) k_nd_solve<true><<<grid, SOLVE_THREADS, sizeof(SolveSmem), ctx->stream>>>(a), ++ctx->launches;
    else k_nd_solve<false><<<grid, SOLVE_THREADS, sizeof(SolveSmem), ctx->stream>>>(a), ++ctx->launches;
    kt_end(ctx, mk);
    MP_CUDA(ctx, cudaGetLastError());
    return MP_OK;
}

static int nd_begin(mp_ctx *ctx, NdState *s, bool control_cleared) {
    if (s->epoch >= 0x7ffffff0u) {
        MP_CUDA(ctx, cudaMemsetAsync(s->flag, 0, sizeof(unsigned) * s->words, ctx->stream));
        s->epoch = 0;
    }
    s->epoch++;
    if (!control_cleared) MP_CUDA(ctx, cudaMemsetAsync(s->ctl, 0, sizeof(unsigned) * 8, ctx->stream));
    return MP_OK;
}

// The words that have to be zero when a factorization starts.
unsigned *nd_control(mp_ctx *ctx, int *words) {
    *words = 8;
    return state_of(ctx)->ctl;
}

// Factors J = K - diag(FP) and solves J y = b.
int nd_factor_solve(mp_ctx *ctx, const double *b, double *y, bool control_cleared) {
    NdState *s = state_of(ctx);
    int rc = nd_begin(ctx, s, control_cleared);
    if (rc) return rc;
    NdArgs a;
    a.task = s->task;
    a.item = s->item;
    a.perm = s->perm;
    a.ent_src = s->ent_src;
    a.ent_at = s->ent_at;
    a.kval = ctx->sp_val;
    a.FP = ctx->FP;
    a.b = b;
    a.tile = s->tile;
    a.zd = s->zd;
    a.x = s->x;
    a.flag = s->flag;
    a.ctl = s->ctl;
    a.flags = ctx->counters + C_FLAGS;
    a.ntask = s->ntask;
    a.ntile = s->plan.ntile;
    a.ncol = s->plan.ncol;
    a.epoch = s->epoch;
    const int grid = std::min(ctx->sm_count, s->ntask);
    const int mk = kt_begin(ctx, MP_KT_UPDATE, 2.0 * T * T * T * (double)s->plan.products);
    k_nd_factor<<<grid, THREADS, sizeof(Smem), ctx->stream>>>(a), ++ctx->launches;
    kt_end(ctx, mk);
    MP_CUDA(ctx, cudaGetLastError());
    return nd_launch_solve(ctx, s, true, b, y, false);
}

// y += J^-1 b with the last factor.
int nd_solve_add(mp_ctx *ctx, const double *b, double *y) {
    NdState *s = state_of(ctx);
    int rc = nd_begin(ctx, s, false);
    if (rc) return rc;
    if ((rc = nd_launch_solve(ctx, s, false, b, nullptr, false))) return rc;
    return nd_launch_solve(ctx, s, true, b, y, true);
}

}  // namespace mp
