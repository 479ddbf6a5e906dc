// Conjugate gradients for J y = G, J = K - diag(FP), with a multilevel
// preconditioner: z = r / diag(J) + sum over levels P D^-1 P^T r (additive, the
// BPX form), P the trilinear functions of a regular grid laid over the mesh and D
// the diagonal of P^T J P.  The finest grid has a cell for about eight rows, every
// next one half as many along each axis.  FP64 throughout; every sum has a fixed
// order.
//
// One cooperative kernel a solve, one grid-wide round an iteration.  The rows are
// split over the blocks by recursive bisection of their positions and renumbered;
// a block keeps y = r / diag(J) and z of its own rows and of their neighbours'
// (its halo) in shared memory, so the product w = J z reads shared memory only.
// The round carries what w changes: w / diag(J) for the neighbours' halos, the
// block's share of P^T w on each level, and the sums that alpha and beta follow
// from.  A block then brings up to date, alike with its neighbours and with no
// further exchange, P^T r of those functions of the finer levels that its rows
// lie under, and of all functions from the first level of at most FULL_MAX.
//
// Measured (B200, a Newton step of SPARSE_CG, ||r|| <= 1e-12 ||G||; conjugate
// gradients with J's diagonal alone -> this): 144 unknowns 0.35 -> 0.25 ms (42 -> 29
// iterations), 1,859 0.83 -> 0.39, 13,678 1.50 -> 0.44, 32,244 2.65 -> 0.50, 112,847
// 5.1 -> 0.66, 255,822 8.3 -> 1.25 ms (437 -> 44 iterations).  An iteration is 10 us
// for one block, 17 at 112,847 unknowns and 28 at 255,822: the round 1.5, and a
// chain of short phases between block barriers, each of them latency- or shared-
// memory-bound; at 255,822 the product 5 (its loads of z, 4 cycles a warp for bank
// conflicts, and K's entries through L2), P^T w 6, the other blocks' data 3.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <exception>
#include <thread>

#include "mp_internal.h"

namespace mp {

namespace {

constexpr int THREADS = 512;                // 1,024 were slower: 1.25 -> 1.80 ms at 255,822 unknowns, for want of registers
constexpr int WARPS = THREADS / 32;
constexpr int ROWS_MAX = 4 * THREADS;       // of a block: their state stays in registers
constexpr unsigned SPIN_LIMIT = 1u << 22;
constexpr int MAX_RESTARTS = 3;
// Fewer rows: by the diagonal alone, which takes fewer than 40 iterations there (at
// 144 rows 0.35 ms against 0.25 by levels; no smaller mesh was measured).
constexpr int ROWS_FROM = 128;
constexpr int LEVELS_MAX = 10;
constexpr int FULL_MAX = 216;               // functions of the first level that every block holds whole
constexpr double WEIGHT = 0.3;              // of each level's correction
constexpr double MASS = 0.35;               // sum of phi^2 over sum of phi, about, of a function of any level
constexpr int HALO_REGS = 4, OWN_REGS = 4, TASK_REGS = 4;  // a thread's halo rows, functions and runs, at most
constexpr int RUN = 8;                      // shares added by one thread
constexpr int SMEM_MAX = 227 * 1024 - 2048; // dynamic shared memory of a plan, beside the kernel's static one

enum Status : unsigned { NOT_SPD = 1, TIMEOUT = 2, MAX_IT = 4 };

// A row's place: the cell's lowest function, and the position within the cell.
struct alignas(16) Loc {
    float f[3];
    int fn;
};
struct alignas(8) Place {                   // the same in shared memory: 1/65536ths, a needed function
    unsigned short f[3], fn;
};
struct Level {
    int dim[3];                             // functions along each axis
    int n, off;                             // functions, and the first one's place in the arrays over all levels
};
// A block's part of a level, boxes of functions: those that its rows are under,
// and those whose correction it needs; their places in its arrays.
struct Box {
    int own0[3], own[3], own_off;
    int need0[3], need[3], need_off;
};
struct Seg {
    int row0, count, block;                 // rows of one cell in one block
};

struct Args {
    int n, nb, nlev, nfn, full, first;      // full: the first level held whole
    int nl_max, nr_max, need_max, u_max;    // local rows, own rows, needed functions, the shared region's doubles
    int nc_max, own_max, task_max, halo_max;
    int hold;                               // columns of 32 pairs of entries of K that a block holds in shared memory
    int shares;                             // in all
    Level lev[LEVELS_MAX];
    const int *row, *row_off, *halo_off, *halo_src;
    const int *slice_off, *slice_ptr;
    const unsigned *col;                    // K's entries in pairs, 32 rows' to a column: two columns, two values
    const double2 *val;
    const double *kd;
    const Loc *loc;
    const Box *box;                         // [nb][nlev]
    const int *cell_off, *cell_row;
    const int *own_off, *own_pos;           // an own function's share's place, -1: none
    const unsigned *own_sum;                // and what it sums of the level below (Stencil)
    const int *ref_off;
    const uint4 *ref;                       // the finest level's own functions: sums of cells
    const int *task_off, *task;             // runs of shares: first / 2 << 3 | count / 2 (the odd one out is 0)
    const int *run_off;
    const unsigned short *run;              // a needed function's runs
    const double *dk;                       // diag(P^T K P), all levels
    const double *FP, *b;
    double *x;
    double *pub, *share, *sums;             // [2][n], [2][shares], [2][4][nb], by the round's parity
    unsigned *flag, *sync;                  // flag: counts the blocks' arrivals
    double *out;
    double rtol2;
    int max_it;
};

// P^T from one level to the next: a function sums its up to 3 x 3 x 3 finer ones,
// by 1 where they coincide along an axis and 1/2 beside.  Packed: the first one's
// index | along each axis, how many (2 bits) and the first one's offset + 1 (2 bits).
__host__ __device__ inline unsigned stencil(const int (&at)[3], const int *first, const int *dim) {
    unsigned code = 0;
    int index = 0, stride = 1;
    for (int d = 0; d < 3; d++) {
        const int c = 2 * at[d] - first[d];             // the coinciding one
        const int lo = c - 1 > 0 ? c - 1 : 0, hi = c + 1 < dim[d] - 1 ? c + 1 : dim[d] - 1;
        if (hi < lo) return 0;
        index += stride * lo;
        stride *= dim[d];
        code |= (unsigned)(hi - lo + 1) << (16 + 4 * d) | (unsigned)(lo - c + 1) << (18 + 4 * d);
    }
    return code | (unsigned)index;
}
// Eight lanes share a sum; all get it.  Lanes without one pass code 0.
__device__ __forceinline__ double stencil_sum(unsigned code, const double *p, int dx, int dxy, int lane) {
    double s = 0.0;
    const int nx = code >> 16 & 3, ny = code >> 20 & 3, nz = code >> 24 & 3;
    const int ox = code >> 18 & 3, oy = code >> 22 & 3, oz = code >> 26 & 3;
    p += code & 0xffffu;
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const int k = (lane & 7) + 8 * m, z = k / 9, y = k / 3 - 3 * z, x = k % 3;
        if (x < nx && y < ny && z < nz) {
            const int beside = (ox + x != 1) + (oy + y != 1) + (oz + z != 1);
            s = fma(__hiloint2double((1023 - beside) << 20, 0), p[x + y * dx + z * dxy], s);
        }
    }
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

__device__ __forceinline__ unsigned ld_relaxed(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void arrive(unsigned *p) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}

// Sums four values over the warp, in six shuffles: returns value (lane >> 3).
__device__ __forceinline__ double sum4(const double (&v)[4], int lane) {
    double a[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const double keep = lane & 16 ? v[k + 2] : v[k], give = lane & 16 ? v[k] : v[k + 2];
        a[k] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    }
    double s = (lane & 8 ? a[1] : a[0]) + __shfl_xor_sync(0xffffffffu, lane & 8 ? a[0] : a[1], 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// k / 65536, without a conversion (a quarter of FP64's rate).
__device__ __forceinline__ double fraction(unsigned short k) { return __hiloint2double(0x3ff00000 | k << 4, 0) - 1.0; }

// The eight functions of the cell, corner bits x, y, z, at a place in it.
__device__ __forceinline__ void weights(double fx, double fy, double fz, double (&w)[8]) {
    const double gx = 1.0 - fx, gy = 1.0 - fy, gz = 1.0 - fz;
    const double a = gy * gz, b = fy * gz, c = gy * fz, d = fy * fz;
    w[0] = gx * a, w[1] = fx * a, w[2] = gx * b, w[3] = fx * b;
    w[4] = gx * c, w[5] = fx * c, w[6] = gx * d, w[7] = fx * d;
}

// ---- before the iteration -----------------------------------------------------

// K in the blocks' layout: the off-diagonal entries and the diagonal.
__global__ void k_levels_gather(int slots, int n, const int *__restrict__ src, const int *__restrict__ kd_src,
                                const double *__restrict__ sp_val, double *val, double *kd) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < slots) val[i] = src[i] >= 0 ? sp_val[src[i]] : 0.0;
    if (i < n) kd[i] = sp_val[kd_src[i]];
}

// A cell's 8 x 8 part of P^T K P (36 numbers), eight lanes a cell, by K's edges:
// -K_ij (u_i - u_j)^2 / 2 from each end, with the cell's functions carried on past
// its faces, and the row sums' u_i^2.
__global__ void __launch_bounds__(128) k_levels_cells(Args a, int ncell, const int *__restrict__ seg_ptr,
                                                      const Seg *__restrict__ seg, double *e) {
    const int c = blockIdx.x * 16 + (threadIdx.x >> 3), lane = threadIdx.x & 7;
    double acc[36];
#pragma unroll
    for (int k = 0; k < 36; k++) acc[k] = 0.0;
    auto add = [&](double t, const double (&w)[8]) {
#pragma unroll
        for (int p = 0; p < 8; p++)
#pragma unroll
            for (int q = 0; q <= p; q++) acc[p * (p + 1) / 2 + q] = fma(t * w[p], w[q], acc[p * (p + 1) / 2 + q]);
    };
    if (c < ncell)
        for (int s = seg_ptr[c]; s < seg_ptr[c + 1]; s++) {
            const Seg sg = seg[s];
            const int r0 = a.row_off[sg.block];
            const Loc *loc = a.loc + r0 + a.halo_off[sg.block];
            for (int k = lane; k < sg.count; k += 8) {
                const int i = sg.row0 - r0 + k;
                const Loc L = loc[i];
                double w[8];
                weights(L.f[0], L.f[1], L.f[2], w);
                const int dx = a.lev[0].dim[0], dy = a.lev[0].dim[1];
                const int slice = a.slice_off[sg.block] + (i >> 5);
                const int base = a.slice_ptr[slice] + (i & 31), width = (a.slice_ptr[slice + 1] - a.slice_ptr[slice]) >> 4;
                double rs = a.kd[r0 + i];
                for (int m = 0; m < width; m++) {
                    const double2 pair = a.val[base + 32 * (m >> 1)];
                    const double v = m & 1 ? pair.y : pair.x;
                    const Loc N = loc[a.col[base + 32 * (m >> 1)] >> (16 * (m & 1)) & 0xffffu];
                    rs += v;
                    double u[8];
                    weights(N.f[0] + (N.fn % dx - L.fn % dx), N.f[1] + (N.fn / dx % dy - L.fn / dx % dy),
                            N.f[2] + (N.fn / dx / dy - L.fn / dx / dy), u);
#pragma unroll
                    for (int p = 0; p < 8; p++) u[p] -= w[p];
                    add(-0.5 * v, u);
                }
                add(rs, w);
            }
        }
#pragma unroll
    for (int k = 0; k < 36; k++) {
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
        if (lane == 0 && c < ncell) e[36 * (size_t)c + k] = acc[k];
    }
}

// diag(P^T K P) of every level's functions, one warp a function: a coarser
// function is piecewise trilinear on the finest level's cells.
__global__ void __launch_bounds__(128) k_levels_diag(Args a, const double *__restrict__ e, double *dk) {
    const int f = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (f >= a.nfn) return;
    int l = 0;
    while (l + 1 < a.nlev && f >= a.lev[l + 1].off) l++;
    const int g = f - a.lev[l].off, s = 1 << l;
    const int X[3] = {g % a.lev[l].dim[0], g / a.lev[l].dim[0] % a.lev[l].dim[1], g / a.lev[l].dim[0] / a.lev[l].dim[1]};
    int lo[3], len[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        lo[d] = max(0, (X[d] - 1) * s);
        len[d] = max(0, min(a.lev[0].dim[d] - 1, (X[d] + 1) * s) - lo[d]);
    }
    const int cx = a.lev[0].dim[0] - 1, cy = a.lev[0].dim[1] - 1;
    double sum = 0.0;
    for (int k = lane; k < len[0] * len[1] * len[2]; k += 32) {
        const int P[3] = {lo[0] + k % len[0], lo[1] + k / len[0] % len[1], lo[2] + k / len[0] / len[1]};
        const size_t id = P[0] + cx * (P[1] + cy * P[2]);
        double h[3][2], w[8];
#pragma unroll
        for (int d = 0; d < 3; d++)
#pragma unroll
            for (int o = 0; o < 2; o++) h[d][o] = fmax(0.0, 1.0 - fabs((double)(P[d] + o) / s - X[d]));
#pragma unroll
        for (int c = 0; c < 8; c++) w[c] = h[0][c & 1] * h[1][(c >> 1) & 1] * h[2][c >> 2];
#pragma unroll
        for (int p = 0; p < 8; p++)
#pragma unroll
            for (int q = 0; q <= p; q++)
                sum = fma((p == q ? 1.0 : 2.0) * w[p] * w[q], e[36 * id + p * (p + 1) / 2 + q], sum);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) dk[f] = sum;
}

// ---- the iteration -----------------------------------------------------------------

#define ROWS(j, i)                                                                                   \
    _Pragma("unroll") for (int j = 0, i = threadIdx.x; j < RPT; j++, i += THREADS) if (i < nr)

template <int RPT>
__global__ void __launch_bounds__(THREADS, 1) k_cg_levels(Args a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, blk = blockIdx.x;
    double2 *hval = reinterpret_cast<double2 *>(smem);  // the first pairs of K's entries
    Place *loc = reinterpret_cast<Place *>(hval + 32 * a.hold);
    double *y = reinterpret_cast<double *>(loc + a.nl_max);
    double *z = y + a.nl_max;
    double *rc = z + a.nl_max;                  // P^T r of the needed functions, level by level
    double *wc = rc + a.need_max;               // P^T q of them
    double *inv = wc + a.need_max;              // WEIGHT / diag(P^T J P)
    double *u = inv + a.need_max;               // before a round: w, cells' sums, own shares; after it: runs, corrections
    double *red = u + a.u_max;                  // [WARPS][4]
    double *tot = red + 4 * WARPS;              // [4]
    unsigned *par = reinterpret_cast<unsigned *>(tot + 4);  // a needed function's lowest parent | odd coordinates << 24
    unsigned short *run = reinterpret_cast<unsigned short *>(par + a.need_max);
    unsigned short *crow = run + a.need_max + 1;              // first rows of the cells
    int *pos = reinterpret_cast<int *>(crow + a.nc_max + 1 + (a.need_max + a.nc_max & 1));
    unsigned *osum = reinterpret_cast<unsigned *>(pos + a.own_max);
    int *task = reinterpret_cast<int *>(osum + a.own_max);
    int *hsrc = task + a.task_max;
    int *hslice = hsrc + a.halo_max;                          // pairs before each slice
    unsigned *hcol = reinterpret_cast<unsigned *>(hslice + a.nr_max / 32 + 2);
    __shared__ Box box[LEVELS_MAX];
    __shared__ unsigned rest[FULL_MAX];         // the coarsest levels' sums of the level below
    const int r0 = a.row_off[blk], nr = a.row_off[blk + 1] - r0;
    const int h0 = a.halo_off[blk], nh = a.halo_off[blk + 1] - h0, nl = nr + nh;
    const int s0 = a.slice_off[blk];
    const int c0 = a.cell_off[blk], nc = a.cell_off[blk + 1] - c0;
    const int t0 = a.task_off[blk], nt = a.task_off[blk + 1] - t0;
    const int own_first = a.own_off[blk], nown = a.own_off[blk + 1] - own_first;
    const double sg = a.kd[a.first] - a.FP[0] < 0 ? -1.0 : 1.0;
    if (t < a.nlev) box[t] = a.box[blk * a.nlev + t];
    __syncthreads();
    const Box &bl = box[a.nlev - 1];
    const int nneed = bl.need_off + bl.need[0] * bl.need[1] * bl.need[2];
    const int nread = a.full + 1 < a.nlev ? box[a.full + 1].need_off : nneed;  // needed functions that shares are read for
    double *ua = u;                             // w of the block's rows
    double *mom = ua + a.nr_max;                // each cell's sums with its eight functions
    double *own = mom + 8 * nc;                 // own functions, level by level
    double *part = u;                           // sums of runs
    double *ec = part + nt;                     // corrections of the needed functions

#pragma unroll 1
    for (int i = t; i < nl; i += THREADS) {
        const Loc L = a.loc[r0 + h0 + i];
        const int dx = a.lev[0].dim[0], dy = a.lev[0].dim[1];
        Place q;
#pragma unroll
        for (int d = 0; d < 3; d++) q.f[d] = (unsigned short)(65536.0f * L.f[d]);
        q.fn = (unsigned short)(L.fn % dx - box[0].need0[0] +
                                box[0].need[0] * (L.fn / dx % dy - box[0].need0[1] +
                                                  box[0].need[1] * (L.fn / dx / dy - box[0].need0[2])));
        loc[i] = q;
    }
    const int e0 = a.slice_ptr[s0], held = min(a.hold, (a.slice_ptr[a.slice_off[blk + 1]] - e0) >> 5);
#pragma unroll 1
    for (int i = t; i < 32 * held; i += THREADS) {
        hval[i] = a.val[e0 + i];
        hcol[i] = a.col[e0 + i];
    }
#pragma unroll 1
    for (int i = t; i <= nread; i += THREADS) run[i] = a.run[a.run_off[blk] + i];
#pragma unroll 1
    for (int l = 0; l < a.nlev; l++) {
        const Box &B = box[l];
#pragma unroll 1
        for (int i = t; i < B.need[0] * B.need[1] * B.need[2]; i += THREADS) {
            const int x = B.need0[0] + i % B.need[0], yy = B.need0[1] + i / B.need[0] % B.need[1],
                      zz = B.need0[2] + i / B.need[0] / B.need[1];
            if (l > a.full) rest[B.need_off + i - nread] = stencil({x, yy, zz}, box[l - 1].need0, box[l - 1].need);
            inv[B.need_off + i] = sg * a.dk[a.lev[l].off + x + a.lev[l].dim[0] * (yy + a.lev[l].dim[1] * zz)];
            if (l + 1 < a.nlev) {
                const Box &C = box[l + 1];
                par[B.need_off + i] = (C.need_off + (x >> 1) - C.need0[0] +
                                       C.need[0] * ((yy >> 1) - C.need0[1] + C.need[1] * ((zz >> 1) - C.need0[2]))) |
                                      (unsigned)((x & 1) | (yy & 1) << 1 | (zz & 1) << 2) << 24;
            }
        }
    }
#pragma unroll 1
    for (int i = t; i < nown; i += THREADS) {
        pos[i] = a.own_pos[own_first + i];
        osum[i] = a.own_sum[own_first + i];
    }
#pragma unroll 1
    for (int i = t; i < nt; i += THREADS) task[i] = a.task[t0 + i];
#pragma unroll 1
    for (int i = t; i < nh; i += THREADS) hsrc[i] = a.halo_src[h0 + i];
#pragma unroll 1
    for (int i = t; i <= nc; i += THREADS) crow[i] = (unsigned short)a.cell_row[c0 + blk + i];
#pragma unroll 1
    for (int i = t; i <= a.slice_off[blk + 1] - s0; i += THREADS) hslice[i] = (a.slice_ptr[s0 + i] - e0) >> 5;

    double X[RPT], P[RPT], V[RPT], D[RPT], Di[RPT], hv[HALO_REGS];
    unsigned st = 0;
    ROWS(j, i) {
        double jd = sg * (a.kd[r0 + i] - a.FP[a.row[r0 + i]]);
        if (!(jd > 0)) {
            st |= NOT_SPD;
            jd = 1;
        }
        D[j] = jd;
        Di[j] = 1.0 / jd;
        X[j] = P[j] = V[j] = 0.0;
        ua[i] = -sg * a.FP[a.row[r0 + i]];
    }
    if (st) atomicOr(a.sync + 1, st);

    // ua = the off-diagonal entries' part of K z, from shared memory
    auto products = [&]() {
        auto entries = [&](int i, const double2 *val, const unsigned *col, int pairs) {
            double s = 0.0, s2 = 0.0;
#pragma unroll 1
            for (int k0 = 0; k0 < pairs; k0 += 8) {
                double2 v[8];
                unsigned c[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const bool in = k0 + k < pairs;
                    v[k] = in ? val[32 * (k0 + k)] : make_double2(0.0, 0.0);
                    c[k] = in ? col[32 * (k0 + k)] : i | i << 16;
                }
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    s = fma(v[k].x, z[c[k] & 0xffffu], s);
                    s2 = fma(v[k].y, z[c[k] >> 16], s2);
                }
            }
            ua[i] = s + s2;
        };
#pragma unroll 1
        for (int i = t; i < nr; i += THREADS) {
            const int p = hslice[i >> 5], w = hslice[(i >> 5) + 1] - p;
            if (p + w > held) entries(i, a.val + e0 + 32 * p + lane, a.col + e0 + 32 * p + lane, w);
            else entries(i, hval + 32 * p + lane, hcol + 32 * p + lane, w);
        }
    };

    // One round: what the block has written to pub, its shares of P^T (ua) and its
    // sums become visible, and every other block's have.  Buffers alternate: a
    // block is at most one round ahead of another's reading.
    unsigned round = 0;
    auto exchange = [&](const double (&s)[4], bool shares) {
        const int parity = round & 1;
        const int nown0 = box[0].own[0] * box[0].own[1] * box[0].own[2];
        const double mine = sum4(s, lane);
        if ((lane & 7) == 0) red[4 * warp + (lane >> 3)] = mine;
        __syncthreads();
        if (warp == WARPS - 1) {
            double v = 0.0;
#pragma unroll
            for (int w = 0; w < WARPS / 8; w++) v += red[4 * (WARPS / 8 * (lane >> 2) + w) + (lane & 3)];
            v += __shfl_xor_sync(0xffffffffu, v, 4);
            v += __shfl_xor_sync(0xffffffffu, v, 8);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            if (lane < 4) __stcg(a.sums + (parity * 4 + lane) * a.nb + blk, v);
        }
        if (shares) {
            // eight lanes a cell, a row each; then a function each
            const int g8 = lane & 7;
            uint4 ref[2];
#pragma unroll
            for (int k = 0; k < 2; k++)
                if (t + k * THREADS < nown0) ref[k] = __ldg(a.ref + a.ref_off[blk] + t + k * THREADS);
#pragma unroll 1
            for (int c = t >> 3; c - (lane >> 3) < nc; c += THREADS / 8) {
                double m[8];
#pragma unroll
                for (int k = 0; k < 8; k++) m[k] = 0.0;
                const int end = c < nc ? crow[c + 1] : 0;
#pragma unroll 1
                for (int i = (c < nc ? crow[c] : 0) + g8; i < end; i += 8) {
                    const Place L = loc[i];
                    double w[8];
                    weights(fraction(L.f[0]), fraction(L.f[1]), fraction(L.f[2]), w);
                    const double q = ua[i];
#pragma unroll
                    for (int k = 0; k < 8; k++) m[k] = fma(w[k], q, m[k]);
                }
                double h[4], f[2];
#pragma unroll
                for (int k = 0; k < 4; k++)
                    h[k] = (g8 & 4 ? m[k + 4] : m[k]) + __shfl_xor_sync(0xffffffffu, g8 & 4 ? m[k] : m[k + 4], 4);
#pragma unroll
                for (int k = 0; k < 2; k++)
                    f[k] = (g8 & 2 ? h[k + 2] : h[k]) + __shfl_xor_sync(0xffffffffu, g8 & 2 ? h[k] : h[k + 2], 2);
                const double v = (g8 & 1 ? f[1] : f[0]) + __shfl_xor_sync(0xffffffffu, g8 & 1 ? f[0] : f[1], 1);
                if (c < nc) mom[8 * c + g8] = v;
            }
            __syncthreads();
            double *out = a.share + (size_t)parity * a.shares;
            auto cells = [&](int f, const uint4 &ref) {
                const unsigned r[4] = {ref.x, ref.y, ref.z, ref.w};
                double v = 0.0;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const unsigned at = (r[k >> 1] >> (16 * (k & 1))) & 0xffffu;
                    if (at != 0xffffu) v += mom[at];
                }
                own[f] = v;
            };
#pragma unroll
            for (int k = 0; k < 2; k++)
                if (t + k * THREADS < nown0) cells(t + k * THREADS, ref[k]);
#pragma unroll 1
            for (int f = t + 2 * THREADS; f < nown0; f += THREADS) cells(f, __ldg(a.ref + a.ref_off[blk] + f));
#pragma unroll 1
            for (int l = 1; l <= a.full; l++) {
                __syncthreads();
                const int o = box[l].own_off, end = o + box[l].own[0] * box[l].own[1] * box[l].own[2];
                const int dx = box[l - 1].own[0], dxy = dx * box[l - 1].own[1];
#pragma unroll 1
                for (int f = o + (t >> 3); f - (lane >> 3) < end; f += THREADS / 8) {
                    const double v = stencil_sum(f < end ? osum[f] : 0, own + box[l - 1].own_off, dx, dxy, lane);
                    if (f < end && (lane & 7) == 0) own[f] = v;
                }
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < OWN_REGS; k++)
                if (t + k * THREADS < nown && pos[t + k * THREADS] >= 0) __stcg(out + pos[t + k * THREADS], own[t + k * THREADS]);
        }
        __syncthreads();
        round++;
        int ok = 1;
        if (t == 0) {
            // release: the block's writes are ordered before this thread by the barrier
            arrive(a.flag);
            const unsigned all = round * a.nb;
#pragma unroll 1
            for (unsigned spins = 1; ld_acquire(a.flag) < all; spins++) {
                if ((spins & 63) == 0 && ld_relaxed(a.sync)) {
                    ok = 0;
                    break;
                }
                if (spins > SPIN_LIMIT) {
                    atomicExch(a.sync, 1u);
                    atomicOr(a.sync + 1, (unsigned)TIMEOUT);
                    ok = 0;
                    break;
                }
            }
        }
        return __syncthreads_and(ok) != 0;
    };
    // After a round: the other blocks' part of what the caller goes on with.
    // hv: the halo's values; tot; part: sums of the runs of shares.
    auto gather = [&](bool shares) {
        const int parity = (round - 1) & 1;
        const double *pub = a.pub + (size_t)parity * a.n;
#pragma unroll
        for (int k = 0; k < HALO_REGS; k++)
            hv[k] = t + k * THREADS < nh ? __ldcg(pub + hsrc[t + k * THREADS]) : 0.0;
        if (warp < 4) {
            double s = 0.0, p[5];
            const double *in = a.sums + (parity * 4 + warp) * a.nb;
#pragma unroll
            for (int k = 0; k < 5; k++) p[k] = lane + 32 * k < a.nb ? __ldcg(in + lane + 32 * k) : 0.0;
#pragma unroll
            for (int k = 0; k < 5; k++) s += p[k];
#pragma unroll 1
            for (int k = lane + 160; k < a.nb; k += 32) s += __ldcg(in + k);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) tot[warp] = s;
        }
        if (shares) {
            const double *in = a.share + (size_t)parity * a.shares;
#pragma unroll
            for (int k = 0; k < TASK_REGS; k++) {
                if (k * THREADS >= nt) break;
                const int q = t + k * THREADS < nt ? task[t + k * THREADS] : 0;
                double2 v[RUN / 2];
                double s = 0.0;
#pragma unroll
                for (int m = 0; m < RUN / 2; m++)
                    v[m] = m < (q & 7) ? __ldcg(reinterpret_cast<const double2 *>(in + 2 * (q >> 3)) + m)
                                             : make_double2(0.0, 0.0);
#pragma unroll
                for (int m = 0; m < RUN / 2; m++) s += v[m].x + v[m].y;
                if (t + k * THREADS < nt) part[t + k * THREADS] = s;
            }
        }
        __syncthreads();
    };
    // From P^T r: the corrections, coarsest level first, and z.
    auto correct = [&]() {
#pragma unroll 1
        for (int l = a.nlev - 1; l >= 0; l--) {
            const int first = box[l].need_off, end = first + box[l].need[0] * box[l].need[1] * box[l].need[2];
            const int ux = l + 1 < a.nlev ? box[l + 1].need[0] : 0, uy = l + 1 < a.nlev ? ux * box[l + 1].need[1] : 0;
#pragma unroll 1
            for (int i = first + t; i < end; i += THREADS) {
                double s = 0.0;
                if (l + 1 < a.nlev) {
                    const unsigned q = par[i];
                    const double *p = ec + (q & 0xffffffu);
                    const int x = q >> 24 & 1, yy = q & 1u << 25 ? ux : 0, zz = q & 1u << 26 ? uy : 0;
                    s = ((p[0] + p[x]) + (p[yy] + p[yy + x])) + ((p[zz] + p[zz + x]) + (p[zz + yy] + p[zz + yy + x]));
                }
                ec[i] = fma(0.125, s, inv[i] * rc[i]);
            }
            __syncthreads();
        }
        const int ox = box[0].need[0], oy = ox * box[0].need[1];
#pragma unroll 2
        for (int i = t; i < nl; i += THREADS) {
            const Place L = loc[i];
            const double *p = ec + L.fn;
            const double fx = fraction(L.f[0]), fy = fraction(L.f[1]), fz = fraction(L.f[2]);
            const double a0 = fma(fx, p[1] - p[0], p[0]), a1 = fma(fx, p[ox + 1] - p[ox], p[ox]);
            const double b0 = fma(fx, p[oy + 1] - p[oy], p[oy]), b1 = fma(fx, p[oy + ox + 1] - p[oy + ox], p[oy + ox]);
            const double c = fma(fy, a1 - a0, a0), d = fma(fy, b1 - b0, b0);
            z[i] = y[i] + fma(fz, d - c, c);
        }
        __syncthreads();
    };

    // One loop for the four kinds of round, so that the code, which is executed from
    // the instruction cache, is there once.
    enum { MASS_SUM, SEND_X, RESIDUAL, STEP } kind = MASS_SUM;
    double bb = 0, rr = 0, gamma = 1.0, pq = 0.0;
    double vh[HALO_REGS], wr[RPT];
    int it = 0, restarts = 0;
    bool first = true, start = true;
    __syncthreads();
#pragma unroll 1
    while (true) {
        double v[4] = {0.0, 0.0, 0.0, 0.0};
        double *pub = a.pub + (size_t)(round & 1) * a.n + r0;
        if (kind == STEP || (kind == RESIDUAL && !first)) products();
        if (kind == STEP) {
            // w = J z; (r, z), (z, w), (z, q) + (p, w) of the last p and q = J p, (r, r)
            ROWS(j, i) {
                const double zi = z[i], w = fma(D[j], zi, sg * ua[i]), ri = D[j] * y[i];
                ua[i] = w;
                wr[j] = __dmul_rn(w, Di[j]);
                __stcg(pub + i, wr[j]);
                v[0] = fma(ri, zi, v[0]);
                v[1] = fma(zi, w, v[1]);
                if (!start) v[2] = fma(zi, D[j] * V[j], fma(P[j], w, v[2]));
                v[3] = fma(ri, ri, v[3]);
            }
        } else if (kind == RESIDUAL) {
            // r = b - J x (x = 0 the first time)
            ROWS(j, i) {
                double ri = sg * a.b[a.row[r0 + i]];
                if (!first) ri -= fma(D[j], z[i], sg * ua[i]);
                y[i] = Di[j] * ri;
                ua[i] = ri;
                __stcg(pub + i, y[i]);
                v[3] = fma(ri, ri, v[3]);
            }
        } else if (kind == SEND_X) {
            ROWS(j, i) __stcg(pub + i, X[j]);
        }
        if (!exchange(v, kind != SEND_X)) break;
        gather(kind != SEND_X);
        if (kind == SEND_X) {
            ROWS(j, i) z[i] = X[j];
#pragma unroll
            for (int k = 0; k < HALO_REGS; k++)
                if (t + k * THREADS < nh) z[nr + t + k * THREADS] = hv[k];
            __syncthreads();
            kind = RESIDUAL;
            continue;
        }
        double alpha = 0.0, beta = 0.0;
        if (kind == RESIDUAL) {
            rr = tot[3];
            if (first) bb = rr;
            if (rr <= a.rtol2 * bb) break;
            if (it >= a.max_it || (!first && restarts >= MAX_RESTARTS)) {
                if (blk == 0 && t == 0) atomicOr(a.sync + 1, (unsigned)MAX_IT);
                break;
            }
            if (!first) restarts++;
            first = false;
            start = true;
#pragma unroll
            for (int k = 0; k < HALO_REGS; k++)
                if (t + k * THREADS < nh) y[nr + t + k * THREADS] = hv[k];
        } else if (kind == STEP) {
            rr = tot[3];
            if (rr <= a.rtol2 * bb || it >= a.max_it) {
                __syncthreads();                // tot has been read
                kind = SEND_X;
                continue;
            }
            beta = start ? 0.0 : tot[0] / gamma;
            pq = start ? tot[1] : fma(beta * beta, pq, fma(beta, tot[2], tot[1]));
            gamma = tot[0];
            if (!(pq > 0)) {
                if (blk == 0 && t == 0) atomicOr(a.sync + 1, (unsigned)NOT_SPD);
                break;
            }
            alpha = gamma / pq;
            // p = z + beta p, v = w / diag(J) + beta v, x += alpha p, y -= alpha v,
            // y alike in a row's block and in its neighbours'
            ROWS(j, i) {
                P[j] = start ? z[i] : fma(beta, P[j], z[i]);
                V[j] = start ? wr[j] : fma(beta, V[j], wr[j]);
                X[j] = fma(alpha, P[j], X[j]);
                y[i] = fma(-alpha, V[j], y[i]);
            }
#pragma unroll
            for (int k = 0; k < HALO_REGS; k++)
                if (t + k * THREADS < nh) {
                    vh[k] = start ? hv[k] : fma(beta, vh[k], hv[k]);
                    y[nr + t + k * THREADS] = fma(-alpha, vh[k], y[nr + t + k * THREADS]);
                }
            start = false;
            it++;
        }
        // P^T q and P^T r; or P^T r itself; or what the levels' diagonals need of FP
#pragma unroll 1
        for (int i = t; i < nread; i += THREADS) {
            double s = 0.0;
#pragma unroll 1
            for (int k = run[i]; k < run[i + 1]; k++) s += part[k];
            if (kind == STEP) {
                wc[i] = fma(beta, wc[i], s);
                rc[i] = fma(-alpha, wc[i], rc[i]);
            } else {
                rc[i] = s;
                wc[i] = 0.0;
            }
        }
        __syncthreads();
        // the levels above `full`, all functions of which every block has
#pragma unroll 1
        for (int l = a.full + 1; l < a.nlev; l++) {
            const Box &B = box[l], &A = box[l - 1];
            const int end = B.need_off + B.need[0] * B.need[1] * B.need[2];
#pragma unroll 1
            for (int f = B.need_off + (t >> 3); f - (lane >> 3) < end; f += THREADS / 8) {
                const double v = stencil_sum(f < end ? rest[f - nread] : 0, rc + A.need_off, A.need[0],
                                             A.need[0] * A.need[1], lane);
                if (f < end && (lane & 7) == 0) rc[f] = v;
            }
            __syncthreads();
        }
        if (kind == MASS_SUM) {
            // diag(P^T J P): P^T K P's, and MASS of P^T (-FP)
#pragma unroll 1
            for (int i = t; i < nneed; i += THREADS) {
                const double d = fma(MASS, rc[i], inv[i]);
                inv[i] = d > 1e-200 ? WEIGHT / d : 0.0;  // 0: a function that no row is under
            }
            __syncthreads();
            kind = RESIDUAL;
            continue;
        }
        correct();
        kind = STEP;
    }
    ROWS(j, i) a.x[a.row[r0 + i]] = X[j];
    if (blk == 0 && t == 0) {
        a.out[0] = it;
        a.out[1] = rr;
        a.out[2] = bb;
        a.out[3] = restarts;
    }
}
#undef ROWS

// ---- the plan -------------------------------------------------------------------------

struct Plan {
    bool usable = false;
    Args a{};
    int slots = 0, ncell = 0, rows_max = 0;
    size_t smem = 0;
    unsigned changes = 0;                   // of sp_val, when val, kd and dk were formed
    bool formed = false;
    void *blob = nullptr;
    double *val = nullptr, *kd = nullptr, *e = nullptr, *dk = nullptr;
    const int *src = nullptr, *kd_src = nullptr, *seg_ptr = nullptr;
    const Seg *seg = nullptr;
};

// Runs work(first, last) over [0, n) on a few threads (or here, where none can be
// had).  An exception in one is thrown again here.
template <typename F>
void in_parallel(int n, F work) {
    const int th = std::max(1, std::min({n, 8, (int)std::thread::hardware_concurrency()}));
    std::vector<std::thread> pool;
    std::vector<std::exception_ptr> failed(th);
    auto part = [&](int k) {
        try {
            work((int)((long long)n * k / th), (int)((long long)n * (k + 1) / th));
        } catch (...) {
            failed[k] = std::current_exception();
        }
    };
    pool.reserve(th);
    for (int k = 1; k < th; k++) {
        try {
            pool.emplace_back(part, k);
        } catch (const std::exception &) {
            part(k);
        }
    }
    part(0);
    for (std::thread &p : pool) p.join();
    for (const std::exception_ptr &f : failed)
        if (f) std::rethrow_exception(f);
}

// Splits idx[first, last) into `parts` runs of equal length, by bisection across
// the longest extent; end[] takes the runs' ends.  The halves go to two threads
// while `fork` lasts and threads can be had.
void bisect(const float *pos, int *idx, int first, int last, int parts, int part0, int *end, int fork) {
    if (parts == 1) {
        end[part0] = last;
        return;
    }
    float lo[3], hi[3];
    for (int d = 0; d < 3; d++) lo[d] = INFINITY, hi[d] = -INFINITY;
    for (int k = first; k < last; k++)
        for (int d = 0; d < 3; d++) {
            const float v = pos[3 * (size_t)idx[k] + d];
            lo[d] = std::min(lo[d], v);
            hi[d] = std::max(hi[d], v);
        }
    int d = 0;
    for (int k = 1; k < 3; k++)
        if (hi[k] - lo[k] > hi[d] - lo[d]) d = k;
    const int left = parts / 2, mid = first + (int)((long long)(last - first) * left / parts);
    std::nth_element(idx + first, idx + mid, idx + last, [&](int p, int q) {
        const float a = pos[3 * (size_t)p + d], b = pos[3 * (size_t)q + d];
        return a != b ? a < b : p < q;
    });
    std::thread other;
    if (fork > 0) {
        try {
            other = std::thread(bisect, pos, idx, first, mid, left, part0, end, fork - 1);
        } catch (const std::exception &) {
        }
    }
    if (!other.joinable()) bisect(pos, idx, first, mid, left, part0, end, 0);
    bisect(pos, idx, mid, last, parts - left, part0 + left, end, fork > 0 ? fork - 1 : 0);
    if (other.joinable()) other.join();
}

Plan *plan_of(mp_ctx *ctx) { return static_cast<Plan *>(ctx->cg_levels); }

}  // namespace

void cg_levels_free(mp_ctx *ctx) {
    Plan *p = plan_of(ctx);
    if (!p) return;
    void *dev[] = {p->blob, p->val};
    for (void *q : dev)
        if (q) cudaFree(q);
    delete p;
    ctx->cg_levels = nullptr;
}

static int make_plan(mp_ctx *ctx, Plan *p, const std::vector<long long> &rowp, const std::vector<int> &cols,
                     const std::vector<long long> &slot) {
    const int n = ctx->neq, nb = std::min(ctx->sm_count, (n + THREADS - 1) / THREADS);
    if (n < ROWS_FROM || nb > THREADS || (n + nb - 1) / nb > ROWS_MAX || ctx->sp_slots > 0x7fffffffll) return MP_OK;
    Args &a = p->a;

    // places: the box of the mesh, in cells of the finest level
    std::vector<float> pos(3 * (size_t)n, 0.0f);
    std::vector<int> cell(n, 0);
    int cells[3];
    std::vector<Loc> place(n);
    {
        std::vector<double> npos(3 * (size_t)ctx->n_nodes);
        std::vector<int> ID(ctx->n_nodes);
        MP_CUDA(ctx, cudaMemcpy(npos.data(), ctx->node_pos, sizeof(double) * npos.size(), cudaMemcpyDeviceToHost));
        MP_CUDA(ctx, cudaMemcpy(ID.data(), ctx->ID, sizeof(int) * ID.size(), cudaMemcpyDeviceToHost));
        double lo[3], ext[3], most = 0;
        for (int d = 0; d < 3; d++) {
            double l = INFINITY, h = -INFINITY;
            for (int k = 0; k < ctx->n_nodes; k++) {
                l = std::min(l, npos[3 * (size_t)k + d]);
                h = std::max(h, npos[3 * (size_t)k + d]);
            }
            lo[d] = l;
            ext[d] = h - l;
            most = std::max(most, ext[d]);
        }
        if (!(most > 0) || !std::isfinite(most)) return MP_OK;
        const double limit = n / 8.0;
        for (int d = 0; d < 3; d++) ext[d] = std::max(ext[d], 1e-6 * most);
        double H = std::cbrt(ext[0] * ext[1] * ext[2] / limit);
        while (true) {
            double c = 1;
            for (int d = 0; d < 3; d++) {
                cells[d] = (int)std::min(1e6, std::max(1.0, std::ceil(ext[d] / H - 1e-9)));
                c *= cells[d];
            }
            if (c <= limit) break;
            H *= 1.02;
        }
        // A thin box one cell thick between planes of fixed nodes: its smooth errors die out across
        // the box by themselves, and functions that do not vanish on the planes only cost.  By levels
        // and by the diagonal, unit boxes of 6^3 to 20^3 hexes made thinner: 0.01 to 0.03 of the
        // extent 0.34 to 1.43 ms and 0.14 to 0.89, 0.05 (8^3 to 16^3) 0.36 to 0.87 and 0.33 to 0.78,
        // 0.07 (8^3, 12^3) 0.34, 0.70 and 0.37, 0.56, but 0.1 (8^3, 10^3) 0.33, 0.43 and 0.42, 0.57.
        for (int d = 0; d < 3; d++) {
            double l = INFINITY, h = -INFINITY;
            for (int k = 0; k < ctx->n_nodes; k++)
                if (ID[k] >= 0) {
                    l = std::min(l, npos[3 * (size_t)k + d]);
                    h = std::max(h, npos[3 * (size_t)k + d]);
                }
            const double edge = 1e-9 * ext[d];
            if (cells[d] == 1 && 14 * ext[d] <= most && l > lo[d] + edge && h < lo[d] + ext[d] - edge) return MP_OK;
        }
        for (int k = 0; k < ctx->n_nodes; k++) {
            const int q = ID[k];
            if (q < 0 || q >= n) continue;
            int c[3];
            for (int d = 0; d < 3; d++) {
                double u = (npos[3 * (size_t)k + d] - lo[d]) / H;
                if (!(u >= 0)) u = 0;       // a position that is no number
                c[d] = std::max(0, std::min((int)u, cells[d] - 1));
                // in 1/65536ths, as the kernel keeps it
                place[q].f[d] = (float)(std::min(65535.0, std::max(0.0, std::floor(65536.0 * (u - c[d]) + 0.5))) / 65536.0);
                pos[3 * (size_t)q + d] = (float)u;
            }
            cell[q] = c[0] + cells[0] * (c[1] + cells[1] * c[2]);
            place[q].fn = c[0] + (cells[0] + 1) * (c[1] + (cells[1] + 1) * c[2]);
        }
    }
    a.nlev = 0;
    a.nfn = 0;
    for (int l = 0, c[3] = {cells[0], cells[1], cells[2]}; l < LEVELS_MAX; l++) {
        Level &L = a.lev[l];
        L.n = 1;
        for (int d = 0; d < 3; d++) L.n *= L.dim[d] = c[d] + 1;
        L.off = a.nfn;
        a.nfn += L.n;
        a.nlev++;
        if (std::max({c[0], c[1], c[2]}) <= 3) break;
        for (int d = 0; d < 3; d++) c[d] = (c[d] + 1) / 2;
    }
    for (a.full = 0; a.full + 1 < a.nlev && a.lev[a.full].n > FULL_MAX;) a.full++;
    const int ncells = cells[0] * cells[1] * cells[2];

    // rows: split over the blocks, sorted by cell within each
    std::vector<int> row(n), end(nb), row_off(nb + 1, 0), where(n), owner(n);
    for (int k = 0; k < n; k++) row[k] = k;
    bisect(pos.data(), row.data(), 0, n, nb, 0, end.data(), 3);
    for (int b = 0; b < nb; b++) row_off[b + 1] = end[b];
    struct Block {
        std::vector<int> halo, cell_row, cell;
        std::vector<int> slice;             // widths
        std::vector<unsigned short> run;
        std::vector<int> src, pos, task;
        std::vector<unsigned> col, sum;
        std::vector<uint4> ref;
        Box box[LEVELS_MAX];
        int nown = 0, nneed = 0;
        bool fits = true;
    };
    std::vector<Block> B(nb);
    in_parallel(nb, [&](int b0, int b1) {
        for (int b = b0; b < b1; b++) {
            std::sort(row.begin() + row_off[b], row.begin() + row_off[b + 1],
                      [&](int u, int v) { return cell[u] != cell[v] ? cell[u] < cell[v] : u < v; });
            for (int k = row_off[b]; k < row_off[b + 1]; k++) {
                where[row[k]] = k;
                owner[row[k]] = b;
            }
        }
    });
    std::vector<int> kd_src(n, 0);
    in_parallel(nb, [&](int b0, int b1) {
        for (int b = b0; b < b1; b++) {
            Block &W = B[b];
            const int r0 = row_off[b], nr = row_off[b + 1] - r0;
            for (int k = r0; k < r0 + nr; k++)
                for (long long e = rowp[row[k]]; e < rowp[row[k] + 1]; e++)
                    if (owner[cols[e]] != b) W.halo.push_back(where[cols[e]]);
            std::sort(W.halo.begin(), W.halo.end());
            W.halo.erase(std::unique(W.halo.begin(), W.halo.end()), W.halo.end());
            W.fits = nr + W.halo.size() <= 65535 && W.halo.size() <= HALO_REGS * THREADS;
            if (!W.fits) continue;
            for (int s = 0; 32 * s < nr; s++) {
                int w = 0;
                for (int l = 0; l < 32 && 32 * s + l < nr; l++) {
                    const int q = row[r0 + 32 * s + l];
                    w = std::max(w, (int)(rowp[q + 1] - rowp[q]) - 1);
                }
                w = (w + 1) / 2;
                W.slice.push_back(w);
                const size_t at = W.col.size();
                W.col.resize(at + 32 * (size_t)w);
                W.src.resize(2 * (at + 32 * (size_t)w), -1);
                for (int l = 0; l < 32; l++) {
                    const int i = std::min(32 * s + l, nr - 1);
                    for (int k = 0; k < w; k++) W.col[at + 32 * (size_t)k + l] = (unsigned)i << 16 | i;
                    if (32 * s + l >= nr) continue;
                    const int q = row[r0 + i];
                    int k = 0;
                    for (long long e = rowp[q]; e < rowp[q + 1]; e++) {
                        const int c = cols[e];
                        if (c == q) {
                            kd_src[r0 + i] = (int)slot[e];
                            continue;
                        }
                        const int li = owner[c] == b
                                           ? where[c] - r0
                                           : nr + (int)(std::lower_bound(W.halo.begin(), W.halo.end(), where[c]) - W.halo.begin());
                        const size_t p = at + 32 * (size_t)(k >> 1) + l;
                        W.col[p] = k & 1 ? (W.col[p] & 0xffffu) | (unsigned)li << 16 : (W.col[p] & 0xffff0000u) | (unsigned)li;
                        W.src[2 * p + (k & 1)] = (int)slot[e];
                        k++;
                    }
                }
            }
            // cells; boxes; the finest level's own functions by the cells' sums
            for (int k = 0; k < nr; k++)
                if (k == 0 || cell[row[r0 + k]] != cell[row[r0 + k - 1]]) {
                    W.cell.push_back(cell[row[r0 + k]]);
                    W.cell_row.push_back(k);
                }
            W.cell_row.push_back(nr);
            W.fits = 8 * W.cell.size() < 0xffff;
            if (!W.fits) continue;
            int lo[3], hi[3];
            auto cover = [&](int c, bool fresh) {
                const int at[3] = {c % cells[0], c / cells[0] % cells[1], c / cells[0] / cells[1]};
                for (int d = 0; d < 3; d++) {
                    lo[d] = fresh ? at[d] : std::min(lo[d], at[d]);
                    hi[d] = fresh ? at[d] + 1 : std::max(hi[d], at[d] + 1);
                }
            };
            for (size_t c = 0; c < W.cell.size(); c++) cover(W.cell[c], c == 0);
            int need0[3], need1[3];
            std::copy(lo, lo + 3, need0);
            std::copy(hi, hi + 3, need1);
            for (int h : W.halo) cover(cell[row[h]], false);
            std::swap(lo, need0);
            std::swap(hi, need1);
            for (int l = 0; l < a.nlev; l++) {
                Box &X = W.box[l];
                int no = 1, nn = 1;
                for (int d = 0; d < 3; d++) {
                    if (l >= a.full) {
                        need0[d] = 0;
                        need1[d] = a.lev[l].dim[d] - 1;
                    }
                    X.own0[d] = lo[d];
                    no *= X.own[d] = l <= a.full ? hi[d] - lo[d] + 1 : 0;
                    X.need0[d] = need0[d];
                    nn *= X.need[d] = need1[d] - need0[d] + 1;
                    lo[d] >>= 1;
                    hi[d] = (hi[d] + 1) >> 1;
                    need0[d] >>= 1;
                    need1[d] = (need1[d] + 1) >> 1;
                }
                X.own_off = W.nown;
                X.need_off = W.nneed;
                W.nown += no;
                W.nneed += nn;
            }
            W.fits = W.nown <= OWN_REGS * THREADS && W.nneed <= 65535;
            if (!W.fits) continue;
            const Box &X = W.box[0];
            std::vector<unsigned short> ref(8 * (size_t)X.own[0] * X.own[1] * X.own[2], 0xffff);
            W.pos.assign(W.nown, -1);       // 0 for now: a function that some row is under
            for (size_t c = 0; c < W.cell.size(); c++)
                for (int k = 0; k < 8; k++) {
                    const int f = W.cell[c] % cells[0] + (k & 1) - X.own0[0] +
                                  X.own[0] * (W.cell[c] / cells[0] % cells[1] + ((k >> 1) & 1) - X.own0[1] +
                                              X.own[1] * (W.cell[c] / cells[0] / cells[1] + (k >> 2) - X.own0[2]));
                    unsigned short *r = &ref[8 * (size_t)f];
                    while (*r != 0xffff) r++;
                    *r = (unsigned short)(8 * c + k);
                    W.pos[f] = 0;
                }
            W.ref.resize(ref.size() / 8);
            std::memcpy(W.ref.data(), ref.data(), ref.size() * 2);
            W.sum.assign(W.nown, 0);
            for (int l = 0; l < a.full; l++) {
                const Box &F = W.box[l], &C = W.box[l + 1];
                for (int k = 0; k < C.own[0] * C.own[1] * C.own[2]; k++)
                    W.sum[C.own_off + k] = stencil({C.own0[0] + k % C.own[0], C.own0[1] + k / C.own[0] % C.own[1],
                                                    C.own0[2] + k / C.own[0] / C.own[1]},
                                                   F.own0, F.own);
                for (int z = 0; z < F.own[2]; z++)
                    for (int y = 0; y < F.own[1]; y++)
                        for (int x = 0; x < F.own[0]; x++)
                            if (!W.pos[F.own_off + x + F.own[0] * (y + F.own[1] * z)])
                                for (int k = 0; k < 8; k++)
                                    W.pos[C.own_off + ((F.own0[0] + x + (k & 1)) >> 1) - C.own0[0] +
                                          C.own[0] * (((F.own0[1] + y + ((k >> 1) & 1)) >> 1) - C.own0[1] +
                                                      C.own[1] * (((F.own0[2] + z + (k >> 2)) >> 1) - C.own0[2]))] = 0;
            }
        }
    });
    for (const Block &W : B)
        if (!W.fits) return MP_OK;

    // the shares, function by function, in block order
    auto each = [&](const Box &X, int l, bool own, auto what) {
        const int *o = own ? X.own0 : X.need0, *d = own ? X.own : X.need;
        int i = own ? X.own_off : X.need_off;
        for (int z = 0; z < d[2]; z++)
            for (int y = 0; y < d[1]; y++)
                for (int x = 0; x < d[0]; x++)
                    what(i++, a.lev[l].off + o[0] + x + a.lev[l].dim[0] * (o[1] + y + a.lev[l].dim[1] * (o[2] + z)));
    };
    std::vector<int> first(a.nfn + 1, 0);
    for (Block &W : B)
        for (int l = 0; l <= a.full; l++) each(W.box[l], l, true, [&](int i, int f) { first[f + 1] += W.pos[i] == 0; });
    for (int f = 0; f < a.nfn; f++) first[f + 1] = first[f] + (first[f + 1] + 1 & ~1);
    a.shares = first[a.nfn];
    {
        std::vector<int> next(first.begin(), first.end() - 1);
        for (Block &W : B)
            for (int l = 0; l <= a.full; l++)
                each(W.box[l], l, true, [&](int i, int f) {
                    if (W.pos[i] == 0) W.pos[i] = next[f]++;
                });
    }
    for (Block &W : B) {
        W.run.push_back(0);
        for (int l = 0; l <= a.full; l++)
            each(W.box[l], l, false, [&](int, int f) {
                for (int k = first[f]; k < first[f + 1]; k += RUN)
                    W.task.push_back((k / 2) << 3 | std::min(RUN, first[f + 1] - k) / 2);
                W.run.push_back((unsigned short)std::min<size_t>(W.task.size(), 0xffff));
            });
        if (W.task.size() > TASK_REGS * THREADS) return MP_OK;
    }

    // the blocks' arrays, one after the other
    std::vector<int> halo_off(nb + 1, 0), halo_src, slice_off(nb + 1, 0), slice_ptr(1, 0), src, cell_off(nb + 1, 0), cell_row,
        own_off(nb + 1, 0), own_pos, ref_off(nb + 1, 0), task_off(nb + 1, 0), task, run_off(nb + 1, 0);
    std::vector<unsigned short> run;
    std::vector<unsigned> col, own_sum;
    std::vector<uint4> ref;
    std::vector<Loc> loc;
    std::vector<Box> box;
    size_t total = 0;
    for (const Block &W : B) total += W.src.size();
    if (total > 0x7fffffff) return MP_OK;
    col.reserve(total / 2);
    src.reserve(total);
    for (int b = 0; b < nb; b++) {
        const Block &W = B[b];
        const int nr = row_off[b + 1] - row_off[b], nl = nr + (int)W.halo.size(), nc = (int)W.cell.size();
        a.nl_max = std::max(a.nl_max, nl);
        a.nr_max = std::max(a.nr_max, nr);
        a.need_max = std::max(a.need_max, W.nneed);
        a.nc_max = std::max(a.nc_max, nc);
        a.own_max = std::max(a.own_max, W.nown);
        a.task_max = std::max(a.task_max, (int)W.task.size());
        a.halo_max = std::max(a.halo_max, (int)W.halo.size());
        auto append = [&](auto &to, const auto &from, std::vector<int> *off) {
            to.insert(to.end(), from.begin(), from.end());
            if (off) (*off)[b + 1] = (int)to.size();
        };
        append(halo_src, W.halo, &halo_off);
        append(own_pos, W.pos, &own_off);
        append(own_sum, W.sum, nullptr);
        append(ref, W.ref, &ref_off);
        append(task, W.task, &task_off);
        append(run, W.run, &run_off);
        append(col, W.col, nullptr);
        append(src, W.src, nullptr);
        append(cell_row, W.cell_row, nullptr);
        box.insert(box.end(), W.box, W.box + a.nlev);
        for (int k = 0; k < nr; k++) loc.push_back(place[row[row_off[b] + k]]);
        for (int h : W.halo) loc.push_back(place[row[h]]);
        slice_off[b + 1] = slice_off[b] + (int)W.slice.size();
        for (int w : W.slice) slice_ptr.push_back(slice_ptr.back() + 32 * w);
        cell_off[b + 1] = cell_off[b] + nc;
    }
    for (const Block &W : B)
        a.u_max = std::max({a.u_max, a.nr_max + 8 * (int)W.cell.size() + W.nown, (int)W.task.size() + W.nneed});
    // the rows of each cell, over the blocks
    std::vector<int> seg_ptr(1, 0);
    std::vector<Seg> seg;
    {
        std::vector<std::vector<Seg>> of(ncells);
        for (int b = 0; b < nb; b++)
            for (size_t c = 0; c < B[b].cell.size(); c++)
                of[B[b].cell[c]].push_back(
                    {row_off[b] + B[b].cell_row[c], B[b].cell_row[c + 1] - B[b].cell_row[c], b});
        for (int c = 0; c < ncells; c++) {
            seg.insert(seg.end(), of[c].begin(), of[c].end());
            seg_ptr.push_back((int)seg.size());
        }
    }

    a.n = n;
    a.nb = nb;
    a.first = where[0];
    p->ncell = ncells;
    p->rows_max = a.nr_max;
    p->slots = (int)total;
    p->smem = sizeof(Place) * a.nl_max + sizeof(double) * (2 * (size_t)a.nl_max + 3 * (size_t)a.need_max + a.u_max + 4 * WARPS + 4) +
              sizeof(unsigned) * a.need_max + sizeof(unsigned short) * (a.need_max + 1 + a.nc_max + 1 + (a.need_max + a.nc_max & 1)) +
              sizeof(int) * (2 * a.own_max + a.task_max + a.halo_max + a.nr_max / 32 + 2);
    const size_t most = SMEM_MAX;
    if (p->smem > most || a.nfn - a.lev[a.full].off - a.lev[a.full].n > FULL_MAX) return MP_OK;
    int columns = 0;
    for (int b = 0; b < nb; b++) columns = std::max(columns, (slice_ptr[slice_off[b + 1]] - slice_ptr[slice_off[b]]) / 32);
    const size_t column = 32 * (sizeof(double2) + sizeof(unsigned));
    a.hold = std::min(columns, (int)((most - p->smem) / column));
    p->smem += a.hold * column;

#define CG_ARRAYS(X)                                                                                                      \
    X(row) X(row_off) X(halo_off) X(halo_src) X(slice_off) X(slice_ptr) X(col) X(src) X(kd_src) X(loc) X(box) X(cell_off) \
        X(cell_row) X(own_off) X(own_pos) X(own_sum) X(ref_off) X(ref) X(task_off) X(task) X(run_off) X(run) X(seg_ptr) X(seg)
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off = (off + bytes + 255) & ~size_t(255);
        return o;
    };
#define X(v) const size_t o_##v = take(v.size() * sizeof(v[0]));
    CG_ARRAYS(X)
#undef X
    if (!device_room((void **)&p->blob, off)) return MP_OK;  // unusable, no error
    unsigned char *base = static_cast<unsigned char *>(p->blob);
#define X(v) \
    if (!v.empty()) MP_CUDA(ctx, upload(ctx, base + o_##v, v.data(), v.size() * sizeof(v[0])));
    CG_ARRAYS(X)
#undef X
#undef CG_ARRAYS
#define X(m, v) a.m = reinterpret_cast<decltype(a.m)>(base + o_##v);
    X(row, row) X(row_off, row_off) X(halo_off, halo_off) X(halo_src, halo_src) X(slice_off, slice_off) X(slice_ptr, slice_ptr)
    X(col, col) X(loc, loc) X(box, box) X(cell_off, cell_off) X(cell_row, cell_row) X(own_off, own_off) X(own_pos, own_pos) X(own_sum, own_sum)
    X(ref_off, ref_off) X(ref, ref) X(task_off, task_off) X(task, task) X(run_off, run_off) X(run, run)
#undef X
    p->src = reinterpret_cast<const int *>(base + o_src);
    p->kd_src = reinterpret_cast<const int *>(base + o_kd_src);
    p->seg_ptr = reinterpret_cast<const int *>(base + o_seg_ptr);
    p->seg = reinterpret_cast<const Seg *>(base + o_seg);

    off = 0;
    const size_t o_val = take(8 * total), o_kd = take(8 * (size_t)n), o_e = take(8 * 36 * (size_t)ncells),
                 o_dk = take(8 * (size_t)a.nfn), o_pub = take(16 * (size_t)n), o_share = take(16 * (size_t)a.shares),
                 o_sums = take(8 * 8 * (size_t)nb), o_flag = take(4);
    if (!device_room((void **)&p->val, off)) return MP_OK;
    base = reinterpret_cast<unsigned char *>(p->val);
    auto at = [&](size_t o) { return reinterpret_cast<double *>(base + o); };
    p->kd = at(o_kd);
    p->e = at(o_e);
    p->dk = at(o_dk);
    a.val = reinterpret_cast<const double2 *>(p->val);
    a.kd = p->kd;
    a.dk = p->dk;
    a.pub = at(o_pub);
    a.share = at(o_share);
    a.sums = at(o_sums);
    a.flag = reinterpret_cast<unsigned *>(base + o_flag);
    MP_CUDA(ctx, cudaMemsetAsync(a.share, 0, 16 * (size_t)a.shares, ctx->stream));  // the odd functions' last places stay zero
    MP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    p->usable = true;
    return MP_OK;
}

// Builds the plan from K's pattern (CSR rows, columns ascending; slot[k] an
// entry's place in sp_val).  It is left unusable for fewer than ROWS_FROM rows, for
// a thin box between fixed planes, and where a block would not hold its rows or
// memory is short.
int cg_levels_setup(mp_ctx *ctx, const std::vector<long long> &rowp, const std::vector<int> &cols,
                    const std::vector<long long> &slot) {
    cg_levels_free(ctx);
    Plan *p = new Plan();
    ctx->cg_levels = p;
    int rc = MP_OK;
    try {
        rc = make_plan(ctx, p, rowp, cols, slot);
    } catch (const std::exception &) {
    }
    if (!p->usable) {
        void *dev[] = {p->blob, p->val};
        for (void *q : dev)
            if (q) cudaFree(q);
        p->blob = nullptr;
        p->val = nullptr;
    }
    return rc;
}

template <int RPT>
static cudaError_t launch(const Plan *p, Args a, cudaStream_t stream) {
    // the attribute is the function's, shared by all contexts: what any plan may need, so that
    // one thread's launch never finds another's smaller limit
    cudaError_t e = cudaFuncSetAttribute(k_cg_levels<RPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX);
    if (e != cudaSuccess) return e;
    void *args[] = {&a};
    return cudaLaunchCooperativeKernel((const void *)k_cg_levels<RPT>, dim3(a.nb), dim3(THREADS), args, p->smem, stream);
}

// J y = G with FP's current J.  *done: enqueued (the plan is usable).  sync: two
// cleared words, abort and status; out: iterations, ||r||^2, ||G||^2, restarts.
int cg_levels_enqueue(mp_ctx *ctx, unsigned *sync, double *out, bool *done) {
    *done = false;
    if (!ctx->cg_levels && !ctx->csr_ptr.empty()) {
        const int rc = cg_levels_setup(ctx, ctx->csr_ptr, ctx->csr_col, ctx->csr_slot);
        if (rc) return rc;
    }
    Plan *p = plan_of(ctx);
    if (!p || !p->usable) return MP_OK;
    Args a = p->a;
    a.FP = ctx->FP;
    a.b = ctx->G;
    a.x = ctx->y;
    a.sync = sync;
    a.out = out;
    a.rtol2 = ctx->cg_rtol * ctx->cg_rtol;
    a.max_it = ctx->cg_max_it;
    cudaStream_t st = ctx->stream;
    if (!p->formed || p->changes != ctx->sp_changes) {
        const int m = std::max(p->slots, a.n);
        k_levels_gather<<<(m + 255) / 256, 256, 0, st>>>(p->slots, a.n, p->src, p->kd_src, ctx->sp_val, p->val, p->kd),
            ++ctx->launches;
        k_levels_cells<<<(p->ncell + 15) / 16, 128, 0, st>>>(a, p->ncell, p->seg_ptr, p->seg, p->e), ++ctx->launches;
        k_levels_diag<<<(a.nfn + 3) / 4, 128, 0, st>>>(a, p->e, p->dk), ++ctx->launches;
        p->formed = true;
        p->changes = ctx->sp_changes;
    }
    MP_CUDA(ctx, cudaMemsetAsync(a.flag, 0, sizeof(unsigned), st));
    const int rpt = (p->rows_max + THREADS - 1) / THREADS;
    const cudaError_t e = rpt == 1 ? launch<1>(p, a, st) : rpt == 2 ? launch<2>(p, a, st) : launch<4>(p, a, st);
    MP_CUDA(ctx, e);
    ++ctx->launches;
    *done = true;
    return MP_OK;
}

}  // namespace mp
