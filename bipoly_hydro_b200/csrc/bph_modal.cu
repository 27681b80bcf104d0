// bph_modal.cu -- the FP64 ADI of every Fourier slot in the vertical
// eigenbasis.
//
// A slot's operator is A = A_r (x) I + I (x) A_z with A_z = gamma T the same
// for every slot, and T has closed-form eigenvectors (bph_direct.h).  The
// Peaceman-Rachford half-steps of helmadi.F90:195-355 are rational functions
// of A_r and A_z, which commute, so on vertical mode q (eigenvalue lambda_q)
// one whole step of the iteration is
//   delta = (A_r + dt)^-1 r,
//   phi  += 2 dt / (dt + lambda_q) delta,
//   r     = (dt - lambda_q) / (dt + lambda_q) (2 dt delta - r),
// with r the residual of the current potential (r = R - A phi at the start,
// Dirichlet terms included): a radial solve whose matrix is the radial
// half-step's own and the same for every q, and two elementwise updates.
// The vertical half-steps, the right-hand sides and the exchange of the slot
// between row and column order after every half-step are gone, and the cost
// of a step no longer depends on where the slot fits.  A solve is
//   k_modal_fwd     r = R - A phi in physical space, transformed: Y = E r
//   k_modal_radial  every step of one line (slot, mode) in registers
//   k_modal_inv     phi += E^T Y
// Rounding differs from the half-step form (no 1/(dt + lambda) amplification
// of the radially stiff components); the iteration is the same one.
//
// The mixed form's refinement takes the half-steps in another order: a radial
// one at the first dt, then (vertical, radial) per step, so that a cycle ends
// on the radial solve, which the radially stiff components of the residual
// need (ended on the vertical one, its residual was 2e-10 for 1e-13 at
// 66 x 66 x 64).  Paired radial first, its n + 1 radial solves (dt a) and n
// vertical ones (dt b) are the step above with two dt:
//   phi += (a + b) / (b + lambda_q) delta,
//   r     = (a - lambda_q) / (b + lambda_q) ((a + b) delta - r),
// and the last solve alone phi += delta, r = (a - lambda_q) delta.
//
// The transforms are the matrix products of the path (2 nz FMA per zone each)
// and run on the FP64 tensor cores, mma.sync m16n8k8.f64: 37 TFLOP/s
// measured for the instruction alone against 33 for FMA.
#include <cmath>
#include <cstdlib>
#include <vector>

#include "bph_internal.cuh"

namespace bph {

static int modal_ldq(const bph_ctx *c);

namespace {

constexpr int kLines = 32;      // radial lines per block: one per lane
constexpr int kMaxSegs = 16;    // warps of a radial block

struct ModalArgs {
    const double *E;         // packed A fragments of E (forward) or E^T (inverse)
    double *P;               // slot arrays [inst][N][nplane]
    const double *R;         // [inst][N][np]
    double *Y;               // modal arrays [row][N][nr][ldq], column q = mode
    double *phi;             // converged form: modal potential, the same layout
    double *pre;             // converged form: the potential before the cycle's last step
    const double *brb;       // [N][numr]
    const double *alphar;    // [numr]
    const double *betar;     // [numr]
    const int *inst_map;     // instance of each row (nullptr: inst0 + row)
    const int *slot_map;     // slot of each block within a row (nullptr: block = slot)
    const double *rad;       // [nsteps][N][block] radial factors
    const double2 *cs;       // [nsteps][nz] (2 dt / (dt + lambda), (dt - lambda) / (dt + lambda))
    const double *dt2;       // [nsteps] 2 dt
    double *norms;           // converged form: [row][N][groups][2]
    const int *skip;         // converged form: not 0: nothing to do (nullptr: always run)
    int inst0, nslots, ntile, groups;
    int numr, numz, nr, nz, ldq, N, isym, mtiles, ksteps;
    int nsteps, source, add;
    unsigned half;           // forward transform: blocks from this one on take the potential into phi
    unsigned ahead;          // blocks of the kernel that the device holds at a time
    int lagged;              // converged form: the refinement's half-step order (nsteps counts its radial solves)
    double gamma;
    // split transforms (p1 > 0)
    const double *Cs;        // packed A fragments of the cosine matrix, then of the sine matrix
    const int *tab;          // [p1][h2]: +-(k + 1) of (a1, a2), 0: none
    int h2, mt2, ks2;        // rows of the second factor's matrices, their 16-row tiles and 8-row steps
    double s1[4][4], c1[4][4];  // sines and cosines of the first factor
};


// What k_modal_fwd transforms.
enum { kResidual = 0, kColdResidual = 1, kPotential = 2 };

__device__ __forceinline__ void dmma(double *c, const double2 &a01, const double2 &a23, double b0, double b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a01.x), "d"(a01.y), "d"(a23.x), "d"(a23.y), "d"(b0), "d"(b1));
}

// Rows of 8 NT columns, padded to 4 modulo the 16 eight-byte banks: the four
// rows of a B fragment then fall into different banks.
template <int NT>
struct TileShape {
    static constexpr int cols = 8 * NT;
    static constexpr int ld = cols + 4;
};

struct TileIndex {
    int tile, slot, row;
    long long inst;
};
__device__ __forceinline__ TileIndex tile_index(const ModalArgs &a, int per_slot, unsigned block) {
    TileIndex t;
    t.tile = block % per_slot;
    const int b = block / per_slot;
    const int local = b % a.nslots;
    t.row = b / a.nslots;
    t.slot = a.slot_map ? a.slot_map[local] : local;
    t.inst = a.inst_map ? a.inst_map[t.row] : a.inst0 + t.row;
    return t;
}

// acc = A(mt) X for the 16 rows of tile mt and every column of the tile in
// shared memory.  The A fragments come from L1/L2 (E is shared by every
// block), one k-step ahead; a 16 x 8 x 8 product holds the tensor pipe for 64
// cycles, so neither operand's path limits it.
// B (k, n) sits at sx[k * kstr + n * nstr].
template <int NT>
__device__ __forceinline__ void tile_product(const ModalArgs &a, const double *sx, int kstr, int nstr, int mt, int lane,
                                             double (*acc)[4]) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[n][v] = 0.0;
    const double2 *ap = reinterpret_cast<const double2 *>(a.E + (long long)mt * a.ksteps * 128) + 2 * lane;
    double2 a01 = __ldg(ap), a23 = __ldg(ap + 1);
    const double *bp = sx + t * kstr + g * nstr;
    for (int ks = 0; ks < a.ksteps; ++ks) {
        double2 n01 = a01, n23 = a23;
        if (ks + 1 < a.ksteps) {
            n01 = __ldg(ap + 64 * (ks + 1));
            n23 = __ldg(ap + 64 * (ks + 1) + 1);
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) dmma(acc[n], a01, a23, bp[8 * n * nstr], bp[4 * kstr + 8 * n * nstr]);
        bp += 8 * kstr;
        a01 = n01;
        a23 = n23;
    }
}

// What a block transforms, 8 NT columns of a slot with all rows, into
// sx[row][column]: the residual is formed once per column tile, a warp per
// band of rows with the rows below and at hand kept in registers.  Waits for
// the previous kernel.
template <int NT>
__device__ __forceinline__ void source_tile(const ModalArgs &a, int source, const TileIndex &ti, double *sx) {
    constexpr int ld = TileShape<NT>::ld;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int nr = a.nr, nz = a.nz, numr = a.numr, j0 = ti.tile * TileShape<NT>::cols;
    const long long np = (long long)nr * nz, nplane = (long long)numr * a.numz;
    const double *__restrict__ Pg = a.P + (ti.inst * a.N + ti.slot) * nplane;
    const double *__restrict__ Rs = a.R + (ti.inst * a.N + ti.slot) * np;
    const bool dirichlet = a.isym == 1;
    const int per = (nz + nwarps - 1) / nwarps, k0 = warp * per, k1 = min(nz, k0 + per);
    pdl_wait();
    for (int cc = lane; cc < TileShape<NT>::cols; cc += 32) {
        const int j = j0 + cc;
        if (j >= nr) {
            for (int k = k0; k < k1; ++k) sx[k * ld + cc] = 0.0;
            continue;
        }
        const double al = a.alphar[j + 1], be = a.betar[j + 1], bd = a.brb[(long long)ti.slot * numr + j + 1];
        const double *p = Pg + (j + 1);
        if (source == kResidual) {
            double dn = 0.0, cur = 0.0;
            if (k0 < k1) {
                dn = (k0 > 0 || dirichlet) ? p[(long long)k0 * numr] : 0.0;
                cur = p[(long long)(k0 + 1) * numr];
            }
#pragma unroll 8
            for (int k = k0; k < k1; ++k) {
                const double *pk = p + (long long)(k + 1) * numr;
                const double up = pk[numr], east = pk[1], west = (j > 0) ? pk[-1] : 0.0;
                const double diag = (k == 0 && !dirichlet) ? cur : 2.0 * cur;
                const double ar = bd * cur + al * east + be * west;
                sx[k * ld + cc] = (Rs[(long long)k * nr + j] - ar) - a.gamma * (diag - up - dn);
                dn = cur;
                cur = up;
            }
        } else if (source == kColdResidual) {
#pragma unroll 4
            for (int k = k0; k < k1; ++k) {
                double v = Rs[(long long)k * nr + j];
                if (k == nz - 1) v += a.gamma * p[(long long)(nz + 1) * numr];
                if (k == 0 && dirichlet) v += a.gamma * p[0];
                if (j == nr - 1) v -= al * p[(long long)(k + 1) * numr + 1];
                sx[k * ld + cc] = v;
            }
        } else {
#pragma unroll 4
            for (int k = k0; k < k1; ++k) sx[k * ld + cc] = p[(long long)(k + 1) * numr];
        }
    }
}

// Block: 8 NT columns of a slot; the tile stays in shared memory as the B
// operand.
template <int NT>
__global__ void __launch_bounds__(256) k_modal_fwd(ModalArgs a) {
    extern __shared__ double sx[];
    constexpr int ld = TileShape<NT>::ld;
    const bool second = blockIdx.x >= a.half;
    const TileIndex ti = tile_index(a, a.ntile, second ? blockIdx.x - a.half : blockIdx.x);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int nr = a.nr, nz = a.nz, j0 = ti.tile * TileShape<NT>::cols;
    for (int e = threadIdx.x; e < (8 * a.ksteps - nz) * ld; e += blockDim.x) sx[nz * ld + e] = 0.0;
    source_tile<NT>(a, second ? kPotential : a.source, ti, sx);
    __syncthreads();
    double *Yb = (second ? a.phi : a.Y) + ((long long)ti.row * a.N + ti.slot) * nr * a.ldq;
    const int g = lane >> 2, t = lane & 3;
    for (int mt = warp; mt < a.mtiles; mt += nwarps) {
        double acc[NT][4];
        tile_product<NT>(a, sx, ld, 1, mt, lane, acc);
        if (mt + nwarps >= a.mtiles) pdl_trigger();
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int j = j0 + 8 * n + 2 * t + (v & 1), q = 16 * mt + g + 8 * (v >> 1);
                if (q < nz && j < nr) Yb[(long long)j * a.ldq + q] = acc[n][v];
            }
    }
}

// Block: 8 NT columns of a slot: P (+)= E^T Y.  The tile keeps the modal
// array's order [column][mode] in shared memory (16-byte copies), rows 4
// modulo 16 words apart.
__host__ __device__ inline int inv_ld(int ksteps) { return (8 * ksteps + 15) / 16 * 16 + 4; }

template <int NT>
__global__ void __launch_bounds__(256) k_modal_inv(ModalArgs a) {
    extern __shared__ __align__(16) double sx[];
    const int ld = inv_ld(a.ksteps);
    const TileIndex ti = tile_index(a, a.ntile, blockIdx.x);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int nr = a.nr, nz = a.nz, numr = a.numr, j0 = ti.tile * TileShape<NT>::cols;
    const long long nplane = (long long)numr * a.numz;
    const double *Yb = a.Y + (((long long)ti.row * a.N + ti.slot) * nr + j0) * a.ldq;
    double *Pg = a.P + (ti.inst * a.N + ti.slot) * nplane;
    pdl_wait();
    for (int cc = warp; cc < TileShape<NT>::cols; cc += nwarps) {
        double *row = sx + cc * ld;
        if (j0 + cc < nr) {
            for (int q = 2 * lane; q < a.ldq; q += 64) {
                const unsigned d = (unsigned)__cvta_generic_to_shared(row + q);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(Yb + (long long)cc * a.ldq + q));
            }
        }
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int cc = warp; cc < TileShape<NT>::cols; cc += nwarps) {  // modes and columns past the slot
        const int from = (j0 + cc < nr) ? nz : 0;
        for (int q = from + lane; q < 8 * a.ksteps; q += 32) sx[cc * ld + q] = 0.0;
    }
    __syncthreads();
    const int g = lane >> 2, t = lane & 3;
    for (int mt = warp; mt < a.mtiles; mt += nwarps) {
        double *p = Pg + (long long)(16 * mt + g + 1) * numr + j0 + 2 * t + 1;
        const bool k0 = 16 * mt + g < nz, k1 = 16 * mt + g + 8 < nz;
        double old[NT][4], acc[NT][4];  // the old potential arrives under the products
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int v = 0; v < 4; ++v)
                old[n][v] = (a.add && (v < 2 ? k0 : k1) && j0 + 8 * n + 2 * t + (v & 1) < nr)
                                ? p[(v >> 1) * 8 * numr + 8 * n + (v & 1)]
                                : 0.0;
        tile_product<NT>(a, sx, 1, ld, mt, lane, acc);
        if (mt + nwarps >= a.mtiles) pdl_trigger();
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int v = 0; v < 4; ++v)
                if ((v < 2 ? k0 : k1) && j0 + 8 * n + 2 * t + (v & 1) < nr)
                    p[(v >> 1) * 8 * numr + 8 * n + (v & 1)] = old[n][v] + acc[n][v];
    }
}

// ---- split transforms ---------------------------------------------------
//
// With a reflecting bottom E[q][k] = 2 / sqrt(L) cos(2 pi (2k+1)(2q+1) / (4L)),
// L = 2 nz + 1.  The sign of 2k+1 is free, so take a = +-(2k+1) and b =
// +-(2q+1) congruent to 1 modulo 4; then the entry is +-sin(2 pi beta a b / L)
// with 4 beta = 1 modulo L: a sine transform of odd functions on Z/L.  Where
// L = p1 p2 with coprime factors, a = (a1, a2) by remainders (Good 1958,
// Thomas 1963) and
//   sin(2 pi beta a b / L) = sin1(a1 b1) cos2(a2 b2) + cos1(a1 b1) sin2(a2 b2),
// so the matrix product becomes p1 products of size (p2 + 1) / 2:
//   P(b1, a2) = sum_a1 f(a1, a2) sin1(a1 b1),  Q likewise with cos1,
//   Y(+-b1, b2) = sum_a2 Q sin2(a2 b2) +- P cos2(a2 b2),
// a2 and b2 in 0 .. (p2 - 1) / 2, b1 in 0 .. (p1 - 1) / 2.  The sums over a1
// are a few FMA per zone, in place in the tile; the products stay on the
// tensor cores (192 heights, 385 = 7 x 55: 56 of 288 fragment products).  The
// modal array's columns are ordered by (b1, sign, b2), so that both kernels
// move whole runs of it; the order and the signs of the modes mean nothing to
// the radial steps.
__host__ __device__ inline int run_plus(int b1, int h2) { return b1 == 0 ? -1 : (h2 - 1) + (b1 - 1) * (2 * h2 - 1); }
__host__ __device__ inline int run_minus(int b1, int h2) { return run_plus(b1, h2) + h2 - 1; }

// The sums over a1 of one column and a2, in place: at(a1) is the place of
// f(a1, a2), sg(a1) its sign (0: no such value).
template <int P1, class At, class Sg>
__device__ __forceinline__ void first_factor(const ModalArgs &a, int a2, At at, Sg sg) {
    constexpr int h = (P1 - 1) / 2;
    double f[P1], *place[P1];
#pragma unroll
    for (int i = 0; i < P1; ++i) {
        const double w = sg(i);
        place[i] = at(i);
        f[i] = w != 0.0 ? w * *place[i] : 0.0;
    }
    double P[h + 1], Q[h + 1];
    Q[0] = f[0];
#pragma unroll
    for (int i = 1; i <= h; ++i) Q[0] += f[i] + f[P1 - i];
#pragma unroll
    for (int b = 1; b <= h; ++b) {
        P[b] = 0.0;
        Q[b] = f[0];
#pragma unroll
        for (int i = 1; i <= h; ++i) {
            P[b] = fma(f[i] - f[P1 - i], a.s1[i][b], P[b]);
            Q[b] = fma(f[i] + f[P1 - i], a.c1[i][b], Q[b]);
        }
    }
    if (a2 > 0) *place[0] = Q[0];
#pragma unroll
    for (int b = 1; b <= h; ++b) {
        *place[b] = P[b];
        if (a2 > 0) *place[P1 - b] = Q[b];
    }
}

// accP = cos2 P, accQ = sin2 Q for row tile mt; the row of (group, a2) and
// column n starts at px[...], qx[...] (one offset per lane and step).
template <int NT, class Row>
__device__ __forceinline__ void second_factor(const ModalArgs &a, const double *sx, int nstr, int mt, int lane, bool with_p,
                                              Row row, double (*accP)[4], double (*accQ)[4]) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int v = 0; v < 4; ++v) accP[n][v] = accQ[n][v] = 0.0;
    const double2 *cp = reinterpret_cast<const double2 *>(a.Cs + (long long)mt * a.ks2 * 128) + 2 * lane;
    const double2 *sp = cp + (long long)a.mt2 * a.ks2 * 64;
    const double *bp = sx + g * nstr;
    for (int ks = 0; ks < a.ks2; ++ks) {
        const int r0 = 8 * ks + t, r1 = r0 + 4;
        {
            const double2 a01 = __ldg(sp + 64 * ks), a23 = __ldg(sp + 64 * ks + 1);
            const double *b0 = bp + row(false, r0), *b1 = bp + row(false, r1);
#pragma unroll
            for (int n = 0; n < NT; ++n) dmma(accQ[n], a01, a23, b0[8 * n * nstr], b1[8 * n * nstr]);
        }
        if (with_p) {
            const double2 a01 = __ldg(cp + 64 * ks), a23 = __ldg(cp + 64 * ks + 1);
            const double *b0 = bp + row(true, r0), *b1 = bp + row(true, r1);
#pragma unroll
            for (int n = 0; n < NT; ++n) dmma(accP[n], a01, a23, b0[8 * n * nstr], b1[8 * n * nstr]);
        }
    }
}

// Asks L2 for rows of count doubles, stride apart: what the block that takes
// this one's place will load.  With one or two blocks per SM nothing else
// covers the HBM latency at a block's start (five steps at 258 x 194 x 512:
// 660 -> 655 us by the transforms' sources, -> 634 with the radial lines; the
// inverse's own old potential, asked for under its products, cost 4 us).
__device__ __forceinline__ void prefetch_rows(const double *p, long long stride, int rows, int count) {
    const int lines = (count + 14) / 16 + 1;  // 128-byte lines that an unaligned row can touch
    for (int i = threadIdx.x; i < rows * lines; i += blockDim.x) {
        const double *at = p + (i / lines) * stride + min(16 * (i % lines), count - 1);
        asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
    }
}

template <int NT, int P1>
__global__ void __launch_bounds__(256, 2) k_modal_fwd_split(ModalArgs a) {
    extern __shared__ double sx[];
    constexpr int ld = TileShape<NT>::ld, cols = TileShape<NT>::cols, h = (P1 - 1) / 2;
    const bool second = blockIdx.x >= a.half;
    const TileIndex ti = tile_index(a, a.ntile, second ? blockIdx.x - a.half : blockIdx.x);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int nr = a.nr, nz = a.nz, h2 = a.h2, k2 = 8 * a.ks2, j0 = ti.tile * cols;
    int *tab = reinterpret_cast<int *>(sx + nz * ld);  // [P1][h2]
    int *rows = tab + P1 * h2;                         // [Q0 .. Qh, P1 .. Ph][k2]: row offsets
    for (int i = threadIdx.x; i < P1 * h2; i += blockDim.x) tab[i] = a.tab[i];
    for (int i = threadIdx.x; i < P1 * k2; i += blockDim.x) {
        // past h2 the matrices are zero, and so is the sine's first column: any row will do there
        const int grp = i / k2, a2 = min(i % k2, h2 - 1);
        const int a1 = grp == 0 ? 0 : grp <= h ? P1 - grp : grp - h;
        const int at = (grp <= h && a2 == 0) ? 1 : a2;
        rows[i] = (abs(a.tab[a1 * h2 + at]) - 1) * ld;
    }
    source_tile<NT>(a, second ? kPotential : a.source, ti, sx);
    if (blockIdx.x + a.ahead < gridDim.x) {
        const unsigned next = blockIdx.x + a.ahead;
        const int source = next >= a.half ? kPotential : a.source;
        const TileIndex tn = tile_index(a, a.ntile, next >= a.half ? next - a.half : next);
        const int jn = tn.tile * cols, count = min(cols, nr - jn);
        const long long at = tn.inst * a.N + tn.slot;
        if (source != kPotential) prefetch_rows(a.R + at * nr * nz + jn, nr, nz, count);
        if (source != kColdResidual)
            prefetch_rows(a.P + at * a.numr * a.numz + a.numr + jn + 1, a.numr, nz, count);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < h2 * cols; i += blockDim.x) {
        const int c = i % cols, a2 = i / cols;
        first_factor<P1>(
            a, a2, [&](int a1) { return sx + max(abs(tab[a1 * h2 + a2]) - 1, 0) * ld + c; },
            [&](int a1) {
                const int t = tab[a1 * h2 + a2];
                return t > 0 ? 1.0 : t < 0 ? -1.0 : 0.0;
            });
    }
    __syncthreads();
    double *Yb = (second ? a.phi : a.Y) + ((long long)ti.row * a.N + ti.slot) * nr * a.ldq;
    const int g = lane >> 2, t = lane & 3;
    for (int u = warp; u < (h + 1) * a.mt2; u += nwarps) {
        const int b1 = u / a.mt2, mt = u % a.mt2;
        double accP[NT][4], accQ[NT][4];
        const int *rq = rows + b1 * k2, *rp = rows + (h + b1) * k2;
        second_factor<NT>(a, sx, 1, mt, lane, b1 > 0, [&](bool p, int r) { return p ? rp[r] : rq[r]; }, accP, accQ);
        if (u + nwarps >= (h + 1) * a.mt2) pdl_trigger();
        const int plus = run_plus(b1, h2), minus = run_minus(b1, h2);
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int j = j0 + 8 * n + 2 * t + (v & 1), b2 = 16 * mt + g + 8 * (v >> 1);
                if (b2 >= h2 || j >= nr) continue;
                double *y = Yb + (long long)j * a.ldq + b2;
                if (b1 > 0 || b2 > 0) y[plus] = accQ[n][v] + accP[n][v];
                if (b1 > 0 && b2 > 0) y[minus] = accQ[n][v] - accP[n][v];
            }
    }
}

template <int NT, int P1>
__global__ void __launch_bounds__(256, 2) k_modal_inv_split(ModalArgs a) {
    extern __shared__ __align__(16) double sx[];
    constexpr int cols = TileShape<NT>::cols, h = (P1 - 1) / 2;
    const int ld = inv_ld(a.ksteps);
    const TileIndex ti = tile_index(a, a.ntile, blockIdx.x);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int nr = a.nr, nz = a.nz, numr = a.numr, h2 = a.h2, j0 = ti.tile * cols;
    int *tab = reinterpret_cast<int *>(sx + cols * ld);
    for (int i = threadIdx.x; i < P1 * h2; i += blockDim.x) tab[i] = a.tab[i];
    const double *Yb = a.Y + (((long long)ti.row * a.N + ti.slot) * nr + j0) * a.ldq;
    double *Pg = a.P + (ti.inst * a.N + ti.slot) * (long long)numr * a.numz;
    pdl_wait();
    for (int cc = warp; cc < cols; cc += nwarps) {
        double *row = sx + cc * ld;
        if (j0 + cc < nr) {
            for (int q = 2 * lane; q < a.ldq; q += 64) {
                const unsigned d = (unsigned)__cvta_generic_to_shared(row + q);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(Yb + (long long)cc * a.ldq + q));
            }
        } else {
            for (int q = lane; q < nz; q += 32) row[q] = 0.0;
        }
    }
    if (blockIdx.x + a.ahead < gridDim.x) {
        const TileIndex tn = tile_index(a, a.ntile, blockIdx.x + a.ahead);
        const int jn = tn.tile * cols;
        prefetch_rows(a.Y + (((long long)tn.row * a.N + tn.slot) * nr + jn) * a.ldq, a.ldq, min(cols, nr - jn), a.ldq);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int cc = warp; cc < cols; cc += nwarps)
        for (int a2 = lane; a2 < h2; a2 += 32)
            first_factor<P1>(
                a, a2,
                [&](int a1) {
                    const int at = a1 == 0 ? a2 - 1 : a1 <= h ? run_plus(a1, h2) + a2 : run_minus(P1 - a1, h2) + a2;
                    return sx + cc * ld + max(at, 0);
                },
                [&](int a1) { return a2 > 0 || (a1 > 0 && a1 <= h) ? 1.0 : 0.0; });
    __syncthreads();
    const int g = lane >> 2, t = lane & 3;
    for (int u = warp; u < (h + 1) * a.mt2; u += nwarps) {
        const int b1 = u / a.mt2, mt = u % a.mt2;
        const int plus = run_plus(b1, h2), minus = b1 == 0 ? -1 : run_minus(b1, h2);
        double accP[NT][4], accQ[NT][4];
        // past h2 the matrices are zero, and so is the sine's first column: any value will do there
        second_factor<NT>(a, sx, ld, mt, lane, b1 > 0,
                          [&](bool p, int r) { return p ? plus + min(r, h2 - 1) : minus + max(min(r, h2 - 1), 1); }, accP,
                          accQ);
        if (u + nwarps >= (h + 1) * a.mt2) pdl_trigger();
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            if (side && b1 == 0) break;
            double old[NT][4];
            int tr[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int b2 = 16 * mt + g + 8 * r;
                tr[r] = (b2 < h2 && !(side && b2 == 0)) ? tab[(side ? P1 - b1 : b1) * h2 + b2] : 0;
            }
            double *p = Pg + j0 + 2 * t + 1;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    old[n][v] = (a.add && tr[v >> 1] && j0 + 8 * n + 2 * t + (v & 1) < nr)
                                    ? p[(long long)abs(tr[v >> 1]) * numr + 8 * n + (v & 1)]
                                    : 0.0;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    if (tr[v >> 1] && j0 + 8 * n + 2 * t + (v & 1) < nr) {
                        const double x = side ? accQ[n][v] - accP[n][v] : accQ[n][v] + accP[n][v];
                        p[(long long)abs(tr[v >> 1]) * numr + 8 * n + (v & 1)] = old[n][v] + (tr[v >> 1] > 0 ? x : -x);
                    }
        }
    }
}

// Radial factor block of one (step, slot): per radius the pairs (1/bet,
// -a/bet) of the way down, the pairs (-gam_{j+1}, G) of the way up with the
// forward segment carry, then the backward carries K; padded to `rows` radii
// with zeros.
__host__ __device__ constexpr int radial_block(int rows) { return 5 * rows; }

__global__ void k_pack_modal(const double *__restrict__ rad, double *__restrict__ out, int nr, int nseg, int seg) {
    // one block per (step, slot), one thread per segment
    const int rows = nseg * seg;
    const double *src = rad + (long long)blockIdx.x * kAdiFactors * nr;
    double *dst = out + (long long)blockIdx.x * radial_block(rows);
    double *back = dst + 2 * rows, *kk = dst + 4 * rows;
    const int s = threadIdx.x;
    double G = 1.0, K = 1.0;
    for (int e = 0; e < seg; ++e) {
        const int j = s * seg + e;
        const bool in = j < nr;
        const double dd = in ? -src[nr + j] : 0.0;
        G = in ? G * dd : 0.0;
        dst[2 * j] = in ? src[j] : 0.0;
        dst[2 * j + 1] = dd;
        back[2 * j] = (j + 1 < nr) ? -src[2 * nr + j + 1] : 0.0;
        back[2 * j + 1] = G;
    }
    for (int e = seg - 1; e >= 0; --e) {
        const int j = s * seg + e;
        K = (j + 1 < nr) ? K * -src[2 * nr + j + 1] : 0.0;
        kk[j] = K;
    }
}

// Step coefficients: blocks 0 .. nsteps - 1 the schedule's steps, the nsteps + 1
// after them the refinement's radial solves.
__global__ void k_modal_coef(const double *__restrict__ dt, const double *__restrict__ lam, double2 *__restrict__ cs,
                             double *__restrict__ dt2, int nz, int nsteps) {
    const int i = (int)blockIdx.x - nsteps;  // refinement solve
    const bool alone = i == nsteps;
    const double a = dt[i < 0 ? (int)blockIdx.x : i > 0 ? i - 1 : 0], b = i < 0 ? a : alone ? 0.0 : dt[i];
    if (threadIdx.x == 0) dt2[blockIdx.x] = alone ? 1.0 : a + b;
    for (int q = threadIdx.x; q < nz; q += blockDim.x) {
        const double den = b + lam[q];
        cs[(long long)blockIdx.x * nz + q] =
            alone ? make_double2(1.0, a - lam[q]) : make_double2((a + b) / den, (a - lam[q]) / den);
    }
}

// All steps of a group of lines (one slot, 32 modes) in registers: a lane per
// line, a warp per segment of SEG consecutive radii.  A solve is the Thomas
// recurrence per segment with zero carry-in, the segment ends exchanged
// through shared memory, and the carry added on the way back (the
// partitioned form of tridagr).  With the modes in the lanes, the factors of
// a radius are one broadcast word for the warp and the modal array is read
// and written in whole rows; eight lanes per line with shuffle scans instead
// spent 250 shared-memory cycles per 512 zones and step (66 us for five steps
// at 130 x 98 x 256).  A step's factors arrive one step ahead by cp.async
// (with the step's line coefficients beside them: 1183 -> 1209 us for 20 steps
// at 258 x 194 x 512, the extra registers spill).
// kCycle (converged form): Y keeps the residual for the next cycle, the
// potential's modal coefficients advance in phi, pre takes those before the
// cycle's last step (the solve ends with that step in half-step form), and the
// block's partial |update|^2 and |phi|^2 go to norms.  The update is what phi
// changed by as stored: the residual carried by the recurrence, and the update
// it gives, shrink without end below the rounding of phi, and a solve would go
// on by figures that are no longer in its potential.  (Formed anew from phi
// every cycle the residual costs 3 to 6 percent of a solve and, at 258 x 194 x
// 512, a fifth in accuracy: 6.5e-13 against 5.3e-13.)
// ROWS, the line length the factor blocks are padded to, is a compile-time
// constant so that every shared-memory operand is one base register and an
// offset.
template <int SEG, int ROWS, bool kCycle>
__global__ void __launch_bounds__(ROWS / SEG *kLines, ROWS == 256 ? 1 : 2) k_modal_radial(ModalArgs a) {
    extern __shared__ __align__(16) double sm[];
    constexpr int NSEG = ROWS / SEG, block = radial_block(ROWS);
    const int nseg = blockDim.x >> 5;
    double *ends = sm + 2 * block;             // [NSEG][32] forward ends
    double *starts = ends + NSEG * kLines;     // [NSEG][32] backward starts
    if (kCycle && a.skip && *a.skip) return;
    const TileIndex ti = tile_index(a, a.groups, blockIdx.x);
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int nr = a.nr, nz = a.nz;
    const double *frad = a.rad + (long long)ti.slot * block;
    const long long fstep = (long long)a.N * block;
    auto fetch = [&](int step) {
        const double *src = frad + (kCycle && a.lagged && step > 0 ? step - 1 : step) * fstep;
        double *dst = sm + (step & 1) * block;
        for (int i = 2 * tid; i < block; i += 2 * blockDim.x) {
            const unsigned d = (unsigned)__cvta_generic_to_shared(dst + i);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src + i));
        }
        asm volatile("cp.async.commit_group;");
    };
    fetch(0);
    pdl_wait();
    const int q = min(ti.tile * kLines + lane, nz - 1);
    const bool mine = ti.tile * kLines + lane < nz;
    const long long base = ((long long)ti.row * a.N + ti.slot) * nr * a.ldq + (long long)w * SEG * a.ldq + q;
    double *Yq = a.Y + base;
    const int count = min(SEG, nr - w * SEG);  // radii of this segment
    double r[SEG], x[SEG], acc[SEG];
#pragma unroll
    for (int e = 0; e < SEG; ++e) {
        r[e] = (e < count && mine) ? Yq[(long long)e * a.ldq] : 0.0;
        acc[e] = 0.0;
    }
    if (blockIdx.x + a.ahead < gridDim.x) {
        const TileIndex tn = tile_index(a, a.groups, blockIdx.x + a.ahead);
        const int qn = tn.tile * kLines;
        prefetch_rows(a.Y + ((long long)tn.row * a.N + tn.slot) * nr * a.ldq + qn, a.ldq, nr, min(kLines, nz - qn));
    }
    if (kCycle) {  // needed after the steps
        const int q0 = ti.tile * kLines;
        prefetch_rows(a.phi + ((long long)ti.row * a.N + ti.slot) * nr * a.ldq + q0, a.ldq, nr, min(kLines, nz - q0));
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int step = 0; step < a.nsteps; ++step) {
        const double *fac = sm + (step & 1) * block;
        const double2 *pair = reinterpret_cast<const double2 *>(fac) + w * SEG;
        const double2 *back = pair + ROWS;
        const double *kk = fac + 4 * ROWS + w * SEG;
        const double2 cs = a.cs[(long long)step * nz + q];
        const double dt2 = a.dt2[step];
        double y = 0.0;
#pragma unroll
        for (int e = 0; e < SEG; ++e) {
            const double2 f = pair[e];
            y = fma(f.y, y, r[e] * f.x);
            x[e] = y;
        }
        if (kCycle && a.lagged && step + 1 == a.nsteps) {  // the solve without a vertical one
#pragma unroll
            for (int e = 0; e < SEG; ++e) r[e] = 0.0;
        }
        ends[w * kLines + lane] = y;
        __syncthreads();  // every warp is past the previous step: its factor buffer is free
        if (step + 1 < a.nsteps) fetch(step + 1);
        double in = 0.0;
        {
            const double2 *g = reinterpret_cast<const double2 *>(fac) + ROWS + SEG - 1;
            const double *en = ends + lane;
#pragma unroll 4
            for (int s = 0; s < w; ++s) in = fma(g[s * SEG].y, in, en[s * kLines]);
        }
        double m = 0.0;
#pragma unroll
        for (int e = SEG - 1; e >= 0; --e) {
            const double2 f = back[e];
            m = fma(f.x, m, fma(f.y, in, x[e]));
            x[e] = m;
        }
        starts[w * kLines + lane] = m;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        in = 0.0;
        {
            const double *k = fac + 4 * ROWS, *st = starts + lane;
#pragma unroll 4
            for (int s = nseg - 1; s > w; --s) in = fma(k[s * SEG], in, st[s * kLines]);
        }
#pragma unroll
        for (int e = 0; e < SEG; e += 2) {
            const double2 k2 = *reinterpret_cast<const double2 *>(kk + e);
            const double v0 = fma(k2.x, in, x[e]), v1 = fma(k2.y, in, x[e + 1]);
            acc[e] = fma(cs.x, v0, acc[e]);
            acc[e + 1] = fma(cs.x, v1, acc[e + 1]);
            r[e] = cs.y * fma(dt2, v0, -r[e]);
            r[e + 1] = cs.y * fma(dt2, v1, -r[e + 1]);
            if (kCycle) {
                x[e] = cs.x * v0;
                x[e + 1] = cs.x * v1;
            }
        }
    }
    pdl_trigger();
    if (!kCycle) {
#pragma unroll
        for (int e = 0; e < SEG; ++e)
            if (e < count && mine) Yq[(long long)e * a.ldq] = acc[e];
        return;
    }
    double *Fq = a.phi + base, *Bq = a.pre ? a.pre + base : nullptr;
    double num = 0.0, den = 0.0;
#pragma unroll
    for (int e = 0; e < SEG; ++e)
        if (e < count && mine) Yq[(long long)e * a.ldq] = r[e];
#pragma unroll
    for (int e = 0; e < SEG; ++e)
        r[e] = (e < count && mine) ? Fq[(long long)e * a.ldq] : 0.0;
#pragma unroll
    for (int e = 0; e < SEG; ++e)
        if (e < count && mine) {
            const double v = r[e] + acc[e];
            Fq[(long long)e * a.ldq] = v;
            if (Bq) Bq[(long long)e * a.ldq] = v - x[e];
            const double change = v - r[e];
            num = fma(change, change, num);
            den = fma(v, v, den);
        }
    // the block's sums in a fixed order, with the slot's Parseval weight
    for (int d = 16; d > 0; d >>= 1) {
        num += __shfl_down_sync(0xffffffffu, num, d);
        den += __shfl_down_sync(0xffffffffu, den, d);
    }
    __syncthreads();
    if (lane == 0) {
        sm[2 * w] = num;
        sm[2 * w + 1] = den;
    }
    __syncthreads();
    if (tid == 0) {
        num = den = 0.0;
        for (int s = 0; s < nseg; ++s) {
            num += sm[2 * s];
            den += sm[2 * s + 1];
        }
        const double wt = (ti.slot == 0 || ti.slot == a.N / 2) ? 1.0 : 2.0;
        double *out = a.norms + 2 * (((long long)ti.row * a.N + ti.slot) * a.groups + ti.tile);
        out[0] = wt * num;
        out[1] = wt * den;
    }
}

// Radii per segment: 16 hold a line's residual, solution and update in 96
// registers; up to 64 radii take 8, which halves the serial chains (the
// smallest grids do not fill the chip).
int radial_seg(int nr) { return nr <= 64 ? 8 : 16; }
int radial_nseg(const bph_ctx *c) { return (c->nr + c->modal_seg - 1) / c->modal_seg; }
int radial_rows(const bph_ctx *c) { return c->nr <= 64 ? 64 : c->nr <= 128 ? 128 : 256; }

template <bool kCycle>
const void *radial_kernel(const bph_ctx *c) {
    switch (radial_rows(c)) {
        case 64: return (const void *)k_modal_radial<8, 64, kCycle>;
        case 128: return (const void *)k_modal_radial<16, 128, kCycle>;
        default: return (const void *)k_modal_radial<16, 256, kCycle>;
    }
}

size_t radial_smem(const bph_ctx *c) {
    const size_t rows = radial_rows(c);
    return sizeof(double) * (2 * (size_t)radial_block((int)rows) + 2 * rows / c->modal_seg * kLines);
}
constexpr int kNT = 4;  // 32 columns per transform tile (64: 161 against 129 us per solve at 130 x 98 x 256)
size_t fwd_smem(const bph_ctx *c) { return sizeof(double) * (size_t)((c->nz + 7) / 8 * 8) * TileShape<kNT>::ld; }
size_t inv_smem(const bph_ctx *c) { return sizeof(double) * (size_t)TileShape<kNT>::cols * inv_ld((c->nz + 7) / 8); }
// Dynamic shared bytes and kernels of the transforms in use.
size_t fwd_bytes(const bph_ctx *c) {
    if (!c->modal_p1) return fwd_smem(c);
    const int h2 = ((2 * c->nz + 1) / c->modal_p1 + 1) / 2, k2 = (h2 + 7) / 8 * 8;
    return sizeof(double) * (size_t)c->nz * TileShape<kNT>::ld + sizeof(int) * (size_t)c->modal_p1 * (h2 + k2);
}
size_t inv_bytes(const bph_ctx *c) {
    if (!c->modal_p1) return inv_smem(c);
    const int h2 = ((2 * c->nz + 1) / c->modal_p1 + 1) / 2;
    return inv_smem(c) + sizeof(int) * (size_t)c->modal_p1 * h2;
}
const void *fwd_kernel(const bph_ctx *c) {
    switch (c->modal_p1) {
        case 3: return (const void *)k_modal_fwd_split<kNT, 3>;
        case 5: return (const void *)k_modal_fwd_split<kNT, 5>;
        case 7: return (const void *)k_modal_fwd_split<kNT, 7>;
        default: return (const void *)k_modal_fwd<kNT>;
    }
}
const void *inv_kernel(const bph_ctx *c) {
    switch (c->modal_p1) {
        case 3: return (const void *)k_modal_inv_split<kNT, 3>;
        case 5: return (const void *)k_modal_inv_split<kNT, 5>;
        case 7: return (const void *)k_modal_inv_split<kNT, 7>;
        default: return (const void *)k_modal_inv<kNT>;
    }
}

// Fragment products (16 x 8 x 8, per eight columns) of one transform: dense, or
// split with first factor p1 (0: p1 does not apply to the height).
int dense_products(int nz) { return ((nz + 15) / 16) * ((nz + 7) / 8); }
int split_products(int nz, int isym, int p1) {
    const int L = 2 * nz + 1, p2 = L / p1;
    if (isym == 1 || L % p1 || p2 % p1 == 0 || p2 < p1) return 0;
    const int h2 = (p2 + 1) / 2;
    return p1 * ((h2 + 15) / 16) * ((h2 + 7) / 8);
}

int tile_threads(const bph_ctx *c) {
    if (c->modal_p1) return 256;
    const int mt = (c->nz + 15) / 16;
    const int rounds = (mt + 7) / 8;
    const int w = (mt + rounds - 1) / rounds;
    return 32 * (w < 4 ? 4 : w);
}

ModalArgs base_args(const bph_ctx *c) {
    ModalArgs a = {};
    a.half = ~0u;
    a.brb = c->d_brb;
    a.alphar = c->d_alphar;
    a.betar = c->d_betar;
    a.nslots = c->N;
    a.ntile = (c->nr + 8 * kNT - 1) / (8 * kNT);
    a.groups = modal_groups(c);
    a.numr = c->g.numr;
    a.numz = c->g.numz;
    a.nr = c->nr;
    a.nz = c->nz;
    a.ldq = modal_ldq(c);
    a.N = c->N;
    a.isym = c->g.isym;
    a.mtiles = (c->nz + 15) / 16;
    a.ksteps = (c->nz + 7) / 8;
    a.gamma = c->gamma;
    if (c->modal_p1) {
        const int h = (c->modal_p1 - 1) / 2;
        a.h2 = ((2 * c->nz + 1) / c->modal_p1 + 1) / 2;
        a.mt2 = (a.h2 + 15) / 16;
        a.ks2 = (a.h2 + 7) / 8;
        a.Cs = c->d_modE;
        a.tab = c->d_modtab;
        const double w = 2.0 * std::acos(-1.0) / c->modal_p1;
        for (int i = 0; i <= h; ++i)
            for (int b = 0; b <= h; ++b) {
                const int r = (c->modal_beta1 * i * b) % c->modal_p1;
                a.s1[i][b] = std::sin(w * r);
                a.c1[i][b] = std::cos(w * r);
            }
    }
    return a;
}

cudaError_t launch(bph_ctx *c, const void *fn, long long blocks, int threads, size_t smem, ModalArgs &a,
                   cudaStream_t st, bool pdl) {
    ++c->launches;
    a.ahead = (unsigned)(fn == fwd_kernel(c)   ? c->modal_resident[0]
                         : fn == inv_kernel(c) ? c->modal_resident[1]
                                               : c->modal_resident[2]);
    void *args[] = {&a};
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = launch_config(c, dim3((unsigned)blocks), dim3(threads), smem, attr);
    cfg.stream = st;
    if (!pdl) cfg.numAttrs = 0;
    return cudaLaunchKernelExC(&cfg, fn, args);
}

}  // namespace

int modal_groups(const bph_ctx *c) { return (c->nz + kLines - 1) / kLines; }
static int modal_ldq(const bph_ctx *c) { return (c->nz + 1) / 2 * 2; }  // 16-byte rows
size_t modal_size(const bph_ctx *c) { return (size_t)c->N * c->nr * modal_ldq(c); }

// A batch works through its instances in passes whose modal array stays well
// inside the 126 MB L2 (the three kernels hand it to each other).
int modal_chunk(const bph_ctx *c, int capacity) {
    const size_t fit = (48ull << 20) / (sizeof(double) * modal_size(c));
    const int most = fit < 1 ? 1 : fit > 64 ? 64 : (int)fit;
    return capacity < most ? capacity : most;
}

// Tables of the split form: the signed heights of (a1, a2), the packed second
// factors (wave: 2 / sqrt(L) cos over a period of 4 L), and the eigenvalues in
// the modal array's order.
static void split_tables(bph_ctx *c, const std::vector<double> &wave, std::vector<double> &pack, std::vector<int> &tab,
                         std::vector<double> &lam) {
    const int nz = c->nz, L = 2 * nz + 1, p1 = c->modal_p1, p2 = L / p1, h = (p1 - 1) / 2, h2 = (p2 + 1) / 2;
    const int alpha = (L % 4 == 1) ? 1 : 3;  // alpha L = 1 modulo 4
    const int beta = (int)(((1LL - (long long)alpha * L) / 4 % L + L) % L);
    auto inverse = [](int v, int m) {
        for (int x = 1; x < m; ++x)
            if ((long long)v % m * x % m == 1) return x;
        return 0;
    };
    c->modal_beta1 = (int)((long long)beta * inverse(p2, p1) % p1);
    const int beta2 = (int)((long long)beta * inverse(p1, p2) % p2);
    tab.assign((size_t)p1 * h2, 0);
    for (int k = 0; k < nz; ++k) {
        const int u = 2 * k + 1, a = (u % 4 == 1) ? u : L - u % L;
        int x1 = a % p1, x2 = a % p2, sg = 1;
        if (x2 >= h2 || (x2 == 0 && x1 > h)) {
            x1 = (p1 - x1) % p1;
            x2 = (p2 - x2) % p2;
            sg = -1;
        }
        tab[(size_t)x1 * h2 + x2] = sg * (k + 1);
    }
    // cos(2 pi r / p2) sits at 4 p1 r of the period 4 L, the sine a quarter period (L) on
    const double sign = (alpha == 1) ? -1.0 : 1.0;
    auto entry = [&](int b2, int a2, bool sine) -> double {
        if (b2 >= h2 || a2 >= h2) return 0.0;
        const long long r = (long long)beta2 * a2 % p2 * b2 % p2;
        return sign * wave[(size_t)((4LL * p1 * r + (sine ? 3LL * L : 0)) % (4LL * L))];
    };
    const int mt2 = (h2 + 15) / 16, ks2 = (h2 + 7) / 8;
    const size_t frag = (size_t)mt2 * ks2 * 128;
    pack.assign(2 * frag, 0.0);
    for (int m = 0; m < mt2; ++m)
        for (int k = 0; k < ks2; ++k)
            for (int l = 0; l < 32; ++l)
                for (int v = 0; v < 4; ++v) {
                    const int row = 16 * m + l / 4 + 8 * (v & 1), col = 8 * k + l % 4 + 4 * (v >> 1);
                    const size_t at = ((size_t)m * ks2 + k) * 128 + 4 * l + v;
                    pack[at] = entry(row, col, false);
                    pack[frag + at] = entry(row, col, true);
                }
    std::vector<double> by_q(lam);
    for (int b1 = 0; b1 <= h; ++b1)
        for (int b2 = 0; b2 < h2; ++b2) {
            const int p = tab[(size_t)b1 * h2 + b2];
            if (p) lam[(size_t)(run_plus(b1, h2) + b2)] = by_q[(size_t)(std::abs(p) - 1)];
            if (b1 > 0 && b2 > 0)
                lam[(size_t)(run_minus(b1, h2) + b2)] = by_q[(size_t)(std::abs(tab[(size_t)(p1 - b1) * h2 + b2]) - 1)];
        }
}

// Decides whether the grid runs the modal form and prepares it.  Lines of up
// to 256 radii fit a block; the transforms cost 4 nz FMA per zone and solve,
// and their column tile has to fit in shared memory (nz <= 640).  BPH_ADI_WARP
// in the environment asks for a half-step kernel by name, BPH_ADI_MODAL=0 for
// the half-step form.
int modal_configure(bph_ctx *c) {
    c->modal = 0;
    const char *want = std::getenv("BPH_ADI_MODAL");
    if ((want && want[0] == '0') || std::getenv("BPH_ADI_WARP")) return BPH_OK;
    if (c->nr > 16 * kMaxSegs || c->nz > 640) return BPH_OK;
    c->modal_seg = radial_seg(c->nr);
    const int nz = c->nz, ks = (nz + 7) / 8, mt = (nz + 15) / 16;
    // E[q][k] from a table of one period: its argument is (2k+1)(2q+1) pi / (2 (2 nz + 1))
    // (reflecting bottom) or (k+1)(q+1) pi / (nz + 1) (Dirichlet)
    const bool dirichlet = c->g.isym == 1;
    const long long period = dirichlet ? 2LL * (nz + 1) : 4LL * (2 * nz + 1);
    std::vector<double> wave((size_t)period), lam((size_t)nz);
    const long double pi = std::acos(-1.0L);
    const long double scale = dirichlet ? std::sqrt(2.0L / (nz + 1.0L)) : 2.0L / std::sqrt(2.0L * nz + 1.0L);
    for (long long i = 0; i < period; ++i) {
        const long double x = 2.0L * pi * (long double)i / (long double)period;
        wave[(size_t)i] = (double)(scale * (dirichlet ? std::sin(x) : std::cos(x)));
    }
    for (int q = 0; q < nz; ++q) {
        const long double half =
            dirichlet ? 0.5L * (q + 1.0L) * pi / (nz + 1.0L) : 0.5L * (q + 0.5L) * pi / (nz + 0.5L);
        const long double sn = std::sin(half);
        lam[(size_t)q] = (double)((long double)c->gamma * 4.0L * sn * sn);
    }
    auto entry = [&](int q, int k) -> double {
        if (q >= nz || k >= nz) return 0.0;
        const long long i = dirichlet ? (long long)(q + 1) * (k + 1) : (2LL * q + 1) * (2LL * k + 1);
        return wave[(size_t)(i % period)];
    };
    // the split form where it leaves at most two thirds of the products (192 heights: 56 of 288)
    c->modal_p1 = 0;
    int least = 2 * dense_products(nz) / 3;
    const char *ps = std::getenv("BPH_MODAL_SPLIT");
    for (int p1 : {3, 5, 7}) {
        const int n = (ps && ps[0] == '0') ? 0 : split_products(nz, c->g.isym, p1);
        if (n > 0 && n <= least) {
            least = n;
            c->modal_p1 = p1;
        }
    }
    const size_t frag = (size_t)mt * ks * 128;
    std::vector<double> pack(2 * frag);
    std::vector<int> tab;
    if (c->modal_p1) {
        split_tables(c, wave, pack, tab, lam);
    } else {
        for (int m = 0; m < mt; ++m)
            for (int k = 0; k < ks; ++k)
                for (int l = 0; l < 32; ++l)
                    for (int v = 0; v < 4; ++v) {
                        const int row = 16 * m + l / 4 + 8 * (v & 1), col = 8 * k + l % 4 + 4 * (v >> 1);
                        const size_t at = ((size_t)m * ks + k) * 128 + 4 * l + v;
                        pack[at] = entry(row, col);         // E: row = mode
                        pack[frag + at] = entry(col, row);  // E^T: row = height
                    }
    }
    // One allocation: both fragment arrays, the eigenvalues, the norm partials, one instance's modal
    // array.  Slots beyond shared memory have their half-steps' scratch, which no solve needs while
    // its steps are modal (d_W >= N nr (nz + 1)): the modal array and the converged form's earlier
    // potential, which is back in P before the last half-steps run, live there.
    const bool scratch = c->adi_smem == 0;
    const size_t norms = 2 * (size_t)c->N * modal_groups(c), lams = ((size_t)nz + 1) / 2 * 2;
    const size_t tabs = (tab.size() + 3) / 4 * 2;  // doubles that hold the index table
    const size_t all = pack.size() + lams + norms + tabs + (scratch ? 0 : modal_size(c));
    if (cudaMalloc((void **)&c->d_modE, sizeof(double) * all) != cudaSuccess) {
        cudaGetLastError();  // no room: the half-step kernels need none of it
        c->d_modE = nullptr;
        return BPH_OK;
    }
    c->d_modlam = c->d_modE + pack.size();
    c->d_modnorm = c->d_modlam + lams;
    c->d_modtab = reinterpret_cast<int *>(c->d_modnorm + norms);
    c->d_modY = scratch ? c->d_W : c->d_modnorm + norms + tabs;
    if (scratch) {
        c->d_modpre = c->d_W2;
        c->modpre_at = kModpreScratch;
    }
    c->bytes += sizeof(double) * all;
    pack.insert(pack.end(), lam.begin(), lam.end());
    BPH_CUDA(cudaMemcpyAsync(c->d_modE, pack.data(), sizeof(double) * pack.size(), cudaMemcpyHostToDevice, c->stream));
    if (!tab.empty())
        BPH_CUDA(cudaMemcpyAsync(c->d_modtab, tab.data(), sizeof(int) * tab.size(), cudaMemcpyHostToDevice, c->stream));
    BPH_CUDA(cudaStreamSynchronize(c->stream));  // pack and tab are this call's own
    BPH_CUDA(raise_smem_limit(fwd_kernel(c), (int)fwd_bytes(c)));
    BPH_CUDA(raise_smem_limit(inv_kernel(c), (int)inv_bytes(c)));
    BPH_CUDA(raise_smem_limit(radial_kernel<false>(c), (int)radial_smem(c)));
    BPH_CUDA(raise_smem_limit(radial_kernel<true>(c), (int)radial_smem(c)));
    // resident blocks of each (one per SM where a tall tile fills its shared memory)
    int sms = 0;
    BPH_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
    const void *kernels[3] = {fwd_kernel(c), inv_kernel(c), radial_kernel<false>(c)};
    const size_t smem[3] = {fwd_bytes(c), inv_bytes(c), radial_smem(c)};
    for (int k = 0; k < 3; ++k) {
        int per_sm = 0;
        BPH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernels[k],
                                                               k < 2 ? tile_threads(c) : kLines * radial_nseg(c), smem[k]));
        c->modal_resident[k] = sms * (per_sm > 1 ? per_sm : 1);
    }
    c->modal = 1;
    return BPH_OK;
}

void modal_free(bph_ctx *c) {
    if (c->d_modE) cudaFree(c->d_modE);
    c->d_modE = c->d_modlam = c->d_modnorm = c->d_modY = nullptr;
    c->modal = 0;
}

size_t modal_radial_doubles(const bph_ctx *c) { return (size_t)radial_block(radial_rows(c)); }

// A schedule's radial blocks and step coefficients (after launch_adi_factors).
cudaError_t modal_pack(bph_ctx *c, Schedule &s) {
    if (!s.d_mod_rad) return cudaSuccess;
    c->launches += 2;
    const int nseg = radial_rows(c) / c->modal_seg;
    k_pack_modal<<<(unsigned)(s.nsteps * c->N), nseg, 0, c->stream>>>(s.d_rad, s.d_mod_rad, c->nr, nseg, c->modal_seg);
    k_modal_coef<<<(unsigned)(2 * s.nsteps + 1), 128, 0, c->stream>>>(s.d_dt, c->d_modlam, s.d_mod_cs, s.d_mod_dt2,
                                                                     c->nz, s.nsteps);
    return cudaGetLastError();
}

// A schedule's form: in the eigenbasis from modal_min steps on.  The
// transforms cost a fixed time and a modal step little; a half-step kernel has
// no fixed part to speak of.
//   Warp-cooperative half-steps (130 x 98 x 256: 70 + 4.6 a step in the
//   eigenbasis against 22 + 10; 66 x 66 x 64: 14 + 0.8 against 4 + 2.3): eight.
//   The other half-step kernels: two (us for one and for two steps, half-steps
//   against eigenbasis: 101 x 75 x 128 26 / 44 against 40 / 42, 67 x 45 x 64
//   15 / 25 against 16 / 17, 258 x 194 x 512 424 / 790 against 485 / 526);
//   one where a slot is so small that the transforms cost no more than a step
//   (40 x 30 x 64 13.5 against 12.5, 50 x 50 x 256 28 against 21).
//   Tall slots, whose transforms' products are long serial chains (serial_steps
//   of 64 clocks and more each): where the set-up's timing says, which for the
//   five steps of a warm solve went to the half-steps at 12 x 500 x 32 (131
//   against 203 us a solve), 8 x 200 x 64 (70 against 83) and 258 x 402 x 16
//   (545 against 605), and to the eigenbasis at 40 x 400 x 64 (328 against
//   269), 20 x 300 x 64 (113 against 87) and 20 x 146 x 64 (71 against 58).
//   The timing has no second stream for the free slots' half-steps, hence a
//   margin of a tenth.  Untimed: eight.
// Batches fill the chip better in either form and take the eigenbasis from two
// steps on (us for one and for sixteen models: 8 x 200 x 64 98 / 466 in
// half-steps, 89 / 325; 258 x 402 x 16 776 / 3484, 674 / 3411), but for the
// longest chains on the segmented kernel (20 x 402 x 128 208 / 2067 against
// 223 / 2177, 12 x 500 x 32 168 / 556 against 232 / 923).
static int serial_steps(const bph_ctx *c) {
    if (!c->modal_p1) {
        const int mt = (c->nz + 15) / 16;
        return (mt + 7) / 8 * ((c->nz + 7) / 8);
    }
    const int h2 = ((2 * c->nz + 1) / c->modal_p1 + 1) / 2, units = (c->modal_p1 + 1) / 2 * ((h2 + 15) / 16);
    return (units + 7) / 8 * 2 * ((h2 + 7) / 8);
}

// Whether the set-up's timing decides: 24 serial steps for the on-chip
// segmented kernel, 100 for the slower grid-wide ones (the kernel with a
// thread per line is the slower form from one step on at every height).
bool modal_tall(const bph_ctx *c) {
    return c->modal && !c->adi_warp && (c->adi_seg || !c->adi_smem) && serial_steps(c) > (c->adi_seg ? 24 : 100);
}

// us[form][k]: contraction and ADI of 1 (k = 0) and 5 steps in half-steps and
// in the eigenbasis, both linear in the steps; nullptr: untimed.
void modal_rule(bph_ctx *c, const float (*us)[2]) {
    c->modal_min = c->adi_warp ? 8 : c->nr <= 64 && c->nz <= 48 ? 1 : 2;
    c->modal_min_batch = c->modal_min;
    if (!modal_tall(c)) return;
    c->modal_min = 8;
    if (us) {
        const float half = (us[0][1] - us[0][0]) / 4, modal = (us[1][1] - us[1][0]) / 4;
        int n = 2;
        while (n < 64 && us[1][0] + modal * (n - 1) >= 0.9f * (us[0][0] + half * (n - 1))) ++n;
        c->modal_min = n;
    }
    if (c->adi_seg && serial_steps(c) > 100) c->modal_min_batch = c->modal_min;
}

bool modal_ready(const bph_ctx *c, const Schedule &s, bool batch) {
    return c->modal && s.d_mod_rad && s.nsteps >= (batch ? c->modal_min_batch : c->modal_min);
}

// Converged cycles stay in the eigenbasis, so only the choice between warp
// kernel and modal steps is one of steps (at most seven: the warp kernel).  The
// grid-wide FP32 refinement cycle costs more than a modal cycle in FP64
// (258 x 194 x 512, ten steps: 2500 against 480 us), so the mixed form runs
// the latter where that refinement would be its choice.
bool modal_converged(const bph_ctx *c, const Schedule &s, bool mixed) {
    return c->modal && s.d_mod_rad && !(c->adi_warp && s.nsteps <= 7) &&
           (!mixed || c->mixed_kind == BPH_MIXED_ADI_GLOBAL);
}

// Whether a solve's slots are worth two passes, the free ones' beside the
// contraction: below this many zones the kernels of a pass are latency, and
// two of each cost more than they hide (us per warm solve with and without:
// 18 x 18 x 16 31 / 18, 50 x 50 x 256 54 / 47, 200 x 30 x 128 92 / 88;
// 101 x 75 x 128 94 / 100, 110 x 90 x 256 154 / 168).
bool modal_overlaps(const bph_ctx *c) { return c->np * c->N >= 800000; }

cudaError_t launch_modal(bph_ctx *c, const Schedule &s, bool cold, double *P, const double *R, double *Y, int chunk,
                         int ninst, const int *inst_map, const int *slot_map, int nslots, cudaStream_t st, bool pdl) {
    ModalArgs a = base_args(c);
    a.P = P;
    a.R = R;
    a.Y = Y;
    a.slot_map = slot_map;
    a.nslots = nslots;
    a.rad = s.d_mod_rad;
    a.cs = s.d_mod_cs;
    a.dt2 = s.d_mod_dt2;
    a.nsteps = s.nsteps;
    const int threads = tile_threads(c);
    for (int r0 = 0; r0 < ninst; r0 += chunk) {
        const int rows = ninst - r0 < chunk ? ninst - r0 : chunk;
        const long long blocks = (long long)rows * nslots;
        a.inst_map = inst_map ? inst_map + r0 : nullptr;
        a.inst0 = r0;
        a.E = c->d_modE;
        a.source = cold ? kColdResidual : kResidual;
        cudaError_t e = launch(c, fwd_kernel(c), blocks * a.ntile, threads, fwd_bytes(c), a, st, pdl);
        if (e == cudaSuccess)
            e = launch(c, radial_kernel<false>(c), blocks * a.groups, kLines * radial_nseg(c), radial_smem(c), a, st, pdl);
        a.E = c->d_modE + (size_t)a.mtiles * a.ksteps * 128;
        a.add = cold ? 0 : 1;
        if (e == cudaSuccess) e = launch(c, inv_kernel(c), blocks * a.ntile, threads, inv_bytes(c), a, st, pdl);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Converged form: the modal residual (and, warm, the modal potential) of
// ninst instances; cycles on them; a potential back in P.  The FP64 form takes
// the one before the last step and runs that step in half-step form: the
// residual it reports is the half-step iteration's, whose rounding floor its
// last vertical half-step sets.  The mixed form (pre: nullptr) takes the last
// one, its cycles in the refinement's half-step order.
cudaError_t launch_modal_begin(bph_ctx *c, bool cold, double *P, const double *R, double *Y, double *phi, int ninst,
                               const int *inst_map) {
    ModalArgs a = base_args(c);
    a.P = P;
    a.R = R;
    a.Y = Y;
    a.inst_map = inst_map;
    a.E = c->d_modE;
    a.source = cold ? kColdResidual : kResidual;
    const long long blocks = (long long)ninst * c->N * a.ntile;
    // warm: both transforms in one launch, side by side where one alone leaves SMs idle (us of a solve
    // of one cycle: 66 x 66 x 64 119 -> 110, 40 x 400 x 64 540 -> 400, 12 x 500 x 32 390 -> 297)
    if (!cold) {
        a.phi = phi;
        a.half = (unsigned)blocks;
    }
    const cudaError_t e =
        launch(c, fwd_kernel(c), cold ? blocks : 2 * blocks, tile_threads(c), fwd_bytes(c), a, c->stream, c->pdl);
    if (e != cudaSuccess || !cold) return e;
    return cudaMemsetAsync(phi, 0, sizeof(double) * (size_t)ninst * modal_size(c), c->stream);
}

cudaError_t launch_modal_cycle(bph_ctx *c, const Schedule &s, double *Y, double *phi, double *pre, int ninst,
                               double *norms, const int *skip) {
    ModalArgs a = base_args(c);
    a.Y = Y;
    a.phi = phi;
    a.pre = pre;
    a.rad = s.d_mod_rad;
    a.lagged = pre ? 0 : 1;
    const int first = a.lagged ? s.nsteps : 0;
    a.cs = s.d_mod_cs + (size_t)first * c->nz;
    a.dt2 = s.d_mod_dt2 + first;
    a.nsteps = s.nsteps + a.lagged;
    a.norms = norms;
    a.skip = skip;
    return launch(c, radial_kernel<true>(c), (long long)ninst * c->N * a.groups, kLines * radial_nseg(c), radial_smem(c), a,
                  c->stream, c->pdl);
}

cudaError_t launch_modal_end(bph_ctx *c, double *P, double *pre, int ninst, const int *inst_map) {
    ModalArgs a = base_args(c);
    a.P = P;
    a.Y = pre;
    a.inst_map = inst_map;
    a.E = c->d_modE + (size_t)a.mtiles * a.ksteps * 128;
    return launch(c, inv_kernel(c), (long long)ninst * c->N * a.ntile, tile_threads(c), inv_bytes(c), a,
                  c->stream, c->pdl);
}

}  // namespace bph
