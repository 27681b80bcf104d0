// The wide (48 x 32) warp tiles and the update sweep of the direct
// defect-solve kernel (bph_direct.h), run on the CPU with the kernel's schedule
// emulated lane by lane: the in-place transform, each block in the tiles that
// wide_block gives it, equals the dense product with every output written once
// and every access inside the shared-memory arrays and the block's columns; the
// update sweep visits every zone once and reads the deltas as aligned 16-byte
// words inside their column.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "bph_direct.h"

using namespace bph::direct;

static int failures = 0;
#define CHECK(c, ...)                      \
    do {                                   \
        if (!(c)) {                        \
            ++failures;                    \
            if (failures < 20) {           \
                std::printf("FAIL: ");     \
                std::printf(__VA_ARGS__);  \
                std::printf("\n");         \
            }                              \
        }                                  \
    } while (0)

// X <- A X on X^T for one warp tile of 16 M x 8 N: (offset, value) of its results.
struct Out {
    int off;
    double val;
};
static void tile(const Shape &d, const std::vector<double> &A, const std::vector<double> &Xt, int i0, int c0, int M, int N,
                 int lo, int hi, std::vector<Out> &outs) {
    for (int m = 0; m < M; ++m)
        for (int n = 0; n < N; ++n) {
            double acc[16][8] = {};
            for (int k0 = 0; k0 < d.nzp; k0 += 8) {
                double At[16][8], Bt[8][8];  // gathered by the lanes
                for (int lane = 0; lane < 32; ++lane) {
                    const int g = lane >> 2, t = lane & 3;
                    for (int v = 0; v < 4; ++v) {
                        const int o = a_offset(i0, m, k0, g, t, d.lda, v);
                        CHECK(o >= 0 && o < d.nzp * d.lda, "A offset %d", o);
                        At[g + 8 * (v & 1)][t + 4 * (v >> 1)] = A[(size_t)o];
                    }
                    for (int v = 0; v < 2; ++v) {
                        const int o = b_offset(c0, n, k0, g, t, d.ldk, v);
                        CHECK(o >= 0 && o < d.nrp * d.ldk && o % d.ldk < d.nzp, "B offset %d", o);
                        Bt[t + 4 * v][g] = Xt[(size_t)o];
                    }
                }
                for (int r = 0; r < 16; ++r)
                    for (int c = 0; c < 8; ++c)
                        for (int k = 0; k < 8; ++k) acc[r][c] += At[r][k] * Bt[k][c];
            }
            for (int lane = 0; lane < 32; ++lane)
                for (int v = 0; v < 4; ++v) {
                    const int g = lane >> 2, t = lane & 3, o = d_offset(i0, m, c0, n, g, t, d.ldk, v);
                    CHECK(o >= 0 && o < d.nrp * d.ldk && o % d.ldk < d.nzp, "D offset %d", o);
                    CHECK(o / d.ldk >= lo && o / d.ldk < hi, "write outside the block");
                    outs.push_back({o, acc[g + 8 * (v >> 1)][2 * t + (v & 1)]});
                }
        }
}

// Returns the number of blocks that took wide tiles.
static int check_transform(int nr, int nz, std::mt19937 &rng) {
    const Shape d = shape(nr, nz);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    std::vector<double> A((size_t)d.nzp * d.lda, 0.0), X((size_t)nz * nr), Xt((size_t)d.nrp * d.ldk, 0.0);
    for (int q = 0; q < nz; ++q)
        for (int k = 0; k < nz; ++k) A[(size_t)q * d.lda + k] = u(rng);
    for (int k = 0; k < nz; ++k)
        for (int j = 0; j < nr; ++j) Xt[(size_t)j * d.ldk + k] = X[(size_t)k * nr + j] = u(rng);
    std::vector<int> writes(Xt.size(), 0);
    int wide = 0;
    for (int cp0 = 0, cp = d.nrp / 16; cp0 < cp; cp0 += d.cpb) {
        const int ncp = (d.cpb < cp - cp0) ? d.cpb : cp - cp0, lo = 16 * cp0, hi = 16 * (cp0 + ncp);
        std::vector<Out> outs;
        int i0, c0;
        if (wide_block(d.nzp, ncp)) {
            ++wide;
            for (int w = 0; w < kWarps; ++w)
                if (wide_tile(w, d.nzp, cp0, ncp, i0, c0)) tile(d, A, Xt, i0, c0, 3, 4, lo, hi, outs);
        } else {
            for (int t = 0; t < (d.nzp / 32) * ncp; ++t) {
                warp_tile(t, cp0, ncp, i0, c0);
                tile(d, A, Xt, i0, c0, 2, 2, lo, hi, outs);
            }
        }
        for (const Out &o : outs) {  // after the block's barrier
            Xt[(size_t)o.off] = o.val;
            ++writes[(size_t)o.off];
        }
    }
    double err = 0.0;
    for (int j = 0; j < d.nrp; ++j)
        for (int q = 0; q < d.nzp; ++q) {
            CHECK(writes[(size_t)j * d.ldk + q] == 1, "nr %d nz %d: (%d, %d) written %d times", nr, nz, q, j,
                  writes[(size_t)j * d.ldk + q]);
            double ref = 0.0;
            if (q < nz && j < nr)
                for (int k = 0; k < nz; ++k) ref += A[(size_t)q * d.lda + k] * X[(size_t)k * nr + j];
            err = std::fmax(err, std::fabs(Xt[(size_t)j * d.ldk + q] - ref));
        }
    CHECK(err < 1e-12, "nr %d nz %d: transform error %g", nr, nz, err);
    return wide;
}

static void check_update(int nr, int nz) {
    const Shape d = shape(nr, nz);
    std::vector<int> seen((size_t)nr * nz, 0);
    for (int it = 0; it < sweep_items(nr); ++it) {
        int jc, k0, k1;
        update_item(it, nr, nz, jc, k0, k1);
        for (int j = jc; j < jc + 32 && j < nr; ++j)
            for (int kb = k0; kb < k1; kb += kUpd)
                for (int u = 0; u < kUpd && kb + u < k1; u += 4) {
                    const long long word = (long long)j * d.ldk + kb + u;
                    CHECK(word % 4 == 0 && kb + u + 3 < d.ldk, "nr %d nz %d: word (%d, %d)", nr, nz, j, kb + u);
                    for (int v = 0; v < 4 && kb + u + v < k1; ++v) ++seen[(size_t)(kb + u + v) * nr + j];
                }
    }
    for (size_t e = 0; e < seen.size(); ++e) CHECK(seen[e] == 1, "nr %d nz %d: zone %zu updated %d times", nr, nz, e, seen[e]);
}

int main() {
    std::mt19937 rng(11);
    // rows 96 and 192: whole blocks, an odd number of column pairs, a short last block (8 pairs, then 2 or
    // 1; at 192 rows 4, then 2); rows that are no multiple of 48
    struct {
        int nr, nz, wide;
    } shapes[] = {{128, 96, 1}, {128, 90, 1}, {130, 96, 1}, {150, 96, 2}, {34, 70, 0},  {20, 66, 1},
                  {16, 96, 0},  {64, 192, 1}, {90, 170, 2}, {70, 192, 1}, {128, 64, 0}, {100, 60, 0}};
    for (const auto &s : shapes) {
        const int wide = check_transform(s.nr, s.nz, rng);
        CHECK(wide == s.wide, "nr %d nz %d: %d wide blocks, expected %d", s.nr, s.nz, wide, s.wide);
    }
    for (int nr : {1, 31, 32, 33, 96, 128, 250, 257, 300})
        for (int nz : {1, 3, 11, 12, 13, 47, 48, 60, 96, 97, 200}) check_update(nr, nz);
    if (failures) {
        std::printf("%d failures\n", failures);
        return 1;
    }
    std::printf("all checks passed\n");
    return 0;
}
