// bph_fft.cu -- azimuthal real FFTs (realft.F90 + the slot reorder of
// helmadi.F90:132-183 and its inverse :357-411).
//
// A block takes a tile of 16 (or 32) consecutive (J,K) columns and all numphi
// samples of each: every row of the tile is a 128-byte segment of the Fortran array
// (J fastest).  The N real samples of a column are M = N/2 complex values,
// transformed in two steps, M = R1 T: T threads per column hold R1 values
// each and transform them in registers, exchange them once through shared
// memory, and do the T-point transforms of the other digit.  The threads'
// second digits are dealt so that k and M - k, which the real spectrum needs
// together, meet in one thread (R1 = 2T) or in two lanes of a warp (R1 = T),
// so the split into the real spectrum and the store to the slots need no
// further exchange.  (An in-place Stockham pass per radix-4 step wrote and
// read the tile ten times with a barrier each; it spent 18.8 + 15.9 us at
// 130 x 98 x 256.)  Results are written slot-major, which is the layout the
// ADI kernels read: the reference's swap_phi_r / swap_r_phi transposes are
// this store / load layout.
//
// Forward convention (realft isign=+1): F_k = sum_l f_l exp(+2 pi i k l / N).
#include <cmath>
#include <cstdlib>

#include "bph_internal.cuh"

namespace bph {
namespace {

// Columns per block: 16, a 128-byte row segment; 32 for the 128-point forward
// transform, whose tiles start one zone into a row and so touch a sector more
// than their length (130 x 98 x 256: 15.8 -> 13.9 us; the inverse, on whole
// rows, 9.9 with 16 and 10.5 with 32).
template <int M, bool kFwd>
constexpr int tile_cols() {
    return M == 128 && kFwd ? 32 : 16;
}

// M = R1 T, both powers of two, R1 = T or 2T.
template <int M>
struct Split {
    static constexpr int T = M >= 256 ? 16 : M >= 64 ? 8 : M >= 16 ? 4 : 2;
    static constexpr int R1 = M / T;
    static constexpr int kOwn = R1 / T;  // second digits k1 per thread: 1 or 2
    static_assert(R1 == T || R1 == 2 * T, "R1 = T or 2T");
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {  // a * conj(b)
    return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

// v <- its R-point transform, natural order; S = +1: e^{+i}, -1: e^{-i}.
template <int S>
__device__ __forceinline__ double2 times_i(double2 a) {
    return (S > 0) ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}
template <int S>
__device__ __forceinline__ void dft4(double2 &a, double2 &b, double2 &c, double2 &d) {
    const double2 s0 = cadd(a, c), s1 = csub(a, c), s2 = cadd(b, d), s3 = times_i<S>(csub(b, d));
    a = cadd(s0, s2);
    b = cadd(s1, s3);
    c = csub(s0, s2);
    d = csub(s1, s3);
}
template <int R, int S>
__device__ __forceinline__ void dft(double2 *v) {
    constexpr double h = 0.70710678118654752440, c1 = 0.92387953251128675613, s1 = 0.38268343236508977173;
    if (R == 2) {
        const double2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if (R == 4) {
        dft4<S>(v[0], v[1], v[2], v[3]);
    } else if (R == 8) {
        double2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        dft4<S>(e[0], e[1], e[2], e[3]);
        dft4<S>(o[0], o[1], o[2], o[3]);
        o[1] = cmul(o[1], make_double2(h, S * h));
        o[2] = times_i<S>(o[2]);
        o[3] = cmul(o[3], make_double2(-h, S * h));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = cadd(e[k], o[k]);
            v[k + 4] = csub(e[k], o[k]);
        }
    } else {  // 16 = 4 x 4
#pragma unroll
        for (int b = 0; b < 4; ++b) dft4<S>(v[b], v[4 + b], v[8 + b], v[12 + b]);
        // v[4 p + b] holds digit p of column b: twiddle e^{2 pi i b p / 16}
        v[5] = cmul(v[5], make_double2(c1, S * s1));
        v[6] = cmul(v[6], make_double2(h, S * h));
        v[7] = cmul(v[7], make_double2(s1, S * c1));
        v[9] = cmul(v[9], make_double2(h, S * h));
        v[10] = times_i<S>(v[10]);
        v[11] = cmul(v[11], make_double2(-h, S * h));
        v[13] = cmul(v[13], make_double2(s1, S * c1));
        v[14] = cmul(v[14], make_double2(-h, S * h));
        v[15] = cmul(v[15], make_double2(-c1, -S * s1));
#pragma unroll
        for (int p = 0; p < 4; ++p) dft4<S>(v[4 * p], v[4 * p + 1], v[4 * p + 2], v[4 * p + 3]);
        // v[4 p + q] = X[p + 4 q]: to natural order
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int q = p + 1; q < 4; ++q) {
                const double2 x = v[4 * p + q];
                v[4 * p + q] = v[4 * q + p];
                v[4 * q + p] = x;
            }
    }
}

// Second digits of thread u of a column.  kOwn = 2: u and R1 - u (u = 0: 0 and
// R1/2), so that k = k1 + R1 k2 of one list pairs with M - k of the other.
// kOwn = 1: lanes 2i and 2i + 1 of a column (16 lanes apart) take i and R1 - i
// (i = 0: 0 and R1/2).
template <int M>
__device__ __forceinline__ int second_digit(int u, int which) {
    constexpr int R1 = Split<M>::R1;
    if (Split<M>::kOwn == 2) return which == 0 ? u : (u == 0 ? R1 / 2 : R1 - u);
    const int i = u >> 1;
    return (u & 1) == 0 ? i : (i == 0 ? R1 / 2 : R1 - i);
}

__device__ __forceinline__ double2 shfl_xor2(double2 v, int mask) {
    return make_double2(__shfl_xor_sync(0xffffffffu, v.x, mask), __shfl_xor_sync(0xffffffffu, v.y, mask));
}

// F_k of the real spectrum from the packed transform's values at k and M - k.
__device__ __forceinline__ double2 real_split(double2 zk, double2 zm, double2 w) {
    const double2 e = make_double2(0.5 * (zk.x + zm.x), 0.5 * (zk.y - zm.y));
    const double2 o = make_double2(0.5 * (zk.y + zm.y), -0.5 * (zk.x - zm.x));
    return cadd(e, cmul(w, o));
}
// Z_k of the packed transform from the real spectrum at k and M - k.
__device__ __forceinline__ double2 real_merge(double2 fk, double2 fm, double2 w) {
    const double2 e = make_double2(0.5 * (fk.x + fm.x), 0.5 * (fk.y - fm.y));
    const double2 o = cmulc(make_double2(0.5 * (fk.x - fm.x), 0.5 * (fk.y + fm.y)), w);
    return make_double2(e.x - o.y, e.y + o.x);
}

// Batched launches: blockIdx.y is the batch position.  in / outp hold each
// position's caller array (forward: rho; inverse: pot), inst its instance
// (nullptr: position = instance); instance i's slot data sits at
// i * inst_stride from the given base, position j's moments at
// j * pos_stride, its non-finite flag at status[j].
struct FftBatch {
    const double *const *in = nullptr;
    double *const *outp = nullptr;
    const int *inst = nullptr;
    long long inst_stride = 0, pos_stride = 0;
    int status_stride = 0;  // 1: a flag per position, 0: one shared flag
};

// Threads and shared bytes of a tile (the same for both register budgets).
template <int M, bool kFwd>
struct FftTile {
    static constexpr int kCols = tile_cols<M, kFwd>();
    static constexpr int kThreads = Split<M>::T * kCols;
    static constexpr size_t kSmem = sizeof(double2) * ((size_t)M * kCols + M + (M + 1));
    static_assert(Split<M>::kOwn == 2 || kCols == 16, "paired lanes are 16 apart");
};

// Resident threads per SM the register budget is sized for: 512 (128
// registers hold 16 values and a transform's temporaries; a thread has all its
// loads in flight at once), or, dense, 768.  The set-up autotuner or
// BPH_FFT_DENSE chooses for single transforms; batched ones run against HBM
// and take the first (130 x 98 x 256, batch of 16: 1788 against 1890 us).
template <int M, bool kFwd, int Dense = 0>
struct FftShape : FftTile<M, kFwd> {
    static constexpr int kMinBlocks = (Dense ? 768 : 512) / FftTile<M, kFwd>::kThreads;
};

// Forward transform of interior columns.  kRho: write R = -4 pi rho_hat
// (zero on the rows potential_solver.F90:66-78 zeroes) and the boundary
// moments of the unzeroed density (bessel.F90:179-185, 226-274) obtained
// from the same spectrum: sum_l rho_l e^{i k (l - 1/2) dphi} = e^{i pi k/N} F_k.
// !kRho: write the warm-start potential into P's interior.
template <int M, bool kRho, int Dense = 0>
__global__ void __launch_bounds__((FftTile<M, true>::kThreads), (FftShape<M, true, Dense>::kMinBlocks))
k_fft_fwd(const double *__restrict__ src, double *__restrict__ out, double *__restrict__ mom,
          const double2 *__restrict__ g_tw, const double2 *__restrict__ g_tw2, const double2 *__restrict__ g_ph,
          int numr, int numz, int nr, int nz, int mmax, int fm, int isym, double four_pi,
          int *__restrict__ status, long long mstride, FftBatch bt) {
    constexpr int kTile = tile_cols<M, true>(), NT = FftTile<M, true>::kThreads;
    constexpr int T = Split<M>::T, R1 = Split<M>::R1, kOwn = Split<M>::kOwn;
    extern __shared__ double2 smem[];
    double2 *C = smem;  // [k1][t][column]
    double2 *tw = C + M * kTile;
    double2 *tw2 = tw + M;
    const int tid = threadIdx.x, c = tid % kTile, t = tid / kTile;
    const long long np = (long long)nr * nz;
    const long long nplane = (long long)numr * numz;
    const long long p = (long long)blockIdx.x * kTile + c;
    for (int i = tid; i < M; i += NT) tw[i] = g_tw[i];
    for (int i = tid; i <= M; i += NT) tw2[i] = g_tw2[i];
    pdl_wait();
    if (bt.in) {
        const int pos = blockIdx.y;
        src = bt.in[pos];
        out += (long long)(bt.inst ? bt.inst[pos] : pos) * bt.inst_stride;
        if (kRho) {
            mom += pos * bt.pos_stride;
            status += pos * bt.status_stride;
        }
    }
    const bool valid = p < np;
    const int jz = valid ? (int)p % nr + 1 : 1, kz = valid ? (int)p / nr + 1 : 1;
    {
        // packed values T r + t, all loads in flight
        const double *col = src + jz + (long long)numr * kz + nplane * (2 * t);
        double2 v[R1];
#pragma unroll
        for (int r = 0; r < R1; ++r)
            v[r] = valid ? make_double2(__ldg(col + nplane * (2 * T * r)), __ldg(col + nplane * (2 * T * r + 1)))
                         : make_double2(0.0, 0.0);
        if (kRho) {
            bool bad = false;
#pragma unroll
            for (int r = 0; r < R1; ++r) bad |= !(isfinite(v[r].x) && isfinite(v[r].y));
            if (bad) atomicOr(status, kStatusNonFinite);
        }
        dft<R1, +1>(v);
        __syncthreads();  // the twiddles
        double2 *mine = C + t * kTile + c;
        mine[0] = v[0];
#pragma unroll
        for (int k = 1; k < R1; ++k) mine[k * T * kTile] = cmul(v[k], tw[t * k]);
    }
    __syncthreads();
    double2 x[kOwn][T];
    int k1[kOwn];
#pragma unroll
    for (int o = 0; o < kOwn; ++o) {
        k1[o] = second_digit<M>(t, o);
        const double2 *in = C + k1[o] * T * kTile + c;
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) x[o][k2] = in[k2 * kTile];
        dft<T, +1>(x[o]);
    }
    pdl_trigger();
    const bool zeroed = (jz == numr - 2) || (kz == numz - 2) || (isym == 1 && kz == 1);
    const double scale = zeroed ? 0.0 : -four_pi;
    double *o_ = kRho ? out + p : out + jz + (long long)numr * kz;
    const long long so = kRho ? np : nplane;
    // Slot values: s = k -> Re F_k (F_0 at 0), s = M + k -> -Im F_k, s = M -> F_M.
    auto emit = [&](int k, double2 F) {
        if (!valid) return;
        if (!kRho) {
            o_[so * k] = F.x;
            o_[so * (M + k)] = -F.y;
            return;
        }
        o_[so * k] = zeroed ? 0.0 : scale * F.x;
        o_[so * (M + k)] = zeroed ? 0.0 : -(scale * F.y);
        // the boundary mode m with fm m = k (fm is 1 or 2; a division by it here took 1.0 of the 6.1 us
        // of 66 x 66 x 64 and 2.1 of the 13.2 of 200 x 150 x 64)
        if (k < fm * mmax && (k & (fm - 1)) == 0) {
            const int m = k >> (fm - 1);
            const double2 ph = g_ph[m];
            mom[m * mstride + p] = ph.x * F.x - ph.y * F.y;
            mom[m * mstride + np + p] = ph.y * F.x + ph.x * F.y;
        }
    };
    auto emit_ends = [&](double2 z) {  // k = 0: F_0 and F_M, both real
        if (!valid) return;
        const double f0 = z.x + z.y, fM = z.x - z.y;
        if (!kRho) {
            o_[0] = f0;
            o_[so * M] = fM;
            return;
        }
        o_[0] = zeroed ? 0.0 : scale * f0;
        o_[so * M] = zeroed ? 0.0 : scale * fM;
        mom[p] = f0;
        mom[np + p] = 0.0;
    };
    if (kOwn == 2) {
        constexpr int B = kOwn - 1;
        if (t > 0) {
#pragma unroll
            for (int k2 = 0; k2 < T; ++k2) {
                const int k = k1[0] + R1 * k2;
                const double2 a = x[0][k2], b = x[B][T - 1 - k2];
                emit(k, real_split(a, b, tw2[k]));
                emit(M - k, real_split(b, a, tw2[M - k]));
            }
        } else {
            emit_ends(x[0][0]);
            emit(M / 2, x[0][T / 2]);
#pragma unroll
            for (int k2 = 1; k2 < T / 2; ++k2) {
                const int k = R1 * k2;
                emit(k, real_split(x[0][k2], x[0][T - k2], tw2[k]));
                emit(M - k, real_split(x[0][T - k2], x[0][k2], tw2[M - k]));
            }
#pragma unroll
            for (int k2 = 0; k2 < T; ++k2) {
                const int k = R1 / 2 + R1 * k2;
                emit(k, real_split(x[B][k2], x[B][T - 1 - k2], tw2[k]));
            }
        }
    } else {
        // t = 0 and 1 (the first warp) pair within themselves, others with the lane across
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) {
            const int k = k1[0] + R1 * k2;
            double2 zm;
            if (t >= 2)
                zm = shfl_xor2(x[0][T - 1 - k2], kTile);
            else
                zm = t == 0 ? x[0][(T - k2) % T] : x[0][T - 1 - k2];
            if (k2 == 0 && t == 0)
                emit_ends(x[0][0]);
            else
                emit(k, (t == 0 && 2 * k2 == T) ? x[0][k2] : real_split(x[0][k2], zm, tw2[k]));
        }
    }
}

// Inverse transform of every (J,K) column of the slot array into the
// physical potential, 1/N normalised (the reference's 2/numphi times the
// n/2-scaled NR inverse), with the axis condition phi(1,K,l) =
// phi(2,K,l+N/2) (isym 3: phi(2,K,l)) and the equator condition
// phi(J,1,l) = phi(J,2,l) (isym 2,3) taken at the source: those columns
// transform the source column's spectrum (shifted by N/2 = sign (-1)^k).
// With phieff != nullptr the epilogue also writes the effective potential
// phieff = pot - 0.5 omega^2 rhf(J)^2 that the hydro source step forms from
// pot (source.F90:156, make_source_temp.F90:121), saving it a full pass.
template <int M, int Dense = 0>
__global__ void __launch_bounds__((FftTile<M, false>::kThreads), (FftShape<M, false, Dense>::kMinBlocks))
k_fft_inv(const double *__restrict__ P, double *__restrict__ pot, const double2 *__restrict__ g_tw,
          const double2 *__restrict__ g_tw2, int numr, int numz, int isym, double *__restrict__ phieff,
          const double *__restrict__ rhf, double omega, FftBatch bt) {
    constexpr int kTile = tile_cols<M, false>(), NT = FftTile<M, false>::kThreads;
    constexpr int T = Split<M>::T, R1 = Split<M>::R1, kOwn = Split<M>::kOwn;
    extern __shared__ double2 smem[];
    double2 *C = smem;  // [k1][t][column]
    double2 *tw = C + M * kTile;
    double2 *tw2 = tw + M;
    const int tid = threadIdx.x, c = tid % kTile, t = tid / kTile;
    const long long nplane = (long long)numr * numz;
    const long long q = (long long)blockIdx.x * kTile + c;
    for (int i = tid; i < M; i += NT) tw[i] = g_tw[i];
    for (int i = tid; i <= M; i += NT) tw2[i] = g_tw2[i];
    pdl_wait();
    if (bt.outp) {
        const int pos = blockIdx.y;
        P += (long long)(bt.inst ? bt.inst[pos] : pos) * bt.inst_stride;
        pot = bt.outp[pos];
    }
    const bool valid = q < nplane;
    {
        const int jz = valid ? (int)q % numr : 0, kz = valid ? (int)q / numr : 0;
        const int js = (jz == 0) ? 1 : jz;
        const int ks = (kz == 0 && isym != 1) ? 1 : kz;
        const bool axis = valid && (jz == 0) && (isym != 3);
        const double *col = P + js + (long long)numr * ks;
        double2 x[kOwn][T];
        int k1[kOwn];
#pragma unroll
        for (int o = 0; o < kOwn; ++o) {
            k1[o] = second_digit<M>(t, o);
#pragma unroll
            for (int k2 = 0; k2 < T; ++k2) {
                const int k = k1[o] + R1 * k2;
                x[o][k2] = valid ? make_double2(__ldg(col + nplane * k), __ldg(col + nplane * (M + k)))
                                 : make_double2(0.0, 0.0);
            }
        }
        __syncthreads();  // the twiddles
        // F_k = slot_k - i slot_{M+k}; k = 0 keeps (F_0, F_M), both real.  R1 is even, so the
        // axis columns' sign (-1)^k is that of k1.
#pragma unroll
        for (int o = 0; o < kOwn; ++o) {
            const double s = (axis && (k1[o] & 1)) ? -1.0 : 1.0;
#pragma unroll
            for (int k2 = 0; k2 < T; ++k2)
                if (k2 > 0 || k1[o] > 0) x[o][k2] = make_double2(s * x[o][k2].x, -s * x[o][k2].y);
        }
        // Z_k = E_k + i O_k
        if (kOwn == 2) {
            constexpr int B = kOwn - 1;
            if (t > 0) {
#pragma unroll
                for (int k2 = 0; k2 < T; ++k2) {
                    const int k = k1[0] + R1 * k2;
                    const double2 a = x[0][k2], b = x[B][T - 1 - k2];
                    x[0][k2] = real_merge(a, b, tw2[k]);
                    x[B][T - 1 - k2] = real_merge(b, a, tw2[M - k]);
                }
            } else {
                const double2 f = x[0][0];
                x[0][0] = make_double2(0.5 * (f.x + f.y), 0.5 * (f.x - f.y));
#pragma unroll
                for (int k2 = 1; k2 < T / 2; ++k2) {
                    const int k = R1 * k2;
                    const double2 a = x[0][k2], b = x[0][T - k2];
                    x[0][k2] = real_merge(a, b, tw2[k]);
                    x[0][T - k2] = real_merge(b, a, tw2[M - k]);
                }
#pragma unroll
                for (int k2 = 0; k2 < T / 2; ++k2) {
                    const int k = R1 / 2 + R1 * k2;
                    const double2 a = x[B][k2], b = x[B][T - 1 - k2];
                    x[B][k2] = real_merge(a, b, tw2[k]);
                    x[B][T - 1 - k2] = real_merge(b, a, tw2[M - k]);
                }
            }
        } else {
            if (t >= 2) {  // with the lane across (the first warp holds t = 0 and 1)
#pragma unroll
                for (int k2 = 0; k2 < T / 2; ++k2) {
                    const int ka = k1[0] + R1 * k2, kb = k1[0] + R1 * (T - 1 - k2);
                    const double2 a = x[0][k2], b = x[0][T - 1 - k2];
                    const double2 fa = shfl_xor2(b, kTile), fb = shfl_xor2(a, kTile);
                    x[0][k2] = real_merge(a, fa, tw2[ka]);
                    x[0][T - 1 - k2] = real_merge(b, fb, tw2[kb]);
                }
            } else if (t == 0) {
                const double2 f = x[0][0];
                x[0][0] = make_double2(0.5 * (f.x + f.y), 0.5 * (f.x - f.y));
#pragma unroll
                for (int k2 = 1; k2 < T / 2; ++k2) {
                    const double2 a = x[0][k2], b = x[0][T - k2];
                    x[0][k2] = real_merge(a, b, tw2[R1 * k2]);
                    x[0][T - k2] = real_merge(b, a, tw2[M - R1 * k2]);
                }
            } else {
#pragma unroll
                for (int k2 = 0; k2 < T / 2; ++k2) {
                    const int k = R1 / 2 + R1 * k2;
                    const double2 a = x[0][k2], b = x[0][T - 1 - k2];
                    x[0][k2] = real_merge(a, b, tw2[k]);
                    x[0][T - 1 - k2] = real_merge(b, a, tw2[M - k]);
                }
            }
        }
#pragma unroll
        for (int o = 0; o < kOwn; ++o) {
            dft<T, -1>(x[o]);
            double2 *dst = C + k1[o] * T * kTile + c;
            dst[0] = x[o][0];
#pragma unroll
            for (int n = 1; n < T; ++n) dst[n * kTile] = cmulc(x[o][n], tw[n * k1[o]]);
        }
    }
    __syncthreads();
    double2 v[R1];
    {
        const double2 *in = C + t * kTile + c;
#pragma unroll
        for (int k = 0; k < R1; ++k) v[k] = in[k * T * kTile];
    }
    dft<R1, -1>(v);
    pdl_trigger();
    if (!valid) return;
    const double scale = 1.0 / (double)M;
    double *col = pot + q + nplane * (2 * t);
#pragma unroll
    for (int r = 0; r < R1; ++r) {
        col[nplane * (2 * T * r)] = v[r].x * scale;
        col[nplane * (2 * T * r + 1)] = v[r].y * scale;
    }
    if (phieff) {
        const double rad = rhf[(int)q % numr];
        const double cen = 0.5 * omega * omega * rad * rad;
        double *pe = phieff + q + nplane * (2 * t);
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            pe[nplane * (2 * T * r)] = v[r].x * scale - cen;
            pe[nplane * (2 * T * r + 1)] = v[r].y * scale - cen;
        }
    }
}

template <int M>
cudaError_t set_fft_attrs(bph_ctx *c) {
    const int fwd = (int)FftTile<M, true>::kSmem, inv = (int)FftTile<M, false>::kSmem;
    cudaError_t e = cudaFuncSetAttribute(k_fft_fwd<M, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, fwd);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_fft_fwd<M, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, fwd);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_fft_inv<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, inv);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_fft_fwd<M, true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, fwd);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_fft_inv<M, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, inv);
    c->fft_smem_fwd = fwd;
    c->fft_smem_inv = inv;
    return e;
}

template <int M>
cudaError_t fwd_rho(bph_ctx *c, const double *rho, double *R, double *mom, long long mstride, int *status,
                    FftBatch bt, int npos) {
    constexpr int kTile = tile_cols<M, true>();
    unsigned blocks = (unsigned)((c->np + kTile - 1) / kTile);
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg =
        launch_config(c, dim3(blocks, (unsigned)npos), dim3(FftTile<M, true>::kThreads), FftTile<M, true>::kSmem, attr);
    if (c->fft_dense && !bt.in)
        return cudaLaunchKernelEx(&cfg, k_fft_fwd<M, true, 1>, rho, R, mom, (const double2 *)c->d_tw,
                                  (const double2 *)c->d_tw2, (const double2 *)c->d_ph, c->g.numr, c->g.numz, c->nr,
                                  c->nz, c->g.mmax, c->fm, c->g.isym, c->four_pi, status, mstride, bt);
    return cudaLaunchKernelEx(&cfg, k_fft_fwd<M, true>, rho, R, mom, (const double2 *)c->d_tw,
                              (const double2 *)c->d_tw2, (const double2 *)c->d_ph, c->g.numr, c->g.numz, c->nr,
                              c->nz, c->g.mmax, c->fm, c->g.isym, c->four_pi, status, mstride, bt);
}

template <int M>
cudaError_t fwd_pot(bph_ctx *c, const double *pot) {
    constexpr int kTile = tile_cols<M, true>();
    unsigned blocks = (unsigned)((c->np + kTile - 1) / kTile);
    k_fft_fwd<M, false><<<blocks, FftTile<M, true>::kThreads, FftTile<M, true>::kSmem, c->stream>>>(
        pot, c->d_P, nullptr, c->d_tw, c->d_tw2, c->d_ph, c->g.numr, c->g.numz, c->nr, c->nz, c->g.mmax, c->fm,
        c->g.isym, c->four_pi, c->d_status, 0, FftBatch());
    return cudaGetLastError();
}

template <int M>
cudaError_t inv(bph_ctx *c, double *pot, double *phieff, double omega, const double *P, FftBatch bt, int npos) {
    constexpr int kTile = tile_cols<M, false>();
    unsigned blocks = (unsigned)((c->nplane + kTile - 1) / kTile);
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg =
        launch_config(c, dim3(blocks, (unsigned)npos), dim3(FftTile<M, false>::kThreads), FftTile<M, false>::kSmem, attr);
    if (c->fft_dense && !bt.outp)
        return cudaLaunchKernelEx(&cfg, k_fft_inv<M, 1>, P, pot, (const double2 *)c->d_tw, (const double2 *)c->d_tw2,
                                  c->g.numr, c->g.numz, c->g.isym, phieff, (const double *)c->d_grid, omega, bt);
    return cudaLaunchKernelEx(&cfg, k_fft_inv<M>, P, pot, (const double2 *)c->d_tw, (const double2 *)c->d_tw2,
                              c->g.numr, c->g.numz, c->g.isym, phieff, (const double *)c->d_grid, omega, bt);
}

#define BPH_FFT_DISPATCH(FN, ...)                  \
    switch (c->M) {                                \
        case 8: return FN<8>(__VA_ARGS__);         \
        case 16: return FN<16>(__VA_ARGS__);       \
        case 32: return FN<32>(__VA_ARGS__);       \
        case 64: return FN<64>(__VA_ARGS__);       \
        case 128: return FN<128>(__VA_ARGS__);     \
        case 256: return FN<256>(__VA_ARGS__);     \
        default: return cudaErrorInvalidValue;     \
    }

cudaError_t set_attrs_dispatch(bph_ctx *c) { BPH_FFT_DISPATCH(set_fft_attrs, c) }
cudaError_t fwd_rho_dispatch(bph_ctx *c, const double *rho, double *R, double *mom, long long mstride, int *status,
                             FftBatch bt, int npos) {
    BPH_FFT_DISPATCH(fwd_rho, c, rho, R, mom, mstride, status, bt, npos)
}
cudaError_t fwd_pot_dispatch(bph_ctx *c, const double *pot) { BPH_FFT_DISPATCH(fwd_pot, c, pot) }
cudaError_t inv_dispatch(bph_ctx *c, double *pot, double *phieff, double omega, const double *P, FftBatch bt,
                         int npos) {
    BPH_FFT_DISPATCH(inv, c, pot, phieff, omega, P, bt, npos)
}

}  // namespace

int fft_configure(bph_ctx *c) {
    const char *dense = std::getenv("BPH_FFT_DENSE");
    c->fft_dense = dense && dense[0] == '1';
    cudaError_t e = set_attrs_dispatch(c);
    if (e != cudaSuccess) return cuda_fail(e, "fft_configure");
    return BPH_OK;
}

cudaError_t launch_fft_fwd_rho(bph_ctx *c, const double *rho, double *R, double *mom, long long mstride,
                               int *status) {
    ++c->launches;
    return fwd_rho_dispatch(c, rho, R ? R : c->d_R, mom ? mom : c->d_mom, mstride ? mstride : 2 * c->np,
                            status ? status : c->d_status, FftBatch(), 1);
}

cudaError_t launch_fft_fwd_pot(bph_ctx *c, const double *pot) {
    ++c->launches;
    return fwd_pot_dispatch(c, pot);
}

cudaError_t launch_fft_inv(bph_ctx *c, double *pot, double *phieff, double omega, const double *P) {
    ++c->launches;
    return inv_dispatch(c, pot, phieff, omega, P ? P : c->d_P, FftBatch(), 1);
}

cudaError_t launch_fft_fwd_rho_batch(bph_ctx *c, int npos, const double *const *d_in, const int *d_inst, double *R,
                                     long long inst_stride, double *mom, long long mstride, long long pos_stride,
                                     int *status, bool status_per_pos) {
    FftBatch bt;
    bt.in = d_in;
    bt.status_stride = status_per_pos ? 1 : 0;
    bt.inst = d_inst;
    bt.inst_stride = inst_stride;
    bt.pos_stride = pos_stride;
    ++c->launches;
    return fwd_rho_dispatch(c, nullptr, R, mom, mstride, status, bt, npos);
}

cudaError_t launch_fft_inv_batch(bph_ctx *c, int npos, double *const *d_out, const int *d_inst, const double *P,
                                 long long inst_stride) {
    FftBatch bt;
    bt.outp = d_out;
    bt.inst = d_inst;
    bt.inst_stride = inst_stride;
    ++c->launches;
    return inv_dispatch(c, nullptr, nullptr, 0.0, P, bt, npos);
}

}  // namespace bph
