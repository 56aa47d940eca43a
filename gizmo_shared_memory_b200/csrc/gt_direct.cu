// O(N_targets * N) direct summation: the replacement for shmem::accel_brute (shmem/tree.cc:946-971)
// and for the reference's only CUDA kernel, accel_bruteforce_kernel (shmem/grav_cuda.cu:66-141).
//
// Each block holds 256 targets in registers, two per thread, and streams one contiguous chunk of the
// sources through shared memory in tiles of 256; the grid's second dimension splits the sources so that
// a few thousand targets (the error sample) still fill all 148 SMs.  Per-chunk partial sums go to a
// scratch array and a second kernel adds the chunks in a fixed order, so results are deterministic.
//   FP64: every operation in double, the pair rule of tree.cc:39-53 with zeta = 0 (kernel of the
//         larger softening, self and r == 0 skipped) -- the error oracle of the walk.
//   FP32: the pair offset is differenced in double and narrowed, everything after it is float
//         (grav_cuda.cu:108-134 without zeta terms or a periodic wrap).
#include <algorithm>
#include <climits>
#include <cmath>
#include <mutex>
#include <type_traits>

#include "gt_internal.cuh"

// Fixed scratch of the allocation-free entry point gt_direct_noalloc: the per-chunk partial sums,
// 8 MiB, present on every GPU that loads this library until the process exits.  Host code must
// never pass this name to a kernel -- on the host it is only a stand-in symbol; its device address
// comes from cudaGetSymbolAddress (see noalloc_scratch below).
static __device__ __align__(256) double g_direct_noalloc_scratch[GT_DIRECT_NOALLOC_SCRATCH_DOUBLES];

namespace gt {
namespace {

constexpr int kDirThreads = 128;
constexpr int kDirPer = 2;  // targets per thread
constexpr int kDirTile = 256;
constexpr int kDirUnroll = 4;  // sources per iteration

__device__ __forceinline__ void spline_d(double r, double h, double& f, double& p) {
    const double hinv = 1.0 / h;
    const double u = r * hinv;
    if (u >= 1.0) {
        f = 1.0 / (r * r * r);
        p = -1.0 / r;
        return;
    }
    const double hinv3 = hinv * hinv * hinv;
    if (u < 0.5) {
        f = hinv3 * (10.666666666666667 + u * u * (32.0 * u - 38.4));
        p = hinv * (-2.8 + u * u * (5.333333333333333 + u * u * (6.4 * u - 9.6)));
    } else {
        f = hinv3 * (21.333333333333332 - 48.0 * u + 38.4 * u * u - 10.666666666666667 * u * u * u -
                     0.06666666666666667 / (u * u * u));
        p = hinv * (-3.2 + 0.06666666666666667 / u +
                    u * u * (10.666666666666667 + u * (-16.0 + u * (9.6 - 2.1333333333333333 * u))));
    }
}

__device__ __forceinline__ void spline_f(float r, float h, float& f, float& p) {
    const float hinv = 1.0f / h;
    const float u = r * hinv;
    if (u >= 1.0f) {
        const float ri = 1.0f / r;
        f = ri * ri * ri;
        p = -ri;
        return;
    }
    const float hinv3 = hinv * hinv * hinv;
    if (u < 0.5f) {
        f = hinv3 * (10.666666666666667f + u * u * (32.0f * u - 38.4f));
        p = hinv * (-2.8f + u * u * (5.333333333333333f + u * u * (6.4f * u - 9.6f)));
    } else {
        const float u3 = u * u * u;
        f = hinv3 * (21.333333333333332f - 48.0f * u + 38.4f * u * u - 10.666666666666667f * u3 -
                     0.06666666666666667f / u3);
        p = hinv * (-3.2f + 0.06666666666666667f / u +
                    u * u * (10.666666666666667f + u * (-16.0f + u * (9.6f - 2.1333333333333333f * u))));
    }
}

// dW/dr of the 3-D cubic spline of support h (shmem/hydro.h:46-54), FP64, zero from r = h.
__device__ __forceinline__ double kernel_dwdr_d(double r, double h) {
    const double q = r / h;
    if (q >= 1.0) return 0.0;
    const double norm = 8.0 / (M_PI * h * h * h);
    double fp;
    if (q < 0.5) {
        fp = -12.0 * q + 18.0 * q * q;
    } else {
        const double u = 1.0 - q;
        fp = -6.0 * u * u;
    }
    return norm * fp / h;
}

// One pair of two particles in double with every case of the pair rule: r = 0, the spline inside the
// larger softening, the zeta terms of a gas-gas pair.
// GAS: the adaptive-softening zeta terms of gas-gas pairs (tree.cc:39-53); type (0 = gas; null =
// every particle gas) and zeta (null = none) are indexed like the particles.
struct GasTarget {
    double tzm = 0.0, tm = 0.0, tzeta = 0.0;  // zeta_t / m_t, m_t and zeta_t of a gas target
    bool gas = false;
};
template <bool GAS>
__device__ __noinline__ void pair_d(double ox, double oy, double oz, double ps, double ss, double m,
                                    const GasTarget& gt, double szeta, bool sgas, double& mf, double& mp) {
    mf = mp = 0.0;
    const double r = sqrt(ox * ox + oy * oy + oz * oz);
    if (r <= 0) return;
    const double e = fmax(fmax(ps, ss), 1e-300);
    double f, p;
    spline_d(r, e, f, p);
    mf = m * f;
    mp = m * p;
    if (GAS && gt.gas && sgas && gt.tm > 0.0) {
        const double es = fmax(ss, 1e-300);
        if (gt.tzeta != 0.0 && r < e) mf -= gt.tzm * kernel_dwdr_d(r, e) / r;
        if (szeta != 0.0 && r < es) mf -= (szeta / gt.tm) * kernel_dwdr_d(r, es) / r;
    }
}

__device__ __noinline__ void pair_f(float dx, float dy, float dz, float ps, float ss, float m, float& mf, float& mp) {
    mf = mp = 0.0f;
    const float r2 = dx * dx + dy * dy + dz * dz;
    if (r2 <= 0.0f) return;
    float e = fmaxf(ps, ss);
    if (!(e > 0.0f)) e = 1e-30f;
    float f, p;
    spline_f(sqrtf(r2), e, f, p);
    mf = m * f;
    mp = m * p;
}

// The sources of one tile, in the order the inner loop reads them: two 16-byte broadcasts of shared
// memory give position and mass, a word the limit below which a pair leaves the short path.
struct alignas(16) DirSrc {
    double x, y, z, m;
};

// 1/sqrt(x) of a normal x: the approximate reciprocal square root y, then one step of the binomial
// series of (1 - e)^(-1/2) about it, y (1 + e/2 + 3/8 e^2) with e = 1 - x y^2.  The approximation's
// relative error is below 2^-20, so e is below 2^-19 and the term left out, 5/16 e^3, below 2^-58: the
// result is off by the rounding of the step's few operations (tests/test_gpu_parity.py bounds the
// direct sum against the oracle).  Five FP64 instructions and no branch, so that the pairs of an
// iteration overlap; the library function's check for special operands would keep them apart.
__device__ __forceinline__ double rsqrt_d(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y * y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// A pair inside the larger softening, or within a part in 10^6 of it, at a normal r^2: the spline of
// spline_d from 1/r by rsqrt_d and 1/h, which every target and source brings along, so that no
// division or square root and no branch keeps the pairs of an iteration apart.  hinv = 1/h.
__device__ __forceinline__ void inside_d(double r2, double h, double hinv, double& ri, double& u, double& f,
                                         double& p) {
    ri = rsqrt_d(r2);
    u = r2 * ri * hinv;
    const double u2 = u * u, iu = h * ri, hinv3 = hinv * hinv * hinv;
    const bool low = u < 0.5;
    f = low ? 10.666666666666667 + u2 * (32.0 * u - 38.4)
            : 21.333333333333332 - 48.0 * u + 38.4 * u2 - 10.666666666666667 * u2 * u -
                  0.06666666666666667 * (iu * iu * iu);
    p = low ? -2.8 + u2 * (5.333333333333333 + u2 * (6.4 * u - 9.6))
            : -3.2 + 0.06666666666666667 * iu +
                  u2 * (10.666666666666667 + u * (-16.0 + u * (9.6 - 2.1333333333333333 * u)));
    f = u < 1.0 ? hinv3 * f : ri * (ri * ri);
    p = u < 1.0 ? hinv * p : -ri;
}
// dW/dr / r (kernel_dwdr_d) from u = r / h
__device__ __forceinline__ double dwdr_r_d(double u, double ri, double hinv) {
    const double v = 1.0 - u, fp = u < 0.5 ? -12.0 * u + 18.0 * u * u : -6.0 * v * v;
    return u < 1.0 ? (8.0 / M_PI) * (hinv * hinv) * (hinv * hinv) * fp * ri : 0.0;
}
// The same in FP32; the root is corrected by its remainder.
__device__ __forceinline__ void inside_f(float r2, float h, float hinv, float& f, float& p) {
    const float ri = rsqrtf(r2);
    float r = r2 * ri;
    r = fmaf(fmaf(-r, r, r2), 0.5f * ri, r);
    const float u = r * hinv, u2 = u * u, iu = h * ri, hinv3 = hinv * hinv * hinv;
    const bool low = u < 0.5f;
    f = low ? 10.666666666666667f + u2 * (32.0f * u - 38.4f)
            : 21.333333333333332f - 48.0f * u + 38.4f * u2 - 10.666666666666667f * u2 * u -
                  0.06666666666666667f * (iu * iu * iu);
    p = low ? -2.8f + u2 * (5.333333333333333f + u2 * (6.4f * u - 9.6f))
            : -3.2f + 0.06666666666666667f * iu +
                  u2 * (10.666666666666667f + u * (-16.0f + u * (9.6f - 2.1333333333333333f * u)));
    f = u < 1.0f ? hinv3 * f : ri * ri * ri;
    p = u < 1.0f ? hinv * p : -ri;
}

// Direct sum of kDirPer targets per thread over one chunk of the sources.
//
// What bounds it: the FP64 pipe (64 lanes a clock per SM).  A pair outside both softenings needs 18
// FP64 instructions -- 3 differences, 3 for r^2, 5 for the reciprocal square root, 3 products for
// m / r^3, 3 + 1 accumulations -- and that path holds nothing else in double: whether a pair is
// outside is an integer comparison of the high words of r^2 and of the larger squared softening.  The
// high word rounds down, so pairs within one part in 10^6 of the softening, the pair of a particle
// with itself, r = 0 and every subnormal, infinite or NaN r^2 are left out of it (1/r taken
// as 0) and evaluated after the iteration's pairs, by inside_d at an ordinary r^2 and else by pair_d,
// which treats each case as the rule says: one branch per kDirUnroll sources and kDirPer targets, rarely
// taken, instead of one per pair, which kept every pair's chain of dependent instructions to itself.
// 4096 targets against 262,144 sources: 5.47 -> 1.48 ms, 0.77 of the FP64 peak (34 TF/s) counting an
// instruction as two operations.
// Where a softening holds most of a warp's pairs of a tile, the short path is work for nothing, and the
// next tile is evaluated by inside_d alone.  20,000 particles against each other with all pairs inside:
// 2.03 ms with one branch per pair, 4.22 with the short path and pair_d, 2.51 with inside_d, 2.09 this way
// (FP32 1.42, 2.63, 1.91, 1.42).
//   FP32: the offset is differenced in double and narrowed, the interaction is FP32 with the
//   approximate reciprocal square root, and each tile's FP32 sums are added into double totals.
template <bool FP64, bool GAS = false>
__global__ void __launch_bounds__(kDirThreads)
direct_kernel(const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z,
              const double* __restrict__ m, const double* __restrict__ soft, int64_t n,
              const uint32_t* __restrict__ targets, int64_t nt, int64_t chunk,
              double* __restrict__ partial, const uint8_t* __restrict__ type = nullptr,
              const double* __restrict__ zeta = nullptr) {
    __shared__ DirSrc sh[kDirTile];
    __shared__ double shs[kDirTile];
    __shared__ std::conditional_t<FP64, double, float> shi[kDirTile];  // 1 / softening
    __shared__ int shlim[kDirTile];
    __shared__ float shm[FP64 ? 1 : kDirTile];
    __shared__ double shzeta[GAS ? kDirTile : 1];
    __shared__ unsigned char shgas[GAS ? kDirTile : 1];
    // high word of the square of a softening: r^2 above it lies outside
    auto limit = [](double s) {
        if (FP64) return max(__double2hiint(s * s), 0x000fffff);  // at least every subnormal r^2
        const float f = (float)s;
        return __float_as_int(f * f);
    };
    auto inverse = [](double s) {
        if constexpr (FP64) return 1.0 / fmax(s, 1e-300);
        else return 1.0f / ((float)s > 0.0f ? (float)s : 1e-30f);
    };
    const int64_t t0 = (int64_t)blockIdx.x * (kDirThreads * kDirPer) + threadIdx.x;
    int64_t self[kDirPer];
    std::conditional_t<FP64, double, float> pinv[kDirPer];
    double px[kDirPer], py[kDirPer], pz[kDirPer], ps[kDirPer];
    int plim[kDirPer];
    GasTarget gas[GAS ? kDirPer : 1];
    double ax[kDirPer], ay[kDirPer], az[kDirPer], ap[kDirPer];
#pragma unroll
    for (int k = 0; k < kDirPer; ++k) {
        // a target index at or beyond n (device target arrays are not checked on the host) reads
        // nothing; its outputs are zero
        const int64_t t = t0 + k * kDirThreads;
        self[k] = t < nt ? (int64_t)targets[t] : n;
        const bool live = self[k] < n;
        // (a target that is none is far from everything, so that its pairs stay on the short path)
        constexpr double kFar = FP64 ? 1e150 : 1e15;
        px[k] = live ? x[self[k]] : kFar;
        py[k] = live ? y[self[k]] : kFar;
        pz[k] = live ? z[self[k]] : kFar;
        ps[k] = (live && soft) ? soft[self[k]] : 0.0;
        plim[k] = limit(ps[k]);
        pinv[k] = inverse(ps[k]);
        ax[k] = ay[k] = az[k] = ap[k] = 0.0;
        if (GAS && live) {
            GasTarget& g = gas[GAS ? k : 0];
            g.gas = !type || type[self[k]] == 0;
            g.tzeta = zeta ? zeta[self[k]] : 0.0;
            g.tm = m[self[k]];
            if (g.tm > 0) g.tzm = g.tzeta / g.tm;
        }
    }
    const int64_t s0 = (int64_t)blockIdx.y * chunk, s1 = min(n, s0 + chunk);
    int n_live = 0;          // targets of this warp
#pragma unroll
    for (int k = 0; k < kDirPer; ++k) n_live += __popc(__ballot_sync(0xffffffffu, self[k] < n));
    bool soft_tile = false;  // most of this warp's pairs of the last tile were inside a softening
    for (int64_t base = s0; base < s1; base += kDirTile) {
        for (int q = threadIdx.x; q < kDirTile; q += kDirThreads) {
            const int64_t j = base + q;
            if (j >= s1) {
                shlim[q] = INT_MAX;  // past the chunk: every pair is left out of the short path
                sh[q] = DirSrc{0.0, 0.0, 0.0, 0.0};
                shs[q] = 0.0;
                shi[q] = 1;
                if (!FP64) shm[q] = 0.0f;
                continue;
            }
            // a mass that is no number times the 0 of a pair left out would be none either: such a
            // source weighs nothing on the short path and takes all its pairs off it
            const double mj = m[j];
            const bool fin = isfinite(FP64 ? mj : (double)(float)mj);
            sh[q] = DirSrc{x[j], y[j], z[j], fin ? mj : 0.0};
            const double s = soft ? soft[j] : 0.0;
            shs[q] = s;
            shi[q] = inverse(s);
            shlim[q] = fin ? limit(s) : INT_MAX;
            if (!FP64) shm[q] = fin ? (float)mj : 0.0f;
            if (GAS) {
                shzeta[q] = zeta ? zeta[j] : 0.0;
                shgas[q] = (!type || type[j] == 0) ? 1 : 0;
            }
        }
        __syncthreads();
        const int nq = (int)min((int64_t)kDirTile, s1 - base);
        float fx[kDirPer], fy[kDirPer], fz[kDirPer], fp[kDirPer];
#pragma unroll
        for (int k = 0; k < kDirPer; ++k) fx[k] = fy[k] = fz[k] = fp[k] = 0.0f;
        int inside = 0;
        for (int q0 = 0; q0 < nq; q0 += kDirUnroll) {
            unsigned slow = soft_tile ? (1u << (kDirUnroll * kDirPer)) - 1u : 0u;
            if (!soft_tile)
#pragma unroll
            for (int i = 0; i < kDirUnroll; ++i) {
                const int q = q0 + i;
                const DirSrc s = sh[q];
                const int sl = shlim[q];
#pragma unroll
                for (int k = 0; k < kDirPer; ++k) {
                    const double ox = s.x - px[k], oy = s.y - py[k], oz = s.z - pz[k];
                    const int lim = max(plim[k], sl);
                    if (FP64) {
                        const double r2 = ox * ox + oy * oy + oz * oz;
                        const int hi = __double2hiint(r2);
                        const bool ok = hi > lim && hi < 0x7ff00000;
                        if (!ok) slow |= 1u << (i * kDirPer + k);
                        const double ri = ok ? rsqrt_d(r2) : 0.0;
                        const double mri = s.m * ri;
                        const double mf = mri * (ri * ri);
                        ax[k] += ox * mf; ay[k] += oy * mf; az[k] += oz * mf;
                        ap[k] -= mri;
                    } else {
                        const float dx = (float)ox, dy = (float)oy, dz = (float)oz;
                        const float r2 = dx * dx + dy * dy + dz * dz;
                        const int hi = __float_as_int(r2);
                        const bool ok = hi > lim && hi < 0x7f800000;
                        if (!ok) slow |= 1u << (i * kDirPer + k);
                        const float ri = ok ? rsqrtf(r2) : 0.0f;
                        const float mri = shm[q] * ri;
                        const float mf = mri * (ri * ri);
                        fx[k] += dx * mf; fy[k] += dy * mf; fz[k] += dz * mf;
                        fp[k] -= mri;
                    }
                }
            }
            if (!soft_tile) inside += __popc(slow);
            if (slow) {
                unsigned odd = 0;  // pairs for the rule in full
#pragma unroll 2
                for (int i = 0; i < kDirUnroll; ++i) {
                    const int q = q0 + i;
                    if (((slow >> (i * kDirPer)) & ((1u << kDirPer) - 1u)) == 0u || q >= nq) continue;
                    const DirSrc s = sh[q];
                    const double ss = shs[q];
                    const bool plain = shlim[q] != INT_MAX;
#pragma unroll
                    for (int k = 0; k < kDirPer; ++k) {
                        const unsigned bit = 1u << (i * kDirPer + k);
                        const bool take = (slow & bit) != 0u && base + q != self[k];
                        const double ox = s.x - px[k], oy = s.y - py[k], oz = s.z - pz[k];
                        if constexpr (FP64) {
                            const double r2 = ox * ox + oy * oy + oz * oz;
                            const int hi = __double2hiint(r2);
                            const bool ok = plain && hi >= 0x00100000 && hi < 0x7ff00000;
                            if (take && !ok) odd |= bit;
                            if (soft_tile && hi <= max(plim[k], shlim[q])) ++inside;
                            double ri, u, f, p;
                            inside_d(r2, fmax(fmax(ps[k], ss), 1e-300), fmin(pinv[k], shi[q]), ri, u, f, p);
                            double mf = s.m * f;
                            if (GAS && gas[GAS ? k : 0].gas && shgas[q] && gas[GAS ? k : 0].tm > 0.0) {
                                const GasTarget& g = gas[GAS ? k : 0];
                                if (g.tzeta != 0.0) mf -= g.tzm * dwdr_r_d(u, ri, fmin(pinv[k], shi[q]));
                                if (shzeta[q] != 0.0) mf -= shzeta[q] / g.tm * dwdr_r_d(r2 * ri * shi[q], ri, shi[q]);
                            }
                            if (take && ok) {
                                ax[k] += ox * mf; ay[k] += oy * mf; az[k] += oz * mf;
                                ap[k] += s.m * p;
                            }
                        } else {
                            const float dx = (float)ox, dy = (float)oy, dz = (float)oz;
                            const float r2 = dx * dx + dy * dy + dz * dz;
                            const int hi = __float_as_int(r2);
                            const bool ok = plain && hi >= 0x00800000 && hi < 0x7f800000;
                            if (take && !ok) odd |= bit;
                            if (soft_tile && hi <= max(plim[k], shlim[q])) ++inside;
                            const float h = fmaxf((float)ps[k], (float)ss);
                            float f, p;
                            inside_f(r2, h > 0.0f ? h : 1e-30f, fminf(pinv[k], shi[q]), f, p);
                            const float mf = shm[q] * f;
                            if (take && ok) {
                                fx[k] += dx * mf; fy[k] += dy * mf; fz[k] += dz * mf;
                                fp[k] += shm[q] * p;
                            }
                        }
                    }
                }
#pragma unroll 1
                for (int i = 0; odd != 0u && i < kDirUnroll; ++i)
#pragma unroll
                    for (int k = 0; k < kDirPer; ++k) {
                        if (!((odd >> (i * kDirPer + k)) & 1u)) continue;
                        const int q = q0 + i;
                        const DirSrc s = sh[q];
                        const double ox = s.x - px[k], oy = s.y - py[k], oz = s.z - pz[k];
                        const double mj = __ldg(m + base + q);  // as it was given
                        if (FP64) {
                            double mf, mp;
                            pair_d<GAS>(ox, oy, oz, ps[k], shs[q], mj, gas[GAS ? k : 0], GAS ? shzeta[q] : 0.0,
                                        GAS && shgas[q], mf, mp);
                            ax[k] += ox * mf; ay[k] += oy * mf; az[k] += oz * mf;
                            ap[k] += mp;
                        } else {
                            const float dx = (float)ox, dy = (float)oy, dz = (float)oz;
                            float mf, mp;
                            pair_f(dx, dy, dz, (float)ps[k], (float)shs[q], (float)mj, mf, mp);
                            fx[k] += dx * mf; fy[k] += dy * mf; fz[k] += dz * mf;
                            fp[k] += mp;
                        }
                    }
            }
        }
        soft_tile = 2 * __reduce_add_sync(0xffffffffu, inside) > n_live * nq;
        if (!FP64) {
#pragma unroll
            for (int k = 0; k < kDirPer; ++k) {
                ax[k] += (double)fx[k]; ay[k] += (double)fy[k]; az[k] += (double)fz[k];
                ap[k] += (double)fp[k];
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < kDirPer; ++k) {
        const int64_t t = t0 + k * kDirThreads;
        if (t >= nt) continue;
        const bool live = self[k] < n && n > 1;  // the sum over no other particle is 0, wherever it is
        double* P = partial + (int64_t)blockIdx.y * 4 * nt;
        P[t] = live ? ax[k] : 0.0;
        P[nt + t] = live ? ay[k] : 0.0;
        P[2 * nt + t] = live ? az[k] : 0.0;
        P[3 * nt + t] = live ? ap[k] : 0.0;
    }
}

__global__ void direct_reduce_kernel(const double* __restrict__ partial, int64_t nt, int nchunk, double G,
                                     double* __restrict__ ax, double* __restrict__ ay, double* __restrict__ az,
                                     double* __restrict__ phi) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nt;
         t += (int64_t)gridDim.x * blockDim.x) {
        double s[4] = {0, 0, 0, 0};
        for (int c = 0; c < nchunk; ++c)
            for (int k = 0; k < 4; ++k) s[k] += partial[((int64_t)c * 4 + k) * nt + t];
        if (ax) ax[t] = G * s[0];
        if (ay) ay[t] = G * s[1];
        if (az) az[t] = G * s[2];
        if (phi) phi[t] = G * s[3];
    }
}

// Source chunking: enough chunks that (target blocks x chunks) fills the GPU, at most
// `max_chunks`.  Returns the chunk length and sets nchunk.
int64_t plan_chunks(int64_t n, int64_t nt, int num_sms, int64_t max_chunks, int& nchunk) {
    const int bx = div_up(nt, kDirThreads * kDirPer);
    int64_t c = std::max(1, div_up((int64_t)num_sms * 4, bx));
    c = std::min<int64_t>(c, std::max<int64_t>(1, div_up(n, 2 * kDirTile)));
    c = std::min<int64_t>(c, std::min<int64_t>(65535, std::max<int64_t>(1, max_chunks)));
    const int64_t chunk = std::max<int64_t>(1, div_up(n, c));
    nchunk = std::max(1, div_up(n, chunk));
    return chunk;
}

void launch_direct(cudaStream_t st, int num_sms, int64_t n, const double* x, const double* y,
                   const double* z, const double* m, const double* soft, int64_t nt,
                   const uint32_t* targets, double G, int precision, double* ax, double* ay,
                   double* az, double* phi, double* partial, int nchunk, int64_t chunk) {
    const dim3 grid(div_up(nt, kDirThreads * kDirPer), nchunk);
    if (precision == GT_DIRECT_FP32)
        direct_kernel<false><<<grid, kDirThreads, 0, st>>>(x, y, z, m, soft, n, targets, nt, chunk, partial);
    else
        direct_kernel<true><<<grid, kDirThreads, 0, st>>>(x, y, z, m, soft, n, targets, nt, chunk, partial);
    direct_reduce_kernel<<<std::max(1, std::min(div_up(nt, 256), num_sms * 4)), 256, 0, st>>>(
        partial, nt, nchunk, G, ax, ay, az, phi);
}

}  // namespace

void run_direct_gas(gt_context* ctx, int64_t n, const double* x, const double* y, const double* z, const double* m,
                    const double* soft, const uint8_t* type, const double* zeta, int64_t nt, const uint32_t* targets,
                    double G, double* ax, double* ay, double* az) {
    if (nt <= 0) return;
    int nchunk = 1;
    const int64_t chunk = plan_chunks(n, nt, ctx->num_sms, 65535, nchunk);
    double* partial = (double*)scratch(ctx, kSlotDirect, (size_t)nchunk * 4 * nt * 8);
    const dim3 grid(div_up(nt, kDirThreads * kDirPer), nchunk);
    direct_kernel<true, true><<<grid, kDirThreads, 0, ctx->stream>>>(x, y, z, m, soft, n, targets, nt, chunk, partial,
                                                                     type, zeta);
    direct_reduce_kernel<<<std::max(1, std::min(div_up(nt, 256), ctx->num_sms * 4)), 256, 0, ctx->stream>>>(
        partial, nt, nchunk, G, ax, ay, az, nullptr);
    ctx->launches += 2;
    check_cuda(cudaGetLastError(), "direct_kernel");
}

void run_direct(gt_context* ctx, int64_t n, const double* x, const double* y, const double* z,
                const double* m, const double* soft, int64_t nt, const uint32_t* targets, double G,
                int precision, double* ax, double* ay, double* az, double* phi) {
    if (nt <= 0) return;
    int nchunk = 1;
    const int64_t chunk = plan_chunks(n, nt, ctx->num_sms, 65535, nchunk);
    double* partial = (double*)scratch(ctx, kSlotDirect, (size_t)nchunk * 4 * nt * 8);
    launch_direct(ctx->stream, ctx->num_sms, n, x, y, z, m, soft, nt, targets, G, precision, ax, ay,
                  az, phi, partial, nchunk, chunk);
    ctx->launches += 2;
    check_cuda(cudaGetLastError(), "direct_kernel");
}

}  // namespace gt

// ---------------------------------------------------------------------------------------------
// gt_direct_noalloc: the direct sum for callers that must not allocate device memory
// ---------------------------------------------------------------------------------------------
namespace {

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
double* g_noalloc_ptr[kNoAllocMaxDevices] = {};
int g_noalloc_sms[kNoAllocMaxDevices] = {};

// Device address of g_direct_noalloc_scratch on `dev` (which is current), looked up once per device.
int noalloc_scratch(int dev, double** ptr, int* sms) {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_direct_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            cudaGetLastError();
            return GT_ERR_CUDA;
        }
        int nsm = 0;
        e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess || nsm <= 0) {
            cudaGetLastError();
            return GT_ERR_CUDA;
        }
        g_noalloc_sms[dev] = nsm;
        g_noalloc_ptr[dev] = (double*)p;
    }
    *ptr = g_noalloc_ptr[dev];
    *sms = g_noalloc_sms[dev];
    return GT_OK;
}

}  // namespace

extern "C" int gt_direct_noalloc(int64_t n, const double* x, const double* y, const double* z,
                                 const double* m, const double* soft, int64_t n_targets,
                                 const uint32_t* targets, double G, int precision, double* ax,
                                 double* ay, double* az, double* phi, void* stream) {
    if (n < 0 || n_targets < 0) return GT_ERR_INVALID;
    if (n > 0 && (!x || !y || !z || !m)) return GT_ERR_INVALID;
    if (n_targets > 0 && (!targets || !ax || !ay || !az)) return GT_ERR_INVALID;
    if (precision != GT_DIRECT_FP64 && precision != GT_DIRECT_FP32) return GT_ERR_INVALID;
    if (n_targets > GT_DIRECT_NOALLOC_MAX_TARGETS) return GT_ERR_OVERFLOW;
    if (n_targets == 0) return GT_OK;
    if (n == 0) return GT_ERR_INVALID;  // no particle can be a target
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) {
        cudaGetLastError();
        return GT_ERR_DEVICE;
    }
    double* partial = nullptr;
    int sms = 0;
    const int st = noalloc_scratch(dev, &partial, &sms);
    if (st != GT_OK) return st;
    // every (chunk, target) partial the reduction reads is written by this call's first kernel,
    // so the scratch needs no clearing; the chunk count is capped so the partials fit
    const int64_t max_chunks = GT_DIRECT_NOALLOC_SCRATCH_DOUBLES / (4 * n_targets);
    int nchunk = 1;
    const int64_t chunk = gt::plan_chunks(n, n_targets, sms, max_chunks, nchunk);
    gt::launch_direct((cudaStream_t)stream, sms, n, x, y, z, m, soft, n_targets, targets, G, precision,
                      ax, ay, az, phi, partial, nchunk, chunk);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? GT_OK : GT_ERR_CUDA;
}
