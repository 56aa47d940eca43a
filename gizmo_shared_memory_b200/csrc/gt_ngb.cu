// Neighbour search and the density solve on the gravity tree: shmem::ngb_search,
// ngb_search_reverse and density (shmem/hydro.h:65-117, hydro.cc:37-327), with the per-node hmax
// of Tree::init_hmax / raise_hmax (tree.cc:287-338).
//
// The search prunes against each node's BOX, not its centre of mass: a 32-byte search node holds
// the float geometric centre and a conservative half side (the build's half side plus 1e-6 of the
// root side plus four float ulps of the largest centre coordinate, tree.cc:490-505), with the
// reference's threading (first child / next).  One thread follows the threading for one centre,
// as the reference's loop does, so every list comes out in tree order -- the reference's order --
// and the density sums accumulate in the reference's order too.  The leaves a thread reaches wait in
// a small buffer, and their particles are tested in a run, where the lanes of a warp meet again.  In
// the density solve a lane whose target is done takes another, and targets with very many candidates
// go to a warp each, which sums in the same order.
//
// Lists are CSR: a counting pass, an exclusive scan, and a filling pass over the same traversal.
//
// Forests (gt_build_systems): roots 0 .. n_systems-1 each stand alone in the threading.  A centre
// searches every system in turn, or the one system its caller names; a density target searches the
// system that owns its particle index.  Each system's search nodes are padded by its own root side,
// so a system searched in a forest finds what it finds in a tree of its own.
//
// SHMEM_NGB_COUNT (hydro.cc:7-35): a context with counting on tallies, per gather search, the nodes
// visited, the particles examined, the neighbours kept and the nodes admitted only by the staleness
// pad, and per density target the iterations it took; the counting variants of the kernels are
// separate instantiations, so the plain ones keep their code.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <vector>

#include "gt_internal.cuh"

namespace gt {
namespace {

constexpr int kBlk = 128;

int grid_of(gt_context* ctx, int64_t n) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + kBlk - 1) / kBlk, (int64_t)ctx->num_sms * 16));
}

__device__ __forceinline__ double min_image(double s, double box) {
    if (box > 0) {
        if (s > 0.5 * box) s -= box;
        else if (s < -0.5 * box) s += box;
    }
    return s;
}

__device__ __forceinline__ float up_float(double h) {  // rounded up to float (tree.cc:288-291)
    const float f = (float)h;
    return (double)f < h ? nextafterf(f, 1e30f) : f;
}

// The pad 1e-6 of the root side is that of the node's own system: root s is node s, and a deeper
// node belongs to the system whose live tree positions hold its first particle.
__global__ void pack_snode_kernel(const GNode* __restrict__ nodes, const int* __restrict__ next,
                                  const double* __restrict__ gc, const double* __restrict__ size, int64_t nn,
                                  const int* __restrict__ sys_off, int n_systems, SNodeG* __restrict__ sn) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += (int64_t)gridDim.x * blockDim.x) {
        const double x = gc[3 * i], y = gc[3 * i + 1], z = gc[3 * i + 2];
        const double cm = fmax(fabs(x), fmax(fabs(y), fabs(z)));
        const int sys = n_systems > 1 ? (i < n_systems ? (int)i : system_of(sys_off, n_systems, nodes[i].plo)) : 0;
        const double eps = 1e-6 * size[sys];
        SNodeG s;
        s.cx = (float)x; s.cy = (float)y; s.cz = (float)z;
        s.half = (float)(0.5 * size[i] + eps + 4.0 * (double)FLT_EPSILON * cm);
        s.first = nodes[i].first;
        s.next = next[i];
        s.plo = nodes[i].plo;
        s.phi = nodes[i].phi;
        sn[i] = s;
    }
}

// Tree::init_hmax: every gas particle i < n_gas with h > 0 raises its leaf and ancestors to h
// rounded up to float; the climb stops at the first ancestor already covering it.  A float max
// through its bit pattern (non-negative), so the result does not depend on the order.
__global__ void hmax_kernel(const double* __restrict__ h, const int* __restrict__ leaf, int64_t n,
                            const int* __restrict__ parent, bool by_particle, float* __restrict__ hmax) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double hi = h[i];
        const int lf = leaf[i];
        if ((by_particle && !(hi > 0)) || lf < 0) continue;
        const unsigned int want = __float_as_uint(up_float(hi));
        for (int no = lf; no >= 0; no = parent[no]) {
            unsigned int* slot = reinterpret_cast<unsigned int*>(hmax + no);
            if (*reinterpret_cast<volatile unsigned int*>(slot) >= want) break;
            atomicMax(slot, want);
        }
    }
}

struct SearchGeom {
    int n_roots;         // roots 0 .. n_roots-1: 1, n_systems in a forest, 0 for a tree without nodes
    int n_systems;
    const int64_t* in_off;  // forest: system s owns the particle indices [in_off[s], in_off[s+1])
    const SNodeG* sn;
    const SrcP* src;
    const uint32_t* order;
    const float* xpad;   // null: 0
    const float* vmax;   // null: 0
    const float* hmax;   // reverse search
    double elapsed, box;
};

// What a gather search tallies under SHMEM_NGB_COUNT (hydro.cc:51-106): nodes visited, particles
// examined in the leaves opened, nodes admitted only by the vmax * elapsed and xpad pads.
struct NgbTally {
    unsigned long long nodes = 0, examined = 0, pad = 0;
};

// The particles [s, e) of one opened leaf against a centre: FP64 |d|^2 as x*x + y*y + z*z without
// contraction (Vec3d::norm_sq).  True when particle s (index j in the input) is a neighbour.
template <bool REVERSE>
__device__ __forceinline__ bool is_neighbour(const SearchGeom& g, int s, double px, double py, double pz,
                                             double r2max, const double* __restrict__ h, int64_t n_gas, uint32_t& j) {
    const double2 xy = __ldg(reinterpret_cast<const double2*>(g.src + s));
    const double zz = __ldg(reinterpret_cast<const double*>(g.src + s) + 2);
    const double ox = min_image(xy.x - px, g.box), oy = min_image(xy.y - py, g.box), oz = min_image(zz - pz, g.box);
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(ox, ox), __dmul_rn(oy, oy)), __dmul_rn(oz, oz));
    if (!REVERSE) return r2 < r2max;
    if (r2 < r2max) return false;
    j = __ldg(g.order + s);
    if ((int64_t)j >= n_gas) return false;
    const double hj = __ldg(h + j);
    return r2 >= r2max && r2 < hj * hj;
}

// One traversal for one centre in the reference's node order, from roots r0 .. r1-1 in turn.
// REVERSE: gas particles j < n_gas with radius <= r < h[j] (ngb_search_reverse); otherwise
// r < radius (ngb_search).  emit(s) receives the tree position; false ends the search.  Every lane of
// mask calls it, each for its own centre.
//
// A thread follows the threading alone, so what bounds the search is how many of a warp's lanes do
// the same thing at once.  Opening each leaf where the traversal meets it kept 5.5 of 32 lanes
// active: the lanes reach their leaves at different steps, and every leaf held up the whole warp.
// Here the traversal only notes the leaves it opens (kLeafBuf of them, in thread-local memory, which
// the hardware interleaves across the warp); then every lane runs through the particles of its own
// leaves in one flat loop, a particle an iteration, and the traversal goes on.  The lanes are brought
// together after each loop: left to themselves they go on from their own last iteration, and two in
// 32 were active by the time the neighbours' sums were formed.
// The prune is the reference's box and circumsphere test in FP32, widened by the rounding of the centre,
// the distances and the squares, so it never drops a node that the FP64 test keeps; the particle test
// decides in FP64, so the lists are the same, in the same order, as long as the nodes' boxes cover their
// particles.  The widening is no more than it must be: at eight times it a cluster of 1e-4 of its box,
// whose lengths are a few hundred roundings of its position, had more nodes visited than by the FP64
// test (reverse search of 100,000 centres: 4.6 ms by the FP64 test, 5.3 at eight times, 3.8 now).
constexpr int kLeafBuf = 32;
template <bool REVERSE, typename F>
__device__ __forceinline__ void search(const SearchGeom& g, int r0, int r1, double px, double py, double pz,
                                       double radius, const double* __restrict__ h, int64_t n_gas, unsigned mask,
                                       F&& emit) {
    const double r2max = radius * radius;
    const float fx = (float)px, fy = (float)py, fz = (float)pz;
    const float fbox = (float)g.box, fhalf = 0.5f * fbox;
    // The rounding of the centre, and twice that of the box side (of itself and of a difference that the
    // minimum image makes small), 2^-24 of each per axis, on three axes 1.74 times that.  Where the squares
    // leave the FP32 range FLT_MIN is above all their roundings.
    const float slack = FLT_EPSILON * (fmaxf(fabsf(fx), fmaxf(fabsf(fy), fabsf(fz))) + 2.0f * fbox);
    const float reach = REVERSE ? slack : __fadd_ru(__double2float_ru(radius), slack);
    const float felapsed = g.elapsed > 0 ? __double2float_ru(g.elapsed) : 0.0f;
    const bool moving = g.elapsed > 0 && g.vmax;
    auto image = [&](float s) {
        if (fbox > 0.0f) {
            if (s > fhalf) s -= fbox;
            else if (s < -fhalf) s += fbox;
        }
        return s;
    };
    int2 leaf[kLeafBuf];
    int root = r0, node = r0 < r1 ? r0 : -1;
    while (__any_sync(mask, node >= 0)) {
        int nl = 0;
        while (node >= 0 && nl < kLeafBuf) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(g.sn + node));
            const int4 b = __ldg(reinterpret_cast<const int4*>(g.sn + node) + 1);
            float dist = reach + a.w;
            bool keep = true;
            if (REVERSE) {
                const float hm = __ldg(g.hmax + node);
                keep = !((double)hm <= radius);
                dist += hm;
            }
            if (g.xpad) dist += __ldg(g.xpad + node);
            if (moving) dist = fmaf(__ldg(g.vmax + node), felapsed, dist);
            dist *= 1.000002f;
            const float dx = image(a.x - fx), dy = image(a.y - fy), dz = image(a.z - fz);
            const float ball = fmaf(0.73205090f, a.w, dist) * 1.000002f;
            keep = keep && !(fmaxf(fabsf(dx), fmaxf(fabsf(dy), fabsf(dz))) > dist) &&
                   !(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > fmaf(ball, ball, FLT_MIN));
            if (keep && b.x < 0) leaf[nl++] = make_int2(b.z, b.w);
            node = keep && b.x >= 0 ? b.x : b.y;
            if (node < 0 && ++root < r1) node = root;  // the next root, where there is one
        }
        __syncwarp(mask);
        int s = 0, e = 0, li = 0;
        for (;;) {
            while (s >= e && li < nl) {
                s = leaf[li].x;
                e = leaf[li].y;
                ++li;
            }
            if (s >= e) break;
            uint32_t j = 0;
            if (is_neighbour<REVERSE>(g, s, px, py, pz, r2max, h, n_gas, j) && !emit(s)) {
                node = -1;  // ended by the caller
                break;
            }
            ++s;
        }
        __syncwarp(mask);
    }
}

// The gather search as the reference counts it (SHMEM_NGB_COUNT): its own FP64 prune, node by node,
// so that the nodes visited and the pads that admitted them are the reference's.  The lists are
// search()'s.
template <typename F>
__device__ __forceinline__ void search_counted(const SearchGeom& g, int r0, int r1, double px, double py, double pz,
                                               double radius, F&& emit, NgbTally* tally) {
    const double r2max = radius * radius;
    for (int root = r0; root < r1; ++root)
    for (int node = root; node >= 0;) {
        ++tally->nodes;
        const float4 a = __ldg(reinterpret_cast<const float4*>(g.sn + node));
        const int4 b = __ldg(reinterpret_cast<const int4*>(g.sn + node) + 1);
        const double half = (double)a.w;
        double dist = radius + half;
        if (g.xpad) dist += (double)__ldg(g.xpad + node);
        if (g.elapsed > 0 && g.vmax) dist += (double)__ldg(g.vmax + node) * g.elapsed;
        const double dx = min_image((double)a.x - px, g.box);
        if (dx > dist || -dx > dist) { node = b.y; continue; }
        const double dy = min_image((double)a.y - py, g.box);
        if (dy > dist || -dy > dist) { node = b.y; continue; }
        const double dz = min_image((double)a.z - pz, g.box);
        if (dz > dist || -dz > dist) { node = b.y; continue; }
        dist += 0.7320508075688772 * half;
        if (dx * dx + dy * dy + dz * dz > dist * dist) { node = b.y; continue; }
        if (g.elapsed > 0) {
            const double nopad = radius + 1.7320508075688772 * half;
            if (dx * dx + dy * dy + dz * dz > nopad * nopad) ++tally->pad;
        }
        if (b.x < 0) {
            tally->examined += (unsigned long long)(b.w - b.z);
            uint32_t j = 0;
            for (int s = b.z; s < b.w; ++s)
                if (is_neighbour<false>(g, s, px, py, pz, r2max, nullptr, 0, j)) emit(s);
            node = b.y;
        } else {
            node = b.x;
        }
    }
}

struct NgbArgs {
    SearchGeom g;
    const double *cx, *cy, *cz, *radius;
    const int* systems;           // per centre, the one system searched; null: every system
    int64_t n;
    int mode;
    const double* h;
    int64_t n_gas;
    uint32_t* count;              // counting pass
    unsigned long long* total;    // counting pass: [0] sum of the counts, [1] centres naming no
                                  // system, [2] centres with more than kcache entries
    const int64_t* start;         // filling pass
    uint32_t* found;
    unsigned long long* tally;    // SHMEM_NGB_COUNT totals (calls, nodes, examined, kept, pad)
    // The counting pass keeps each centre's first kcache entries (entry k of centre c at
    // cache[k * n + c]); the lists of centres with at most kcache entries are then copied from
    // there, and only the others are searched again.  kcache 0: no cache.
    uint32_t* cache;
    int kcache;
};

// Sums v over the warp and adds it to *dst from lane 0; every lane of the warp calls it.
__device__ __forceinline__ void warp_flush(unsigned long long v, unsigned long long* dst) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(dst, v);
}

// The roots a centre searches: every system's, or those of the system it names (checked: a
// system outside [0, n_systems) searches nothing and is counted in *bad).
__device__ __forceinline__ void roots_of(const SearchGeom& g, const int* systems, int64_t c, int& r0, int& r1,
                                         unsigned long long* bad) {
    r0 = 0;
    r1 = g.n_roots;
    if (!systems) return;
    const int s = systems[c];
    if (s < 0 || s >= g.n_systems) {
        if (bad) atomicAdd(bad, 1ull);
        r1 = 0;
        return;
    }
    r0 = s;
    r1 = min(s + 1, g.n_roots);
}

template <bool FILL, bool COUNT>
__global__ void __launch_bounds__(kBlk) ngb_kernel(const NgbArgs a) {
    unsigned long long mine = 0, calls = 0, kept = 0, over = 0;
    NgbTally tl;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t c0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); c0 < a.n; c0 += step) {
        const int64_t c = c0 + (threadIdx.x & 31);
        // lists within the cache's room are copied from there
        const bool have = c < a.n && !(FILL && a.kcache > 0 && a.count[c] <= (uint32_t)a.kcache);
        const unsigned mask = __ballot_sync(0xffffffffu, have);
        if (!have) continue;
        const double px = a.cx[c], py = a.cy[c], pz = a.cz[c], r = a.radius[c];
        int r0, r1;
        roots_of(a.g, a.systems, c, r0, r1, FILL ? nullptr : a.total + 1);
        int64_t k = FILL ? a.start[c] : 0;
        const int64_t end = FILL ? a.start[c + 1] : 0;
        auto emit = [&](int s) {
            if (FILL && k >= end) return false;  // never past the centre's own entries
            if (FILL) a.found[k] = __ldg(a.g.order + s);
            else if (k < a.kcache) a.cache[k * a.n + c] = __ldg(a.g.order + s);
            ++k;
            return true;
        };
        if (a.mode != GT_NGB_REVERSE) {
            if (COUNT) search_counted(a.g, r0, r1, px, py, pz, r, emit, &tl);
            else search<false>(a.g, r0, r1, px, py, pz, r, nullptr, 0, mask, emit);
            if (COUNT) {
                ++calls;
                kept += (unsigned long long)k;
            }
        }
        if (COUNT) __syncwarp(mask);
        if (a.mode != GT_NGB_GATHER) search<true>(a.g, r0, r1, px, py, pz, r, a.h, a.n_gas, mask, emit);
        if (!FILL) {
            a.count[c] = (uint32_t)k;
            mine += (unsigned long long)k;
            over += k > a.kcache ? 1ull : 0ull;
        }
    }
    __syncwarp();
    if (!FILL) {
        warp_flush(mine, a.total);
        warp_flush(over, a.total + 2);
    }
    if (COUNT && !FILL) {
        warp_flush(calls, a.tally + 0);
        warp_flush(tl.nodes, a.tally + 1);
        warp_flush(tl.examined, a.tally + 2);
        warp_flush(kept, a.tally + 3);
        warp_flush(tl.pad, a.tally + 4);
    }
}

// The lists of the centres the counting pass kept whole in the cache, into their CSR slots.
__global__ void ngb_copy_kernel(const uint32_t* __restrict__ cache, int kcache, const uint32_t* __restrict__ cnt,
                                const int64_t* __restrict__ start, int64_t n, uint32_t* __restrict__ found) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t m = cnt[c];
        if (m > (uint32_t)kcache) continue;
        const int64_t s0 = start[c];
        for (uint32_t k = 0; k < m; ++k) found[s0 + k] = cache[(int64_t)k * n + c];
    }
}

__global__ void widen_kernel(const uint32_t* __restrict__ ex, const uint32_t* __restrict__ cnt, int64_t n,
                             int64_t* __restrict__ start) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        start[i] = (int64_t)ex[i];
        if (i == n - 1) start[n] = (int64_t)ex[i] + (int64_t)cnt[i];
    }
}

// ---- the density solve ------------------------------------------------------------------------
// The cubic spline of support h in n_dims dimensions (shmem/hydro.h:25-63).
__device__ __forceinline__ double kernel_norm(double h, int dim) {
    if (dim == 1) return (4.0 / 3.0) / h;
    if (dim == 2) return 40.0 / (7.0 * M_PI * h * h);
    return 8.0 / (M_PI * h * h * h);
}
__device__ __forceinline__ double ball_vol(double h, int dim) {
    if (dim == 1) return 2.0 * h;
    if (dim == 2) return M_PI * h * h;
    return 4.0 * M_PI / 3.0 * h * h * h;
}

struct DensSums {
    double wsum, dwdh, rho, mom[6], face[3];
    int inside;
};

struct DensArgs {
    SearchGeom g;
    const double* smass;
    const uint8_t* stype;  // tree order; null: every particle gas
    const uint32_t* rank;
    const uint32_t* targets;
    int64_t nt;
    double des_ngb, ngb_tol, h_default;
    const double* h_default_sys;  // forest without h_start: the default h of each system
    const double* h_start;
    const double* cond_prev;  // per particle index
    int n_dims, face_corr;
    double *h, *rho;
    int *nngb, *iters;
    unsigned long long* tally;  // SHMEM_NGB_COUNT: calls, nodes, examined, kept, pad, iterations [8]
    // candidate cache: per thread of the grid, cand_cap tree positions, interleaved (entry k of
    // thread i at cand[k * n_threads + i])
    uint32_t* cand;
    int cand_cap;
    int64_t n_threads;
    int run;  // targets a warp takes at a time
    // targets with more candidates than a thread's cache holds, finished by a warp each:
    // heavy_ctr[0] the targets handed over, [1] the next one to take, [2] the next target of density_kernel
    struct DensHeavy* heavy;
    int heavy_cap;
    unsigned int* heavy_ctr;
    uint32_t* warp_cand;  // kWarpCand tree positions per warp
};
// A target's solve at the evaluation that found too many candidates.
struct DensHeavy {
    double h, h_lo, h_hi;
    int t, iter;
};
constexpr int kHeavyCap = 1 << 18;  // 8 MB; a target beyond it is finished by its own thread

__device__ __forceinline__ void dens_zero(DensSums& s) {
    s.wsum = s.dwdh = s.rho = 0.0;
    for (int c = 0; c < 6; ++c) s.mom[c] = 0.0;
    s.face[0] = s.face[1] = s.face[2] = 0.0;
    s.inside = 0;
}

// One gas neighbour's terms at offset (dx, dy, dz) from the target (hydro.cc:209-222): its kernel
// weight w and dW/dh.  Every rounding is spelled out, so that the solve's forms -- a thread per target
// and a warp per target -- add the same terms in the same order and agree to the last bit.
struct DensNorm {
    double h, hinv, norm, dnorm;  // dnorm: -dim / h of the kernel's norm
    bool plain;                   // h is far from the ends of the FP64 range
};
__device__ __forceinline__ DensNorm dens_norm(double h, int dim) {
    const double norm = kernel_norm(h, dim);
    return DensNorm{h, 1.0 / h, norm, __dmul_rn(-((double)dim / h), norm), h > 1e-100 && h < 1e100};
}

// x / h from the rounded reciprocal of h: the quotient's remainder is exact in one fused operation and
// corrects it (Markstein's division), three instructions where a division takes a dozen and a branch.
__device__ __forceinline__ double over_h(double x, const DensNorm& n) {
    if (!n.plain) return x / n.h;
    const double q = __dmul_rn(x, n.hinv);
    return __fma_rn(__fma_rn(-n.h, q, x), n.hinv, q);
}

// The square root of r2 from its reciprocal square root: y by the approximation and one step of the
// binomial series (gt_direct.cu, rsqrt_d), then s = r2 y corrected by the exact remainder r2 - s^2.
__device__ __forceinline__ double root_of(double r2) {
    if (!(r2 > 1e-280 && r2 < 1e280)) return r2 == 0.0 ? 0.0 : sqrt(r2);
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r2));
    const double e = __fma_rn(-r2, __dmul_rn(y, y), 1.0);
    y = __fma_rn(__dmul_rn(y, e), __fma_rn(0.375, e, 0.5), y);
    const double s = __dmul_rn(r2, y);
    return __fma_rn(__fma_rn(-s, s, r2), __dmul_rn(0.5, y), s);
}

__device__ __forceinline__ void dens_terms(double dx, double dy, double dz, const DensNorm& n, double& w, double& dh,
                                           bool& inside) {
    const double r = root_of(__fma_rn(dz, dz, __fma_rn(dx, dx, __dmul_rn(dy, dy))));
    const double q = over_h(r, n);
    // the spline and its derivative on either side of q = 1/2, without a branch
    const double q6 = __dmul_rn(6.0, q), q66 = __dmul_rn(q6, q);
    const double u = __dadd_rn(1.0, -q);
    const bool low = q < 0.5;
    const double f = low ? __fma_rn(q66, q, __dadd_rn(1.0, -q66)) : __dmul_rn(__dmul_rn(__dmul_rn(2.0, u), u), u);
    const double fp = low ? __fma_rn(__dmul_rn(18.0, q), q, __dmul_rn(-12.0, q)) : __dmul_rn(__dmul_rn(-6.0, u), u);
    const bool some = q < 1.0;
    w = some ? __dmul_rn(n.norm, f) : 0.0;
    dh = some ? __fma_rn(-__dmul_rn(over_h(q, n), n.norm), fp, __dmul_rn(n.dnorm, f)) : 0.0;
    inside = r < n.h;
}
__device__ __forceinline__ void dens_sum(double dx, double dy, double dz, double m, double w, double dh, bool inside,
                                         DensSums& s) {
    s.wsum = __dadd_rn(s.wsum, w);
    s.dwdh = __dadd_rn(s.dwdh, dh);
    s.rho = __fma_rn(m, w, s.rho);
    s.mom[0] = __fma_rn(__dmul_rn(dx, dx), w, s.mom[0]);
    s.mom[1] = __fma_rn(__dmul_rn(dy, dy), w, s.mom[1]);
    s.mom[2] = __fma_rn(__dmul_rn(dz, dz), w, s.mom[2]);
    s.mom[3] = __fma_rn(__dmul_rn(dx, dy), w, s.mom[3]);
    s.mom[4] = __fma_rn(__dmul_rn(dy, dz), w, s.mom[4]);
    s.mom[5] = __fma_rn(__dmul_rn(dx, dz), w, s.mom[5]);
    s.face[0] = __fma_rn(dx, w, s.face[0]);
    s.face[1] = __fma_rn(dy, w, s.face[1]);
    s.face[2] = __fma_rn(dz, w, s.face[2]);
    if (inside) ++s.inside;
}
__device__ __forceinline__ void dens_add(double dx, double dy, double dz, double m, const DensNorm& n, DensSums& s) {
    double w, dh;
    bool inside;
    dens_terms(dx, dy, dz, n, w, dh, inside);
    dens_sum(dx, dy, dz, m, w, dh, inside, s);
}

// One evaluation at h: the sums over the GAS neighbours inside h, in tree order (hydro.cc:205-222).
// The neighbours found are buffered and their kernel sums evaluated in runs, in the order found:
// interleaving the FP64 sums with the traversal made the lanes of a warp that were still walking
// wait on every neighbour another lane had found.
constexpr int kDensBuf = 64;
// The candidate cache (below): capacity per thread, and the radius of a refill relative to the h
// that outgrew the cache.
constexpr int kCandCap = 160;
constexpr double kCacheFirst = 1.1;
constexpr double kCacheGrow = 1.4;

template <bool COUNT>
__device__ __noinline__ void dens_eval(const DensArgs& a, int r0, int r1, double px, double py, double pz, double h, DensSums& s,
                          NgbTally& tl, unsigned long long& kept, unsigned mask) {
    dens_zero(s);
    const DensNorm nrm = dens_norm(h, a.n_dims);
    int buf[kDensBuf];
    int nb = 0;
    auto drain = [&]() {
        for (int i = 0; i < nb; ++i) {
            const int sp = buf[i];
            if (a.stype && __ldg(a.stype + sp) != 0) continue;
            const double2 xy = __ldg(reinterpret_cast<const double2*>(a.g.src + sp));
            const double zz = __ldg(reinterpret_cast<const double*>(a.g.src + sp) + 2);
            dens_add(min_image(xy.x - px, a.g.box), min_image(xy.y - py, a.g.box), min_image(zz - pz, a.g.box),
                     __ldg(a.smass + sp), nrm, s);
        }
        nb = 0;
    };
    auto found = [&](int sp) {
        if (COUNT) ++kept;
        if (nb == kDensBuf) drain();
        buf[nb++] = sp;
        return true;
    };
    if (COUNT) search_counted(a.g, r0, r1, px, py, pz, h, found, &tl);
    else search<false>(a.g, r0, r1, px, py, pz, h, nullptr, 0, mask, found);
    drain();
}

// The candidate cache of the Newton iterations.  One search at radius R stores the GAS particles it
// finds (their tree positions, in the search's order) in the thread's slice of a global array; an
// evaluation at any h <= R then scans them and keeps those with r^2 < h^2, with the search's own
// r^2 expression.  That is the set a search at h would keep, in the same order (a larger radius
// only adds particles between them: the order is the threading's), so the sums are bit-identical,
// and an iteration that shrinks h costs a scan of a few dozen candidates instead of a traversal.
// A search that finds more than cand_cap gas particles ends there and returns -1.
__device__ __forceinline__ int cache_fill(const DensArgs& a, int r0, int r1, double px, double py, double pz,
                                          double R, uint32_t* __restrict__ slot, int64_t stride, unsigned mask) {
    int k = 0;
    const int cap = a.cand_cap;
    search<false>(a.g, r0, r1, px, py, pz, R, nullptr, 0, mask, [&](int sp) {
        if (a.stype && __ldg(a.stype + sp) != 0) return true;
        if (k < cap) slot[(int64_t)k * stride] = (uint32_t)sp;
        return ++k <= cap;
    });
    return k <= cap ? k : -1;
}

// Two candidates at a time, the next two's positions on their way: what bounds the evaluation is the
// latency of its loads and of the FP64 chains to the weights, which two independent candidates
// overlap.  The sums take the kept ones in order.
__device__ __forceinline__ void cache_eval(const DensArgs& a, const uint32_t* __restrict__ slot, int64_t stride, int n,
                                           double px, double py, double pz, double h, DensSums& s) {
    dens_zero(s);
    const DensNorm nrm = dens_norm(h, a.n_dims);
    const double r2max = h * h;
    auto at = [&](int k) { return (int)slot[(int64_t)min(k, n - 1) * stride]; };
    auto load = [&](int sp, double& x, double& y, double& z) {
        const double2 xy = __ldg(reinterpret_cast<const double2*>(a.g.src + sp));
        x = xy.x; y = xy.y;
        z = __ldg(reinterpret_cast<const double*>(a.g.src + sp) + 2);
    };
    if (n <= 0) return;
    int s0 = at(0), s1 = at(1), s2 = at(2), s3 = at(3);
    double x0, y0, z0, x1, y1, z1;
    load(s0, x0, y0, z0);
    load(s1, x1, y1, z1);
    for (int k = 0; k < n; k += 2) {
        const double m0 = __ldg(a.smass + s0), m1 = __ldg(a.smass + s1);
        const double dx0 = min_image(x0 - px, a.g.box), dy0 = min_image(y0 - py, a.g.box), dz0 = min_image(z0 - pz, a.g.box);
        const double dx1 = min_image(x1 - px, a.g.box), dy1 = min_image(y1 - py, a.g.box), dz1 = min_image(z1 - pz, a.g.box);
        s0 = s2; s1 = s3;
        s2 = at(k + 4); s3 = at(k + 5);
        load(s0, x0, y0, z0);
        load(s1, x1, y1, z1);
        const double r0 = __dadd_rn(__dadd_rn(__dmul_rn(dx0, dx0), __dmul_rn(dy0, dy0)), __dmul_rn(dz0, dz0));
        const double r1 = __dadd_rn(__dadd_rn(__dmul_rn(dx1, dx1), __dmul_rn(dy1, dy1)), __dmul_rn(dz1, dz1));
        const bool keep0 = r0 < r2max, keep1 = k + 1 < n && r1 < r2max;
        if (keep0 || keep1) {
            double w0, e0, w1, e1;
            bool in0, in1;
            dens_terms(dx0, dy0, dz0, nrm, w0, e0, in0);
            dens_terms(dx1, dy1, dz1, nrm, w1, e1, in1);
            if (keep0) dens_sum(dx0, dy0, dz0, m0, w0, e0, in0, s);
            if (keep1) dens_sum(dx1, dy1, dz1, m1, w1, e1, in1, s);
        }
    }
}

// Rank-d inverse of the symmetric moments (xx yy zz xy yz xz), row-major, zero when degenerate
// (shmem/vec.h:43-66; 3-D: cofactors over the determinant).
__device__ bool invert_moments(const double* m, double* B, int n_dims) {
    for (int i = 0; i < 9; ++i) B[i] = 0.0;
    if (n_dims == 1) {
        if (fabs(m[0]) < 1e-300) return false;
        B[0] = 1.0 / m[0];
        return true;
    }
    if (n_dims == 2) {
        const double det = m[0] * m[1] - m[3] * m[3];
        if (fabs(det) < 1e-300) return false;
        B[0] = m[1] / det; B[1] = -m[3] / det;
        B[3] = -m[3] / det; B[4] = m[0] / det;
        return true;
    }
    const double a00 = m[0], a01 = m[3], a02 = m[5], a11 = m[1], a12 = m[4], a22 = m[2];
    const double a10 = a01, a20 = a02, a21 = a12;
    const double d = a00 * (a11 * a22 - a12 * a21) - a01 * (a10 * a22 - a12 * a20) + a02 * (a10 * a21 - a11 * a20);
    if (d == 0.0 || d != d) return false;
    const double id = 1.0 / d;
    B[0] = (a11 * a22 - a12 * a21) * id; B[1] = (a02 * a21 - a01 * a22) * id; B[2] = (a01 * a12 - a02 * a11) * id;
    B[3] = (a12 * a20 - a10 * a22) * id; B[4] = (a00 * a22 - a02 * a20) * id; B[5] = (a02 * a10 - a00 * a12) * id;
    B[6] = (a10 * a21 - a11 * a20) * id; B[7] = (a01 * a20 - a00 * a21) * id; B[8] = (a00 * a11 - a01 * a10) * id;
    return true;
}

// The convergence test and the bisection-guarded Newton step of one iteration with the
// face-closure and condition-number corrections and the growing tolerance (hydro.cc:224-272) for
// particle p after an evaluation at h: true when converged (h kept), else h moves.
struct NewtonParams {
    double des_ngb, ngb_tol;
    const double* cond_prev;
    int n_dims, face_corr;
};

// Not inlined: one compiled copy, so that every form of the solve takes the same steps to the last bit.
__device__ __noinline__ bool dens_newton(const NewtonParams a, uint32_t p, const DensSums& s, int iter, double& h,
                                         double& h_lo, double& h_hi) {
    const int dim = a.n_dims;
    const double n_eff = ball_vol(h, dim) * s.wsum;
    double ncorr = 1.0;
    if (a.cond_prev) {
        const double cn = a.cond_prev[p];
        if (cn > 100.0) ncorr = fmin(sqrt(1.0 + (cn - 100.0) / 1000.0), 2.0);
    }
    double des_eff = a.des_ngb * ncorr, tol_eff = a.ngb_tol * ncorr;
    if (a.face_corr && s.wsum > 0) {
        double B[9];
        if (invert_moments(s.mom, B, dim)) {
            const double vol = 1.0 / s.wsum;
            const double dx_i = sqrt(vol * (s.mom[0] + s.mom[1] + s.mom[2]));
            double sum_abs = 0.0;
            for (int r = 0; r < 3; ++r) {
                const double leak =
                    (B[3 * r] * s.face[0] + B[3 * r + 1] * s.face[1] + B[3 * r + 2] * s.face[2]) * (2.0 * vol);
                sum_abs += fabs(leak) / dim;
            }
            const double denom = 2.0 * dim * pow(dx_i, dim - 1);
            if (denom > 0) {
                const double fce = sum_abs / denom;
                if (fce > 0.35) ncorr = fmax(ncorr, fmin(fce / 0.35, 2.0));
                des_eff = a.des_ngb * ncorr;
                tol_eff = a.ngb_tol * ncorr;
            }
        }
    }
    if (iter > 1) tol_eff = fmin(0.25 * des_eff, tol_eff * exp(0.1 * log(des_eff / (16.0 * tol_eff)) * iter));
    const double res = n_eff - des_eff;
    if (fabs(res) < tol_eff) return true;
    if (res > 0) h_hi = h; else h_lo = h;
    const double dn = ball_vol(h, dim) * ((double)dim / h * s.wsum + s.dwdh);
    double hn = dn > 0 ? h - res / dn : 0.0;
    if (hn <= h_lo || (h_hi > 0 && hn >= h_hi) || hn <= 0) {
        if (h_hi > 0) hn = h_lo > 0 ? sqrt(h_lo * h_hi) : 0.5 * h_hi;
        else hn = h * (res > 0 ? 0.7 : 1.6);
    }
    h = hn;
    return false;
}

__device__ __forceinline__ NewtonParams newton_params(const DensArgs& a) {
    return NewtonParams{a.des_ngb, a.ngb_tol, a.cond_prev, a.n_dims, a.face_corr};
}

// The counting solve, one thread per target: up to 100 iterations of evaluation and Newton step, then,
// when the solve did not converge, one more evaluation at the final h (hydro.cc:189-297).  Every
// evaluation is one gather search of the tally, and the target's iterations go to the histogram
// (hydro.cc:293-296).  In a forest the target searches the system that owns its particle index.
__global__ void __launch_bounds__(kBlk, 6) density_count_kernel(const DensArgs a) {
    NgbTally tl;
    unsigned long long calls = 0, kept = 0, hist[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < a.nt; t += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t p = a.targets[t];
        const uint32_t sp = a.rank[p];
        const double px = a.g.src[sp].x, py = a.g.src[sp].y, pz = a.g.src[sp].z;
        int r0 = 0, r1 = a.g.n_roots;
        if (a.g.in_off) {
            r0 = system_of(a.g.in_off, a.g.n_systems, (int64_t)p);
            r1 = r0 + 1;
        }
        double h = a.h_start ? a.h_start[t] : (a.h_default_sys ? a.h_default_sys[r0] : a.h_default);
        double h_lo = 0.0, h_hi = 0.0;
        int iter = 0;
        bool converged = false;
        DensSums s;
        for (; iter < 100; ++iter) {
            dens_eval<true>(a, r0, r1, px, py, pz, h, s, tl, kept, 0u);
            ++calls;
            if (dens_newton(newton_params(a), p, s, iter, h, h_lo, h_hi)) { converged = true; break; }
        }
        if (!converged) {  // rho of the final h (hydro.cc:281-293)
            dens_eval<true>(a, r0, r1, px, py, pz, h, s, tl, kept, 0u);
            ++calls;
        }
        ++hist[min(converged ? iter + 1 : 100, 8) - 1];
        a.h[t] = h;
        a.rho[t] = s.rho;
        a.nngb[t] = s.inside;
        a.iters[t] = iter;
    }
    warp_flush(calls, a.tally + 0);
    warp_flush(tl.nodes, a.tally + 1);
    warp_flush(tl.examined, a.tally + 2);
    warp_flush(kept, a.tally + 3);
    warp_flush(tl.pad, a.tally + 4);
    for (int k = 0; k < 8; ++k) warp_flush(hist[k], a.tally + 5 + k);
}

// The solve: a lane per target, refilled as targets finish.
//
// The targets of a warp take between 1 and 10 iterations, three on average, so with a target per
// thread for good most lanes waited for the slowest.  Here a warp takes a run of consecutive targets
// at a time and its lanes are a pool: a lane whose target is done takes the next one.  The loop's two
// phases each run for as many lanes at once as can be gathered: the search that fills a lane's
// candidate cache (a new target, or an h that outgrew the cache) waits until kGather lanes are idle or
// want it, or nobody can do anything else, and an evaluation with its Newton step runs for every lane
// that holds candidates.  Each target's own sequence of searches, sums and steps is that of the
// counting solve's thread, so its results are the same bits whichever lane it gets.  Warm solve of a
// 2^20 galaxy, lengths 5 % off: 26.0 ms before leaves were collected (search) and crowded targets
// went to warps, 14.2 then, 13.2 with the square root and quotients of dens_terms, 12.2 with two
// candidates at a time and the four blocks per SM whose registers that needs (six spill: 13.5).
// ONE_ROOT: a single-system tree, whose one root (node 0) the compiler then knows.
constexpr int kGather = 16;
template <bool ONE_ROOT>
__global__ void __launch_bounds__(kBlk, 4) density_kernel(const DensArgs a) {
    const int lane = threadIdx.x & 31;
    uint32_t* __restrict__ slot = a.cand + ((int64_t)blockIdx.x * blockDim.x + threadIdx.x);
    unsigned next = 0, end = 0;  // the warp's run of targets still to take
    bool more = true;            // targets are left beyond it
    int t = -1, iter = 0, ncand = 0, r0 = 0, r1 = 1;
    bool direct = false;         // too many candidates and no room to hand over: search at every evaluation
    bool ready_now = false;      // searched for this h (also where h is not a number), or direct
    double px = 0, py = 0, pz = 0, h = 0, h_lo = 0, h_hi = 0, R = -1.0;
    for (;;) {
        // idle lanes take targets
        const unsigned idle = __ballot_sync(0xffffffffu, t < 0);
        const unsigned out = __ballot_sync(0xffffffffu, t < 0 || (!ready_now && !(R >= h)));  // idle or to search
        if (idle != 0u && __popc(out) >= kGather && (more || next < end)) {
            if (next >= end) {
                if (lane == 0) next = atomicAdd(a.heavy_ctr + 2, (unsigned)a.run);
                next = __shfl_sync(0xffffffffu, next, 0);
                end = (unsigned)min((int64_t)next + a.run, a.nt);
                more = (int64_t)next + a.run < a.nt;
            }
            const unsigned mine = next + __popc(idle & ((1u << lane) - 1u));
            if (t < 0 && mine < end) {
                t = (int)mine;
                const uint32_t p = a.targets[t];
                const uint32_t sp = a.rank[p];
                px = a.g.src[sp].x; py = a.g.src[sp].y; pz = a.g.src[sp].z;
                if (!ONE_ROOT) {
                    r1 = a.g.n_roots;
                    if (a.g.in_off) {
                        r0 = system_of(a.g.in_off, a.g.n_systems, (int64_t)p);
                        r1 = r0 + 1;
                    }
                }
                h = a.h_start ? a.h_start[t] : (a.h_default_sys ? a.h_default_sys[r0] : a.h_default);
                h_lo = h_hi = 0.0;
                R = -1.0;
                iter = 0;
                direct = ready_now = false;
            }
            next = min(end, next + (unsigned)__popc(idle));
            continue;
        }
        const bool have = t >= 0, want = have && !ready_now && !(R >= h);
        const unsigned wants = __ballot_sync(0xffffffffu, want), ready = __ballot_sync(0xffffffffu, have && !want);
        if ((wants | ready) == 0u) break;
        if (__popc(wants) >= kGather || ready == 0u) {
            if (want) {
                const double rad = (R < 0 ? kCacheFirst : kCacheGrow) * h;
                ncand = cache_fill(a, r0, r1, px, py, pz, rad, slot, a.n_threads, wants);
                R = rad;
                ready_now = true;
                if (ncand < 0) {
                    // more candidates than the cache holds: to a warp of density_heavy_kernel
                    const unsigned at = atomicAdd(a.heavy_ctr, 1u);
                    if (at < (unsigned)a.heavy_cap) {
                        a.heavy[at] = DensHeavy{h, h_lo, h_hi, t, iter};
                        t = -1;
                    } else {
                        direct = true;
                    }
                }
            }
            __syncwarp();
            continue;
        }
        if (have && !want) {
            DensSums s;
            // (no lane searches directly unless the hand-over list is full)
            const unsigned straight = __ballot_sync(ready, direct);
            if (direct) {
                NgbTally none;
                unsigned long long kept = 0;
                dens_eval<false>(a, r0, r1, px, py, pz, h, s, none, kept, straight);
            } else {
                cache_eval(a, slot, a.n_threads, ncand, px, py, pz, h, s);
            }
            __syncwarp(ready);
            // after 100 steps, the sums of the final h (hydro.cc:281-293)
            if (iter == 100 || dens_newton(newton_params(a), a.targets[t], s, iter, h, h_lo, h_hi)) {
                a.h[t] = h;
                a.rho[t] = s.rho;
                a.nngb[t] = s.inside;
                a.iters[t] = iter;
                t = -1;
            } else {
                ++iter;
                ready_now = direct;
            }
        }
        __syncwarp();
    }
}

// The targets that a thread handed over, a warp each.  A Newton step from a poor guess can ask for an
// h that holds tens of thousands of neighbours; in one thread such an evaluation took 28 ms, the time
// of the whole solve of 86,000 targets.  Here the lanes test 32 consecutive particles at a time and
// compute their terms, and twelve lanes, one per sum, add the 32 terms in order from shared memory:
// the sums are those of the thread's loop to the last bit.  The traversal is the thread's, in all
// lanes alike, and stops at nodes of up to kWarpLeaf particles, whose consecutive range is tested
// whole: the particle test alone decides, so the neighbours and their order are the same where the
// boxes cover their particles.
constexpr int kHeavyWarps = 4;
constexpr int kWarpLeaf = 64;
constexpr int kWarpCand = 2048;  // cached candidates per warp; a larger search is repeated instead

// The particles within `radius` in tree order, 32 at a time: use(s, keep) in every lane.
template <typename F>
__device__ __forceinline__ void warp_search(const SearchGeom& g, int r0, int r1, double px, double py, double pz,
                                            double radius, F&& use) {
    const int lane = threadIdx.x & 31;
    const double r2max = radius * radius;
    for (int root = r0; root < r1; ++root)
        for (int node = root; node >= 0;) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(g.sn + node));
            const int4 b = __ldg(reinterpret_cast<const int4*>(g.sn + node) + 1);
            double dist = radius + (double)a.w;
            if (g.xpad) dist += (double)__ldg(g.xpad + node);
            if (g.elapsed > 0 && g.vmax) dist += (double)__ldg(g.vmax + node) * g.elapsed;
            const double dx = min_image((double)a.x - px, g.box), dy = min_image((double)a.y - py, g.box),
                         dz = min_image((double)a.z - pz, g.box);
            const double ball = dist + 0.7320508075688772 * (double)a.w;
            if (fabs(dx) > dist || fabs(dy) > dist || fabs(dz) > dist || dx * dx + dy * dy + dz * dz > ball * ball) {
                node = b.y;
            } else if (b.x < 0 || b.w - b.z <= kWarpLeaf) {
                for (int s0 = b.z; s0 < b.w; s0 += 32) {
                    const int s = s0 + lane;
                    uint32_t j = 0;
                    const bool keep = s < b.w && is_neighbour<false>(g, s, px, py, pz, r2max, nullptr, 0, j);
                    use(s, keep);
                }
                node = b.y;
            } else {
                node = b.x;
            }
        }
}

__global__ void __launch_bounds__(kHeavyWarps * 32) density_heavy_kernel(const DensArgs a) {
    // terms of 32 particles: the factors of each sum's fused multiply-add
    __shared__ double term[kHeavyWarps][12][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double(*T)[32] = term[w];
    uint32_t* __restrict__ list = a.warp_cand + (int64_t)(blockIdx.x * kHeavyWarps + w) * kWarpCand;
    const unsigned n_heavy = min(a.heavy_ctr[0], (unsigned)a.heavy_cap);
    // lane c < 12 keeps sum c = sum of T[fa] * T[fb] (wsum and dwdh: of T[fb])
    const int fb = lane == 1 ? 1 : 0, fa = lane == 2 ? 2 : lane < 9 ? lane + 3 : lane - 6;
    for (;;) {
        unsigned i = 0;
        if (lane == 0) i = atomicAdd(a.heavy_ctr + 1, 1u);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= n_heavy) break;
        const DensHeavy st = a.heavy[i];
        const uint32_t p = a.targets[st.t];
        const uint32_t pos = a.rank[p];
        const double px = a.g.src[pos].x, py = a.g.src[pos].y, pz = a.g.src[pos].z;
        int r0 = 0, r1 = a.g.n_roots;
        if (a.g.in_off) {
            r0 = system_of(a.g.in_off, a.g.n_systems, (int64_t)p);
            r1 = r0 + 1;
        }
        double h = st.h, h_lo = st.h_lo, h_hi = st.h_hi;
        int iter = st.iter;
        bool converged = false;
        double R = -1.0;  // radius of the cached search; < 0: nothing cached
        int ncand = 0;
        DensSums s;
        auto evaluate = [&](double hh) {
            const DensNorm nrm = dens_norm(hh, a.n_dims);
            double acc = 0.0;
            int inside = 0;
            const double r2max = hh * hh;
            // 32 particles of the search at hh, in order
            auto add = [&](int sp, bool keep) {
                double q[12];
                for (int c = 0; c < 12; ++c) q[c] = 0.0;
                bool in = false;
                if (keep) {
                    const double2 xy = __ldg(reinterpret_cast<const double2*>(a.g.src + sp));
                    const double zz = __ldg(reinterpret_cast<const double*>(a.g.src + sp) + 2);
                    const double dx = min_image(xy.x - px, a.g.box), dy = min_image(xy.y - py, a.g.box),
                                 dz = min_image(zz - pz, a.g.box);
                    dens_terms(dx, dy, dz, nrm, q[0], q[1], in);
                    q[2] = __ldg(a.smass + sp);
                    q[3] = dx; q[4] = dy; q[5] = dz;
                    q[6] = __dmul_rn(dx, dx); q[7] = __dmul_rn(dy, dy); q[8] = __dmul_rn(dz, dz);
                    q[9] = __dmul_rn(dx, dy); q[10] = __dmul_rn(dy, dz); q[11] = __dmul_rn(dx, dz);
                }
                inside += __popc(__ballot_sync(0xffffffffu, in));
#pragma unroll
                for (int c = 0; c < 12; ++c) T[c][lane] = q[c];
                __syncwarp();
                if (lane < 12) {
#pragma unroll 8
                    for (int k = 0; k < 32; ++k)
                        acc = lane < 2 ? __dadd_rn(acc, T[fb][k]) : __fma_rn(T[fa][k], T[fb][k], acc);
                }
                __syncwarp();
            };
            if (!(R >= hh)) {
                const double rad = (R < 0 ? kCacheFirst : kCacheGrow) * hh;
                int k = 0;
                warp_search(a.g, r0, r1, px, py, pz, rad, [&](int sp, bool keep) {
                    keep = keep && !(a.stype && __ldg(a.stype + sp) != 0);
                    const unsigned m = __ballot_sync(0xffffffffu, keep);
                    const int at = k + __popc(m & ((1u << lane) - 1u));
                    if (keep && at < kWarpCand) list[at] = (uint32_t)sp;
                    k += __popc(m);
                });
                __syncwarp();
                ncand = k;
                R = k <= kWarpCand ? rad : -1.0;
            }
            if (R >= hh) {
                for (int k0 = 0; k0 < ncand; k0 += 32) {
                    const bool have = k0 + lane < ncand;
                    const int sp = have ? (int)list[k0 + lane] : 0;
                    uint32_t j = 0;
                    add(sp, have && is_neighbour<false>(a.g, sp, px, py, pz, r2max, nullptr, 0, j));
                }
            } else {
                warp_search(a.g, r0, r1, px, py, pz, hh, [&](int sp, bool keep) {
                    keep = keep && !(a.stype && __ldg(a.stype + sp) != 0);
                    if (__any_sync(0xffffffffu, keep)) add(sp, keep);
                });
            }
            auto get = [&](int c) { return __shfl_sync(0xffffffffu, acc, c); };
            s.wsum = get(0); s.dwdh = get(1); s.rho = get(2);
            for (int c = 0; c < 6; ++c) s.mom[c] = get(3 + c);
            for (int c = 0; c < 3; ++c) s.face[c] = get(9 + c);
            s.inside = inside;
        };
        for (; iter < 100; ++iter) {
            evaluate(h);
            if (dens_newton(newton_params(a), p, s, iter, h, h_lo, h_hi)) { converged = true; break; }
        }
        if (!converged) evaluate(h);
        if (lane == 0) {
            a.h[st.t] = h;
            a.rho[st.t] = s.rho;
            a.nngb[st.t] = s.inside;
            a.iters[st.t] = iter;
        }
    }
}

// Per system of a forest, the bounding box of all its particles (massless too) for its default h:
// block b reduces chunk b % chunks of system b / chunks, through the particles' tree positions.
__global__ void density_bbox_kernel(const SrcP* __restrict__ src, const uint32_t* __restrict__ rank,
                                    const int64_t* __restrict__ in_off, int chunks, double* __restrict__ part) {
    const int s = blockIdx.x / chunks, c = blockIdx.x % chunks;
    const int64_t lo0 = in_off[s], len = in_off[s + 1] - lo0;
    const int64_t b = lo0 + len * c / chunks, e = lo0 + len * (c + 1) / chunks;
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int64_t i = b + threadIdx.x; i < e; i += blockDim.x) {
        const SrcP q = src[rank[i]];
        const double v[3] = {q.x, q.y, q.z};
        for (int k = 0; k < 3; ++k) { lo[k] = fmin(lo[k], v[k]); hi[k] = fmax(hi[k], v[k]); }
    }
    __shared__ double sh[6][kBlk];
    for (int k = 0; k < 3; ++k) { sh[k][threadIdx.x] = lo[k]; sh[3 + k][threadIdx.x] = hi[k]; }
    __syncthreads();
    for (int o = kBlk / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o)
            for (int k = 0; k < 3; ++k) {
                sh[k][threadIdx.x] = fmin(sh[k][threadIdx.x], sh[k][threadIdx.x + o]);
                sh[3 + k][threadIdx.x] = fmax(sh[3 + k][threadIdx.x], sh[3 + k][threadIdx.x + o]);
            }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int k = 0; k < 6; ++k) part[6 * (int64_t)blockIdx.x + k] = sh[k][0];
}

// bounding box of every particle (massless too), for the density solve's default h
__global__ void bbox_all_kernel(const SrcP* __restrict__ src, int64_t n, double* __restrict__ part) {
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double v[3] = {src[i].x, src[i].y, src[i].z};
        for (int k = 0; k < 3; ++k) { lo[k] = fmin(lo[k], v[k]); hi[k] = fmax(hi[k], v[k]); }
    }
    __shared__ double sh[6][kBlk];
    for (int k = 0; k < 3; ++k) { sh[k][threadIdx.x] = lo[k]; sh[3 + k][threadIdx.x] = hi[k]; }
    __syncthreads();
    for (int o = kBlk / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o)
            for (int k = 0; k < 3; ++k) {
                sh[k][threadIdx.x] = fmin(sh[k][threadIdx.x], sh[k][threadIdx.x + o]);
                sh[3 + k][threadIdx.x] = fmax(sh[3 + k][threadIdx.x], sh[3 + k][threadIdx.x + o]);
            }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int k = 0; k < 6; ++k) part[6 * blockIdx.x + k] = sh[k][0];
}

SearchGeom geom_of(gt_context* ctx, gt_tree* t, double elapsed, double box) {
    ensure_snodes(ctx, t);
    SearchGeom g;
    g.n_roots = t->n_nodes > 0 ? t->n_systems : 0;
    g.n_systems = t->n_systems;
    g.in_off = t->n_systems > 1 ? t->in_off_dev : nullptr;
    g.sn = t->snode;
    g.src = t->src;
    g.order = t->order;
    g.xpad = t->xpad;
    g.vmax = t->vmax;
    g.hmax = t->hmax;
    g.elapsed = elapsed;
    g.box = box;
    return g;
}

}  // namespace

// Made once per tree, under the tree's lock: contexts on other threads and streams may search the
// same tree, so the nodes are complete on the device before the pointer is published.
void ensure_snodes(gt_context* ctx, gt_tree* t) {
    if (t->n_nodes <= 0) return;
    std::lock_guard<std::mutex> lk(t->lazy_mu);
    if (t->snode) return;
    SNodeG* p = nullptr;
    check_cuda(cudaMallocAsync((void**)&p, (size_t)t->n_nodes * sizeof(SNodeG), ctx->stream), "cudaMallocAsync");
    pack_snode_kernel<<<grid_of(ctx, t->n_nodes), kBlk, 0, ctx->stream>>>(t->nodes, t->next, t->gc, t->size,
                                                                          t->n_nodes, t->sys_off_dev, t->n_systems, p);
    check_launch(ctx, "pack_snode_kernel");
    check_cuda(cudaStreamSynchronize(ctx->stream), "sync");
    t->snode = p;
}

namespace {
// The context's device tally, zeroed for one call (allocated on first use).
unsigned long long* fresh_tally(gt_context* ctx) {
    if (!ctx->tally_dev) {
        unsigned long long* p = nullptr;
        check_cuda(cudaMalloc((void**)&p, GT_NGB_COUNTERS * sizeof(unsigned long long)), "cudaMalloc");
        ctx->tally_dev = p;
    }
    check_cuda(cudaMemsetAsync(ctx->tally_dev, 0, GT_NGB_COUNTERS * sizeof(unsigned long long), ctx->stream),
               "memset");
    return ctx->tally_dev;
}
}  // namespace

void tree_hmax(gt_context* ctx, gt_tree* t, const double* h, int64_t n_gas) {
    const int64_t nn = std::max<int64_t>(t->n_nodes, 1);
    if (!t->hmax) check_cuda(cudaMallocAsync((void**)&t->hmax, (size_t)nn * 4, ctx->stream), "cudaMallocAsync");
    check_cuda(cudaMemsetAsync(t->hmax, 0, (size_t)nn * 4, ctx->stream), "memset");
    const int64_t n = std::min<int64_t>(n_gas, t->n);
    if (n > 0) {
        hmax_kernel<<<grid_of(ctx, n), kBlk, 0, ctx->stream>>>(h, t->leaf_of, n, t->parent, true, t->hmax);
        check_launch(ctx, "hmax_kernel");
    }
}

void raise_hmax(gt_context* ctx, gt_tree* t, int64_t n, const int* leaf, const double* h) {
    if (!t->hmax || n <= 0) return;  // Tree::raise_hmax is a no-op before init_hmax
    hmax_kernel<<<grid_of(ctx, n), kBlk, 0, ctx->stream>>>(h, leaf, n, t->parent, false, t->hmax);
    check_launch(ctx, "hmax_kernel");
}

int64_t run_ngb(gt_context* ctx, gt_tree* t, int64_t n, const double* cx, const double* cy, const double* cz,
                const double* radius, const int* systems, int mode, const double* h, int64_t n_gas, double box,
                double elapsed, int64_t* start, uint32_t* found, int64_t capacity, int64_t* tally,
                uint32_t** list_out) {
    if (mode != GT_NGB_GATHER && !t->hmax) throw Fail{GT_ERR_INVALID, "the reverse search needs gt_tree_hmax first"};
    cudaStream_t st = ctx->stream;
    NgbArgs a;
    a.g = geom_of(ctx, t, elapsed, box);
    a.cx = cx; a.cy = cy; a.cz = cz; a.radius = radius;
    a.systems = systems;
    a.tally = tally ? fresh_tally(ctx) : nullptr;
    a.n = n;
    a.mode = mode;
    a.h = h;
    a.n_gas = n_gas;
    uint32_t* cnt = (uint32_t*)scratch(ctx, kSlotNgb0, (size_t)std::max<int64_t>(n, 1) * 4);
    uint32_t* ex = (uint32_t*)scratch(ctx, kSlotNgb1, (size_t)std::max<int64_t>(n, 1) * 4);
    unsigned long long* tot = (unsigned long long*)scratch(ctx, kSlotNgb2, 24);
    check_cuda(cudaMemsetAsync(tot, 0, 24, st), "memset");
    a.count = cnt;
    a.total = tot;
    a.start = nullptr;
    a.found = nullptr;
    // the first entries of every centre, kept by the counting pass when the lists are wanted: up
    // to 64 per centre within 2 GiB (none below 8)
    const bool want = (found && capacity > 0) || list_out;
    a.kcache = want ? (int)std::min<int64_t>(64, ((int64_t)1 << 31) / (4 * std::max<int64_t>(n, 1))) : 0;
    if (a.kcache < 8) a.kcache = 0;
    a.cache = a.kcache ? (uint32_t*)scratch(ctx, kSlotNgb3, (size_t)n * a.kcache * 4) : nullptr;
    if (a.tally) ngb_kernel<false, true><<<grid_of(ctx, n), kBlk, 0, st>>>(a);
    else ngb_kernel<false, false><<<grid_of(ctx, n), kBlk, 0, st>>>(a);
    check_launch(ctx, "ngb_kernel");
    unsigned long long total[3] = {0, 0, 0};
    check_cuda(cudaMemcpyAsync(ctx->pinned, tot, 24, cudaMemcpyDeviceToHost, st), "d2h");
    if (a.tally)
        check_cuda(cudaMemcpyAsync((char*)ctx->pinned + 64, a.tally, 5 * 8, cudaMemcpyDeviceToHost, st), "d2h");
    check_cuda(cudaStreamSynchronize(st), "sync");
    std::memcpy(total, ctx->pinned, 24);
    if (a.tally) std::memcpy(tally, (char*)ctx->pinned + 64, 5 * 8);
    if (total[1] > 0) throw Fail{GT_ERR_INVALID, "a centre names a system outside [0, n_systems)"};
    if (total[0] >= (1ull << 32)) throw Fail{GT_ERR_OVERFLOW, "more than 2^32 neighbours in one call"};
    scan_exclusive_u32(ctx, cnt, ex, n, nullptr);
    widen_kernel<<<grid_of(ctx, n), kBlk, 0, st>>>(ex, cnt, n, start);
    check_launch(ctx, "widen_kernel");
    uint32_t* dst = nullptr;
    if ((int64_t)total[0] <= capacity && total[0] > 0) {
        if (found) dst = found;
        else if (list_out) dst = (uint32_t*)scratch(ctx, kSlotOut1, (size_t)total[0] * 4);
    }
    if (dst) {
        if (a.kcache) {
            ngb_copy_kernel<<<grid_of(ctx, n), kBlk, 0, st>>>(a.cache, a.kcache, cnt, start, n, dst);
            check_launch(ctx, "ngb_copy_kernel");
        }
        if (!a.kcache || total[2] > 0) {  // the centres the cache did not hold whole
            a.start = start;
            a.found = dst;
            // by the traversal that counted them: on a tree whose boxes do not cover its moved
            // particles the two prunes need not find the same
            if (a.tally) ngb_kernel<true, true><<<grid_of(ctx, n), kBlk, 0, st>>>(a);
            else ngb_kernel<true, false><<<grid_of(ctx, n), kBlk, 0, st>>>(a);
            check_launch(ctx, "ngb_kernel");
        }
    }
    if (list_out) *list_out = dst;
    return (int64_t)total[0];
}

// The default h of a particle set: des_ngb particles at the mean number density of its bounding
// box (lo, hi) over n particles (hydro.cc:169-183).
double default_h(const double* lo, const double* hi, double n, double des_ngb, int n_dims) {
    const double vol = (hi[0] - lo[0]) * (hi[1] - lo[1]) * (hi[2] - lo[2]);
    double hd = std::cbrt(3.0 * des_ngb * vol / (4.0 * M_PI * n));
    if (n_dims == 1) hd = 0.5 * des_ngb * (hi[0] - lo[0]) / n;
    if (n_dims == 2) hd = std::sqrt(des_ngb * (hi[0] - lo[0]) * (hi[1] - lo[1]) / (M_PI * n));
    return hd;
}

void run_density(gt_context* ctx, gt_tree* t, int64_t nt, const uint32_t* targets, double des_ngb, double ngb_tol,
                 const double* h_start, double box, int n_dims, const double* cond_prev, int face_corr,
                 double elapsed, double* h, double* rho, int* nngb, int* iters, int64_t* tally) {
    cudaStream_t st = ctx->stream;
    DensArgs a;
    a.g = geom_of(ctx, t, elapsed, box);
    a.smass = t->smass;
    a.stype = t->stype;
    a.rank = t->rank;
    a.targets = targets;
    a.nt = nt;
    a.des_ngb = des_ngb;
    a.ngb_tol = ngb_tol;
    a.h_start = h_start;
    a.cond_prev = cond_prev;
    a.n_dims = n_dims;
    a.face_corr = face_corr;
    a.h = h; a.rho = rho; a.nngb = nngb; a.iters = iters;
    a.tally = tally && nt > 0 ? fresh_tally(ctx) : nullptr;
    a.cand = nullptr;
    a.heavy = nullptr;
    a.heavy_ctr = nullptr;
    a.warp_cand = nullptr;
    a.heavy_cap = 0;
    a.run = 32;
    const int solve_blocks = (int)std::min<int64_t>((nt + kBlk - 1) / kBlk, (int64_t)ctx->num_sms * 4);
    const int heavy_blocks = (int)std::min<int64_t>((nt + kHeavyWarps - 1) / kHeavyWarps, (int64_t)ctx->num_sms * 6);
    a.cand_cap = kCandCap;
    a.n_threads = 0;
    if (!a.tally && nt > 0) {
        a.n_threads = (int64_t)solve_blocks * kBlk;
        // eight runs per warp, so that the warps end together, of 32 to 256 targets
        a.run = (int)std::min<int64_t>(256, std::max<int64_t>(32, nt * 32 / (8 * a.n_threads) / 32 * 32));
        a.cand = (uint32_t*)scratch(ctx, kSlotNgb0, (size_t)a.n_threads * kCandCap * sizeof(uint32_t));
        a.heavy_cap = (int)std::min<int64_t>(nt, kHeavyCap);
        const int64_t warps = (int64_t)heavy_blocks * kHeavyWarps;
        char* hb = (char*)scratch(ctx, kSlotNgb3, 64 + (size_t)a.heavy_cap * sizeof(DensHeavy) +
                                                      (size_t)warps * kWarpCand * sizeof(uint32_t));
        a.heavy_ctr = (unsigned int*)hb;
        a.heavy = (DensHeavy*)(hb + 64);
        a.warp_cand = (uint32_t*)(hb + 64 + (size_t)a.heavy_cap * sizeof(DensHeavy));
        check_cuda(cudaMemsetAsync(a.heavy_ctr, 0, 12, st), "memset");
    }
    a.h_default = 0.0;
    a.h_default_sys = nullptr;
    if (!h_start && t->n_systems > 1) {
        // each system's own default, from its own particles (all of them, massless too)
        const int S = t->n_systems;
        int64_t nmax = 0;
        for (int s = 0; s < S; ++s) nmax = std::max<int64_t>(nmax, t->in_off[s + 1] - t->in_off[s]);
        const int chunks = (int)std::min<int64_t>(64, std::max<int64_t>(1, (nmax + 8191) / 8192));
        const size_t nparts = (size_t)S * chunks;
        double* part = (double*)scratch(ctx, kSlotNgb2, nparts * 6 * 8);
        density_bbox_kernel<<<(int)nparts, kBlk, 0, st>>>(t->src, t->rank, t->in_off_dev, chunks, part);
        check_launch(ctx, "density_bbox_kernel");
        std::vector<double> hp(nparts * 6), hd(S, 0.0);
        check_cuda(cudaMemcpyAsync(hp.data(), part, hp.size() * 8, cudaMemcpyDeviceToHost, st), "d2h");
        check_cuda(cudaStreamSynchronize(st), "sync");
        for (int s = 0; s < S; ++s) {
            const int64_t ns = t->in_off[s + 1] - t->in_off[s];
            if (ns == 0) continue;  // an empty system owns no target
            double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
            for (int c = 0; c < chunks; ++c)
                for (int k = 0; k < 3; ++k) {
                    lo[k] = std::min(lo[k], hp[6 * ((size_t)s * chunks + c) + k]);
                    hi[k] = std::max(hi[k], hp[6 * ((size_t)s * chunks + c) + 3 + k]);
                }
            hd[s] = default_h(lo, hi, (double)ns, des_ngb, n_dims);
        }
        double* dhd = (double*)scratch(ctx, kSlotNgb1, (size_t)S * 8);
        check_cuda(cudaMemcpyAsync(dhd, hd.data(), (size_t)S * 8, cudaMemcpyHostToDevice, st), "h2d");
        check_cuda(cudaStreamSynchronize(st), "sync");  // hd is pageable and goes out of scope
        a.h_default_sys = dhd;
    } else if (!h_start) {
        // des_ngb particles at the mean number density of the bounding box of all particles
        const int nb = std::max(1, std::min(grid_of(ctx, t->n), ctx->num_sms * 2));
        double* part = (double*)scratch(ctx, kSlotNgb2, (size_t)nb * 6 * 8);
        bbox_all_kernel<<<nb, kBlk, 0, st>>>(t->src, t->n, part);
        check_launch(ctx, "bbox_all_kernel");
        std::vector<double> hp((size_t)nb * 6);
        check_cuda(cudaMemcpyAsync(hp.data(), part, hp.size() * 8, cudaMemcpyDeviceToHost, st), "d2h");
        check_cuda(cudaStreamSynchronize(st), "sync");
        double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
        for (int b = 0; b < nb; ++b)
            for (int k = 0; k < 3; ++k) {
                lo[k] = std::min(lo[k], hp[6 * b + k]);
                hi[k] = std::max(hi[k], hp[6 * b + 3 + k]);
            }
        a.h_default = default_h(lo, hi, (double)t->n, des_ngb, n_dims);
    }
    if (nt <= 0) return;
    if (a.tally) density_count_kernel<<<grid_of(ctx, nt), kBlk, 0, st>>>(a);
    else if (a.g.n_roots == 1) density_kernel<true><<<solve_blocks, kBlk, 0, st>>>(a);
    else density_kernel<false><<<solve_blocks, kBlk, 0, st>>>(a);
    check_launch(ctx, "density_kernel");
    if (!a.tally) {
        density_heavy_kernel<<<heavy_blocks, kHeavyWarps * 32, 0, st>>>(a);
        check_launch(ctx, "density_heavy_kernel");
    }
    if (a.tally) {
        check_cuda(cudaMemcpyAsync(ctx->pinned, a.tally, GT_NGB_COUNTERS * 8, cudaMemcpyDeviceToHost, st), "d2h");
        check_cuda(cudaStreamSynchronize(st), "sync");
        std::memcpy(tally, ctx->pinned, GT_NGB_COUNTERS * 8);
    }
}

}  // namespace gt
