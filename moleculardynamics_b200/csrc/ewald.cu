// ewald.cu -- Ewald summation and the SPC/E force field (forcefield/ewald.cpp,
// forcefield/spce_forcefield.cpp) on the device.
//
//   real space   erfc(alpha r)/r over intermolecular pairs with r < cutoff, taken
//                from a Verlet list built at cutoff + skin (the reference scans all
//                i<j pairs; the list holds exactly the pairs that can pass r < rc,
//                and membership uses the reference's exact min-image r^2);
//   self         -C alpha/sqrt(pi) sum q^2;
//   intra        -C q_i q_j erf(alpha r)/r over same-molecule pairs (min image),
//                from per-atom partner lists built once from the molecule ids;
//   reciprocal   sum_j q_j of the eight cos/sin products per k vector of one octant,
//                which together hold S(k) = sum_j q_j exp(i k.r_j) for every sign of
//                k's components, with the per-axis factors built by recurrence.
// The SPC/E force field adds O-O Lennard-Jones (oxygens = atoms with original
// index divisible by 3, as SpceForceField::gatherOxygens takes them) in the same
// pass over the real-space list.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "md_device.cuh"
#include "md_internal.cuh"

namespace mdb {
int verlet_build(md_verlet* v, md_system* sys, bool conditional);
int verlet_check(md_verlet* v, md_system* sys);
DispArgs disp_args(md_verlet* v, md_context* ctx, double* part);
int verlet_ensure_ready(md_verlet* v, md_system* sys, const char* who);
}  // namespace mdb

namespace mdb {

namespace {

constexpr double kPi = 3.14159265358979323846;
constexpr int kBlock = 256;
constexpr int kRealBlock = 64;  // the real-space pass

// ewald.hpp:10-13, ewald.cpp:17-21
double coulomb_prefactor() {
    const double e = 1.602176565e-19, eps0 = 8.854187817e-12, kB = 1.3806488e-23;
    return (e * e) / (4.0 * kPi * eps0) * 1e10 / kB;
}

struct RealArgs {
    double rc2, alpha, coulomb, two_alpha_over_sqrt_pi, neg_alpha2;
    int spce_lj;            // add O-O LJ (SPC/E)
    double sig2, four_eps, tf_eps;
    int lj_lfs;             // O-O LJ with linear force shift at the cutoff
    double rc, uc, dudrc;
    int quotient_r2;        // above this r^2 every dividend and quotient is finite: the bits
                            // of an FP32 square, the high word of an FP64 one
};

// Terms of one pair inside the cutoff: force coefficient (F = s d), real-space energy and
// virial, LJ energy and virial (zero where the pair has no such term).
template <class T>
struct RealTerms {
    T s, er, wr, el, wl;
};

// The real-space Coulomb (ewald.cpp:60-68) and O-O LJ (lennard_jones.cpp:62-77) terms of a
// pair at r2 in arithmetic T (FP32: MD_PRECISION_MIXED); div2 divides by r2, div1 by r.
template <class T, class Div2, class Div1>
__device__ __forceinline__ RealTerms<T> real_terms(T r2, T r, T cqq, bool coulomb, bool lj,
                                                   const RealArgs& a, Div2 div2, Div1 div1) {
    RealTerms<T> t = {T(0), T(0), T(0), T(0), T(0)};
    if (coulomb) {
        T erfc_ar, gauss;
        if constexpr (sizeof(T) == 4) {
            erfc_ar = erfcf(static_cast<T>(a.alpha) * r);
            gauss = expf(static_cast<T>(a.neg_alpha2) * r2);
        } else {
            erfc_ar = erfc(a.alpha * r);
            gauss = exp(a.neg_alpha2 * r2);
        }
        t.wr = cqq * (static_cast<T>(a.two_alpha_over_sqrt_pi) * gauss + div1(erfc_ar));
        t.s = div2(t.wr);
        t.er = div1(cqq * erfc_ar);
    }
    if (lj) {
        const T s2 = div2(static_cast<T>(a.sig2));
        const T s6 = s2 * s2 * s2;
        t.wl = static_cast<T>(a.tf_eps) * (T(2) * s6 * s6 - s6);
        t.el = static_cast<T>(a.four_eps) * (s6 * s6 - s6);
        if (a.lj_lfs) {
            t.el = t.el - static_cast<T>(a.uc) - (r - static_cast<T>(a.rc)) * static_cast<T>(a.dudrc);
            t.wl = t.wl + r * static_cast<T>(a.dudrc);
        }
        t.s += div2(t.wl);
    }
    return t;
}

// Separations whose dividends or quotients could leave the normal range (quotient() turns an
// infinite dividend into NaN, a division does not), and in FP64 the squares that
// reciprocal() does not serve with sigma^2 a power of two, divide in IEEE arithmetic.
template <class T>
__device__ __noinline__ RealTerms<T> real_terms_ieee(T r2, T cqq, bool coulomb, bool lj,
                                                     const RealArgs* a) {
    const T r = sqrt(r2);
    return real_terms<T>(r2, r, cqq, coulomb, lj, *a, [r2](T x) { return x / r2; },
                         [r](T x) { return x / r; });
}

template <class T>
__device__ __forceinline__ RealTerms<T> real_pair(T r2, T cqq, bool coulomb, bool lj,
                                                  const RealArgs& a) {
    bool fast;
    if constexpr (sizeof(T) == 4) fast = __float_as_int(r2) > a.quotient_r2;
    else fast = __double2hiint(r2) > a.quotient_r2 && !low_ones(r2);
    if (!fast) return real_terms_ieee<T>(r2, cqq, coulomb, lj, &a);
    T r;
    if constexpr (sizeof(T) == 4) r = __fsqrt_rn(r2);
    else r = __dsqrt_rn(r2);
    const T y2 = reciprocal(r2), y1 = reciprocal(r);
    return real_terms<T>(r2, r, cqq, coulomb, lj, a, [r2, y2](T x) { return quotient(x, r2, y2); },
                         [r, y1](T x) { return quotient(x, r, y1); });
}

// Real-space (and SPC/E O-O LJ) pair terms over the Verlet list.  out[0..3]:
// E_real, W_real, E_lj, W_lj.  mode 1 writes forces, mode 2 adds to them.
// MIXED: the displacement, the cutoff test and every sum stay FP64; the pair
// terms (erfc, exp, the LJ powers) are evaluated in FP32.
// A pair's five divisions are by r and r^2 alone and share two reciprocals; the next
// entry's index and site are requested while the current pair is evaluated.  Blocks of
// kRealBlock threads: small, so that the last wave of a few thousand sites is short.
// 12,288 sites, 16 threads a site: FP32 terms 120 us with five
// IEEE divisions, no prefetch and 128-thread blocks, 85 us so; FP64 terms 157 and 122 us.
template <int TPA, bool MIXED>
__global__ void __launch_bounds__(kRealBlock, MIXED ? 14 : 10)
k_ewald_real(const double4* __restrict__ pos, const double* __restrict__ q,
             const int64_t* __restrict__ mol, const int* __restrict__ nbr,
             const int* __restrict__ count, int stride, int64_t n, Box3 box,
             const __grid_constant__ RealArgs a, int mode, double* fxo, double* fyo, double* fzo,
             double* part, unsigned* ticket, double* out) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    const int64_t i = t / TPA;
    const int g = static_cast<int>(t % TPA);
    const Fold3 f3 = fold3_of(box);
    double fx = 0.0, fy = 0.0, fz = 0.0, er = 0.0, wr = 0.0, el = 0.0, wl = 0.0;
    if (i < n) {
        const double4 pi = pos[i];
        const double qi = q[i];
        const int64_t mi = mol[i];
        const bool oxy_i = a.spce_lj && (static_cast<int>(pi.w) % 3) == 0;
        const int cnt = min(count[i], stride);
        const int* row = nbr + i * static_cast<int64_t>(stride);
        int k = g;
        int j = k < cnt ? __ldg(row + k) : static_cast<int>(i);
        int jn = k + TPA < cnt ? __ldg(row + k + TPA) : static_cast<int>(i);
        double4 pj = ldg4(pos + j);
        double qj = __ldg(q + j);
        int64_t mj = __ldg(mol + j);
        for (; k < cnt; k += TPA) {
            const double4 pc = pj;
            const double qc = qj;
            const bool coul = mj != mi;
            // the next entry
            pj = ldg4(pos + jn);
            qj = __ldg(q + jn);
            mj = __ldg(mol + jn);
            jn = k + 2 * TPA < cnt ? __ldg(row + k + 2 * TPA) : jn;
            // r_lower - r_higher by original index has the reference's rounding
            const bool lo = pi.w < pc.w;
            double dx, dy, dz;
            min_image_pair(f3, pi, pc, lo, dx, dy, dz);
            const double r2 = norm2_exact(dx, dy, dz);
            if (!(r2 < a.rc2)) continue;
            const bool lj = oxy_i && (static_cast<int>(pc.w) % 3) == 0;
            using T = typename std::conditional<MIXED, float, double>::type;
            const RealTerms<T> p = real_pair<T>(static_cast<T>(r2), static_cast<T>(a.coulomb * (qi * qc)),
                                                coul, lj, a);
            if (lo) {
                er += p.er;
                wr += p.wr;
                el += p.el;
                wl += p.wl;
            }
            const double s = p.s;
            fx = fma(dx, s, fx);
            fy = fma(dy, s, fy);
            fz = fma(dz, s, fz);
        }
    }
#pragma unroll
    for (int o = TPA / 2; o > 0; o >>= 1) {
        fx += __shfl_xor_sync(0xffffffffu, fx, o);
        fy += __shfl_xor_sync(0xffffffffu, fy, o);
        fz += __shfl_xor_sync(0xffffffffu, fz, o);
    }
    if (i < n && g == 0) {
        if (mode == 1) {
            fxo[i] = fx;
            fyo[i] = fy;
            fzo[i] = fz;
        } else {
            fxo[i] += fx;
            fyo[i] += fy;
            fzo[i] += fz;
        }
    }
    double v[4] = {er, wr, el, wl};
    grid_reduce<4>(v, part, ticket, out);
}

// Intramolecular correction (ewald.cpp:79-110) per atom over its molecule partners
// (original indices, CSR); adds to forces, and the sum of q^2 of the self term with it.
// out[0..2]: E_intra, W_intra, sum q^2.
__global__ void k_ewald_intra(const double4* __restrict__ pos, const double* __restrict__ q,
                              const int* __restrict__ orig, const int* __restrict__ slot,
                              const int* __restrict__ off, const int* __restrict__ partner,
                              int64_t n, Box3 box, RealArgs a, int add_forces, double* fxo,
                              double* fyo, double* fzo, double* part, unsigned* ticket,
                              double* out) {
    const int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    const Fold3 f3 = fold3_of(box);
    double e = 0.0, vir = 0.0, q2 = 0.0;
    if (k < n) {
        const double4 pi = pos[k];
        const int oi = orig[k];
        q2 = q[k] * q[k];
        double fx = 0.0, fy = 0.0, fz = 0.0;
        for (int p = off[oi]; p < off[oi + 1]; ++p) {
            const int oj = partner[p];
            const int j = slot[oj];
            const double4 pj = pos[j];
            const bool lo = oi < oj;
            double dx, dy, dz;
            if (lo) min_image_wrapped(f3, pi.x, pi.y, pi.z, pj.x, pj.y, pj.z, dx, dy, dz);
            else min_image_wrapped(f3, pj.x, pj.y, pj.z, pi.x, pi.y, pi.z, dx, dy, dz);
            const double r2 = norm2_exact(dx, dy, dz);
            const double r = __dsqrt_rn(r2);
            const double cqq = a.coulomb * (q[k] * q[j]);
            const double erf_ar = erf(a.alpha * r);
            const double w = cqq * (a.two_alpha_over_sqrt_pi * exp(a.neg_alpha2 * r2) - erf_ar / r);
            const double s = lo ? w / r2 : -(w / r2);
            fx = fma(dx, s, fx);
            fy = fma(dy, s, fy);
            fz = fma(dz, s, fz);
            if (lo) {
                e += -cqq * erf_ar / r;
                vir += w;
            }
        }
        if (add_forces) {
            fxo[k] += fx;
            fyo[k] += fy;
            fzo[k] += fz;
        }
    }
    double v[3] = {e, vir, q2};
    grid_reduce<3>(v, part, ticket, out);
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// Reciprocal sums in separable real form.  With a, b, c each cos or sin,
//   A_abc(nx, ny, nz) = sum_j q_j a(nx kx0 x_j) b(ny ky0 y_j) c(nz kz0 z_j),  n >= 0,
// the eight sums of an octant vector carry every sign combination of (nx, ny, nz) at
// once: the coefficient f depends on |k| alone, and summing cos(k.(r_i - r_j)) over the
// signs leaves g(nx) g(ny) g(nz) times a product of three cosines (g(0) = 1, else 2), so
//   E = sum_octant f g g g sum_abc A_abc^2,
//   dE/dq(r) = U(r) = sum_octant 2 f g g g sum_abc A_abc a(x) b(y) c(z),  F = -q grad U.
// That is two multiply-adds per site and k vector for A and four for grad U, against
// about ten and sixteen with one complex exponential per vector.  A task is one (nx, ny)
// column of kColZ consecutive nz: a thread's register tile.
constexpr int kColZ = 4;            // nz per task
constexpr int kColSums = 8 * kColZ; // sums A_abc per task
constexpr int kTaskChunk = 32;      // tasks with one nz0, padded to whole warps
constexpr int kSumBlock = 128;

struct KArgs {
    const int4* task;   // nx, ny, nz0, 1 (0: padding)
    const double2* fac; // per task and nz: f g g g (0 outside the sphere), k^2
    int ntask, kmax;
    double a, b, c;     // 2 pi / L per axis
};

constexpr int kSiteTile = 32;

// Entries per axis of a site's factor table: nz0 + kColZ may pass kmax.
__host__ __device__ constexpr int table_axis(int kmax) { return (kmax / kColZ + 1) * kColZ; }

// Partial sums A_abc: block (tb, sb) takes tasks [tb * 128, +128) over the sites of slice
// sb, one task per thread, 32 sums in registers.  Per tile of 32 sites the factors
// e^{i m theta} of each axis (the charge folded into x) are built in shared memory by
// complex recurrence; a site then costs a thread four products, 32 multiply-adds and six
// 16-byte shared loads, four of them broadcasts (one nz0 per warp), so the FP64 pipe
// bounds the kernel (a register-operand outer product of this shape reaches 47 of its 64
// multiply-adds per clock and SM here).  12,288 sites, kmax 18 (12.2k half-space
// vectors): 268 us with one complex product chain per vector, 48 us in this form.
__global__ void __launch_bounds__(kSumBlock)
k_structure_factor(const double4* __restrict__ pos, const double* __restrict__ q, int64_t n,
                   KArgs ka, int64_t sites_per_slice, double* __restrict__ part) {
    extern __shared__ double2 tab[];  // 3 axes x table_axis(kmax) x (kSiteTile + 1)
    constexpr int kPad = kSiteTile + 1;  // consecutive m on different banks
    const int nT = table_axis(ka.kmax);
    const int t = blockIdx.x * kSumBlock + threadIdx.x;
    const int4 tk = t < ka.ntask ? __ldg(ka.task + t) : make_int4(0, 0, 0, 0);
    const double2* X = tab + tk.x * kPad;
    const double2* Y = tab + (nT + tk.y) * kPad;
    const double2* Z = tab + (2 * nT + tk.z) * kPad;
    const int64_t s0 = blockIdx.y * sites_per_slice;
    const int64_t s1 = min(n, s0 + sites_per_slice);
    double acc[kColZ][8];
#pragma unroll
    for (int z = 0; z < kColZ; ++z)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[z][j] = 0.0;
    for (int64_t base = s0; base < s1; base += kSiteTile) {
        __syncthreads();
        for (int w = threadIdx.x; w < 3 * kSiteTile; w += kSumBlock) {
            const int site = w % kSiteTile, axis = w / kSiteTile;
            const int64_t s = base + site;
            double2* T = tab + axis * nT * kPad + site;
            double2 v = make_double2(0.0, 0.0), e1 = v;
            if (s < s1) {
                const double4 p = pos[s];
                const double coord = axis == 0 ? p.x : (axis == 1 ? p.y : p.z);
                sincos((axis == 0 ? ka.a : (axis == 1 ? ka.b : ka.c)) * coord, &e1.y, &e1.x);
                v.x = axis == 0 ? q[s] : 1.0;
            }
            for (int m = 0; m < nT; ++m) {
                T[m * kPad] = v;
                v = cmul(v, e1);
            }
        }
        __syncthreads();
#pragma unroll 2
        for (int site = 0; site < kSiteTile; ++site) {
            const double2 x = X[site], y = Y[site];
            const double xy[4] = {x.x * y.x, x.x * y.y, x.y * y.x, x.y * y.y};
#pragma unroll
            for (int z = 0; z < kColZ; ++z) {
                const double2 zz = Z[z * kPad + site];
#pragma unroll
                for (int ab = 0; ab < 4; ++ab) {
                    acc[z][2 * ab] = fma(xy[ab], zz.x, acc[z][2 * ab]);
                    acc[z][2 * ab + 1] = fma(xy[ab], zz.y, acc[z][2 * ab + 1]);
                }
            }
        }
    }
    if (t >= ka.ntask) return;
    double* o = part + static_cast<int64_t>(blockIdx.y) * kColSums * ka.ntask + t;
#pragma unroll
    for (int z = 0; z < kColZ; ++z)
#pragma unroll
        for (int j = 0; j < 8; ++j) o[static_cast<int64_t>(8 * z + j) * ka.ntask] = acc[z][j];
}

// Adds the slices (eight groups of lanes, group g slices g, g + 8, ... in order, then the
// groups in order), reduces the reciprocal energy and virial, W = sum E(k)
// (1 - k^2 / (2 a^2)), and leaves the coefficients 2 f g g g A_abc of U, eight per
// octant vector.
constexpr int kFinalGroups = 8;

__global__ void __launch_bounds__(32 * kFinalGroups)
k_structure_final(const double* __restrict__ part, int slices, KArgs ka, double inv_2alpha2,
                  double* __restrict__ coef, double* rpart, unsigned* ticket, double* out) {
    __shared__ double sums[kFinalGroups][32];
    const int lane = threadIdx.x % 32, g = threadIdx.x / 32;
    const int idx = blockIdx.x * 32 + lane;  // kColSums * ntask is a multiple of 32
    const int64_t count = static_cast<int64_t>(kColSums) * ka.ntask;
    double A = 0.0;
#pragma unroll 8
    for (int s = g; s < slices; s += kFinalGroups) A += part[s * count + idx];
    sums[g][lane] = A;
    __syncthreads();
    double v[2] = {0.0, 0.0};
    if (g == 0) {
#pragma unroll
        for (int k = 1; k < kFinalGroups; ++k) A += sums[k][lane];
        const int j = idx / ka.ntask, t = idx % ka.ntask;
        const double2 f = ka.fac[t * kColZ + j / 8];
        const double e = f.x * A * A;
        v[0] = e;
        v[1] = e * (1.0 - f.y * inv_2alpha2);
        coef[static_cast<int64_t>(t) * kColSums + j] = 2.0 * f.x * A;
    }
    grid_reduce<2>(v, rpart, ticket, out);
}

// F = -q grad U (or, with CHARGE, dE_recip/dq = U) of one site per thread over a 2-D
// grid: blockIdx.x picks 128 sites, blockIdx.y a range of task chunks, so small systems
// still fill the GPU; k_recip_sum adds the ranges in order (deterministic).  A chunk's
// coefficients are staged in shared memory and read as broadcasts; the site's z factors
// of the chunk's kColZ nz stay in registers, x and y factors start with sincos at each
// chunk and continue by complex recurrence.  Per task and site 64 multiply-adds form
// G_ab = sum_c coef_abc c(z) and dG_ab/dz, about 23 more the gradient: the FP64 pipe
// bounds the kernel.  12,288 sites, kmax 18: 769 us with one complex exponential per
// vector, 108 us in this form; two sites a thread, sharing the broadcasts, measured the
// same.
template <bool CHARGE>
__global__ void __launch_bounds__(kSumBlock)
k_recip_force(const double4* __restrict__ pos, const double* __restrict__ q, int64_t n, KArgs ka,
              int chunks_per_slice, const double* __restrict__ coef, double4* __restrict__ part) {
    __shared__ double2 cs[kTaskChunk * kColSums / 2];
    __shared__ int4 tks[kTaskChunk];
    const int64_t s = blockIdx.x * static_cast<int64_t>(kSumBlock) + threadIdx.x;
    const double4 p = pos[s < n ? s : n - 1];
    double2 ex, ey, ez;
    sincos(ka.a * p.x, &ex.y, &ex.x);
    sincos(ka.b * p.y, &ey.y, &ey.x);
    sincos(ka.c * p.z, &ez.y, &ez.x);
    double ux = 0.0, uy = 0.0, uz = 0.0;
    const int chunks = ka.ntask / kTaskChunk;
    const int c0 = blockIdx.y * chunks_per_slice, c1 = min(chunks, c0 + chunks_per_slice);
    for (int c = c0; c < c1; ++c) {
        __syncthreads();
        const double2* src = reinterpret_cast<const double2*>(
            coef + static_cast<int64_t>(c) * kTaskChunk * kColSums);
        for (int w = threadIdx.x; w < kTaskChunk * kColSums / 2; w += kSumBlock) cs[w] = __ldg(src + w);
        if (threadIdx.x < kTaskChunk) tks[threadIdx.x] = __ldg(ka.task + c * kTaskChunk + threadIdx.x);
        __syncthreads();
        int4 tk = tks[0];
        double2 X, Y, Z[kColZ];
        double kz[kColZ];
        sincos(static_cast<double>(tk.x) * ka.a * p.x, &X.y, &X.x);
        sincos(static_cast<double>(tk.y) * ka.b * p.y, &Y.y, &Y.x);
        sincos(static_cast<double>(tk.z) * ka.c * p.z, &Z[0].y, &Z[0].x);
#pragma unroll
        for (int z = 0; z < kColZ; ++z) {
            if (z > 0) Z[z] = cmul(Z[z - 1], ez);
            kz[z] = static_cast<double>(tk.z + z) * ka.c;
        }
        for (int i = 0; i < kTaskChunk; ++i) {
            const int4 nt = tks[i];
            if (!nt.w) break;  // padding ends a chunk
            if (nt.x != tk.x) {  // the next column of x: ny starts again at 0
                X = cmul(X, ex);
                Y = make_double2(1.0, 0.0);
            } else if (nt.y != tk.y) {
                Y = cmul(Y, ey);
            }
            tk = nt;
            double G[4], D[4];
#pragma unroll
            for (int ab = 0; ab < 4; ++ab) G[ab] = D[ab] = 0.0;
#pragma unroll
            for (int z = 0; z < kColZ; ++z) {
                const double dc = kz[z] * Z[z].x, ds = -kz[z] * Z[z].y;
#pragma unroll
                for (int ab = 0; ab < 4; ++ab) {
                    const double2 B = cs[i * (kColSums / 2) + z * 4 + ab];
                    G[ab] = fma(B.x, Z[z].x, fma(B.y, Z[z].y, G[ab]));
                    if (!CHARGE) D[ab] = fma(B.x, ds, fma(B.y, dc, D[ab]));
                }
            }
            const double pc = fma(Y.x, G[0], Y.y * G[1]), ps = fma(Y.x, G[2], Y.y * G[3]);
            if (CHARGE) {
                ux = fma(X.x, pc, fma(X.y, ps, ux));
            } else {
                const double kx = static_cast<double>(tk.x) * ka.a;
                const double ky = static_cast<double>(tk.y) * ka.b;
                const double qc = fma(Y.x, G[1], -Y.y * G[0]), qsn = fma(Y.x, G[3], -Y.y * G[2]);
                const double rc = fma(Y.x, D[0], Y.y * D[1]), rs = fma(Y.x, D[2], Y.y * D[3]);
                ux = fma(kx, fma(X.x, ps, -X.y * pc), ux);
                uy = fma(ky, fma(X.x, qc, X.y * qsn), uy);
                uz = fma(X.x, rc, fma(X.y, rs, uz));
            }
        }
    }
    if (s >= n) return;
    if (CHARGE) {
        part[blockIdx.y * n + s] = make_double4(ux, 0.0, 0.0, 0.0);
    } else {
        const double mq = -q[s];
        part[blockIdx.y * n + s] = make_double4(mq * ux, mq * uy, mq * uz, 0.0);
    }
}

// Adds the slices' partial k-space forces (CHARGE: charge gradients), `lanes` (a power
// of two up to 32) per site: lane l sums slices l, l + lanes, ... in order, then the
// lanes combine by a fixed butterfly, so the result does not depend on scheduling.
template <bool CHARGE>
__global__ void k_recip_sum(const double4* __restrict__ part, int slices, int lanes, int64_t n,
                            double* fxo, double* fyo, double* fzo, double* dq) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    const int64_t s = t / lanes;
    const int lane = static_cast<int>(t % lanes);
    double fx = 0.0, fy = 0.0, fz = 0.0;
    if (s < n)
        for (int k = lane; k < slices; k += lanes) {
            const double4 v = part[k * n + s];
            fx += v.x;
            fy += v.y;
            fz += v.z;
        }
    for (int o = lanes / 2; o > 0; o >>= 1) {
        fx += __shfl_xor_sync(0xffffffffu, fx, o);
        fy += __shfl_xor_sync(0xffffffffu, fy, o);
        fz += __shfl_xor_sync(0xffffffffu, fz, o);
    }
    if (s >= n || lane != 0) return;
    if (CHARGE) {
        dq[s] += fx;
    } else {
        fxo[s] += fx;
        fyo[s] += fy;
        fzo[s] += fz;
    }
}

// Task chunks per block of the k-space force pass: enough slices for six blocks an SM,
// which take turns on the four resident, at most one per chunk.  12,288 sites: 126 us with
// as many blocks as are resident at once (the longest block sets the time), 108 us so.
int recip_chunks_per_slice(const md_context* ctx, int64_t n, int ntask) {
    const int chunks = ntask / kTaskChunk;
    const int64_t site_blocks = (n + kSumBlock - 1) / kSumBlock;
    int64_t slices = (6 * static_cast<int64_t>(ctx->sm_count) + site_blocks - 1) / site_blocks;
    slices = std::max<int64_t>(1, std::min<int64_t>(slices, chunks));
    return static_cast<int>((chunks + slices - 1) / slices);
}

__global__ void k_to_slot4(const int* __restrict__ slot, int64_t n, const double4* in, double4* out) {
    const int64_t o = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (o < n) out[slot[o]] = in[o];
}

__global__ void k_to_orig4(const int* __restrict__ orig, int64_t n, const double4* in, double4* out) {
    const int64_t s = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (s < n) out[orig[s]] = in[s];
}

__global__ void k_to_orig1(const int* __restrict__ orig, int64_t n, const double* in, double* out) {
    const int64_t s = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (s < n) out[orig[s]] = in[s];
}

// Charge gradient of the real-space and intramolecular terms, plus the self
// term, per atom (device order):
//   dE/dq_i = sum_j C q_j erfc(a r)/r (other molecules, r < rc)
//           - sum_j C q_j erf(a r)/r (same molecule) - 2 C a/sqrt(pi) q_i
__global__ void __launch_bounds__(kBlock)
k_ewald_dq(const double4* __restrict__ pos, const double* __restrict__ q,
           const int64_t* __restrict__ mol, const int* __restrict__ nbr,
           const int* __restrict__ count, int stride, const int* __restrict__ orig,
           const int* __restrict__ slot, const int* __restrict__ off,
           const int* __restrict__ partner, int64_t n, Box3 box, RealArgs a, double* dq) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const Fold3 f3 = fold3_of(box);
    const double4 pi = pos[i];
    const int64_t mi = mol[i];
    double acc = 0.0;
    const int cnt = min(count[i], stride);
    const int* row = nbr + i * static_cast<int64_t>(stride);
    for (int k = 0; k < cnt; ++k) {
        const int j = __ldg(row + k);
        if (mol[j] == mi) continue;
        const double4 pj = ldg4(pos + j);
        double dx, dy, dz;
        min_image_wrapped(f3, pi.x, pi.y, pi.z, pj.x, pj.y, pj.z, dx, dy, dz);
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (!(r2 < a.rc2)) continue;
        const double r = sqrt(r2);
        acc += a.coulomb * q[j] * erfc(a.alpha * r) / r;
    }
    const int oi = orig[i];
    for (int p = off[oi]; p < off[oi + 1]; ++p) {
        const int j = slot[partner[p]];
        const double4 pj = pos[j];
        double dx, dy, dz;
        min_image_wrapped(f3, pi.x, pi.y, pi.z, pj.x, pj.y, pj.z, dx, dy, dz);
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        acc -= a.coulomb * q[j] * erf(a.alpha * r) / r;
    }
    acc -= a.coulomb * a.two_alpha_over_sqrt_pi * q[i];  // 2 C a / sqrt(pi) q_i
    dq[i] = acc;
}

// Hessian-vector product of the real-space Coulomb forces (other molecules,
// r < rc): out_i = sum_j [g (u_i - u_j) + 2 g' d (d . (u_i - u_j))] with
// F_i = sum_j g(r^2) d, g = C q_i q_j (A e^{-a^2 r^2}/r^2 + erfc(a r)/r^3), A = 2a/sqrt(pi).
__global__ void __launch_bounds__(kBlock)
k_ewald_real_hvp(const double4* __restrict__ pos, const double* __restrict__ q,
                 const int64_t* __restrict__ mol, const int* __restrict__ nbr,
                 const int* __restrict__ count, int stride, int64_t n, Box3 box, RealArgs a,
                 const double4* __restrict__ u, double4* out) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const Fold3 f3 = fold3_of(box);
    const double4 pi = pos[i], ui = u[i];
    const int64_t mi = mol[i];
    const double qi = q[i];
    const double a3 = a.alpha * a.alpha * a.two_alpha_over_sqrt_pi;  // 2 a^3 / sqrt(pi)
    const double a1 = 1.5 * a.two_alpha_over_sqrt_pi;                 // 3 a / sqrt(pi)
    double hx = 0.0, hy = 0.0, hz = 0.0;
    const int cnt = min(count[i], stride);
    const int* row = nbr + i * static_cast<int64_t>(stride);
    for (int k = 0; k < cnt; ++k) {
        const int j = __ldg(row + k);
        if (mol[j] == mi) continue;
        const double4 pj = ldg4(pos + j);
        double dx, dy, dz;
        min_image_wrapped(f3, pi.x, pi.y, pi.z, pj.x, pj.y, pj.z, dx, dy, dz);
        const double s = dx * dx + dy * dy + dz * dz;
        if (!(s < a.rc2)) continue;
        const double r = sqrt(s);
        const double cqq = a.coulomb * qi * q[j];
        const double ex = exp(a.neg_alpha2 * s), ec = erfc(a.alpha * r);
        const double g = cqq * (a.two_alpha_over_sqrt_pi * ex / s + ec / (s * r));
        const double gs = -cqq * (a3 * ex / s + a1 * ex / (s * s) + 1.5 * ec / (s * s * r));
        const double4 uj = u[j];
        const double ux = ui.x - uj.x, uy = ui.y - uj.y, uz = ui.z - uj.z;
        const double dm = dx * ux + dy * uy + dz * uz;
        hx += g * ux + 2.0 * gs * dx * dm;
        hy += g * uy + 2.0 * gs * dy * dm;
        hz += g * uz + 2.0 * gs * dz * dm;
    }
    out[i] = make_double4(hx, hy, hz, 0.0);
}

// Threads per atom of the real-space pass: the fewest (at least 4) that put
// about a thousand threads on every SM, so that a few thousand sites still
// spread over the whole GPU instead of a dozen SMs; at most a warp.
int real_tpa(const md_context* ctx, int64_t n) {
    const int64_t want = 1024 * static_cast<int64_t>(ctx->sm_count);
    int tpa = 4;
    while (tpa < 32 && n * tpa < want) tpa *= 2;
    return tpa;
}

template <int TPA, bool MIXED>
void launch_real_t(md_system* sys, md_verlet* v, const RealArgs& a, int mode, double* fx,
                   double* fy, double* fz, double* part, unsigned* ticket, double* out) {
    const int64_t threads = std::max<int64_t>(sys->n * TPA, 1);
    k_ewald_real<TPA, MIXED><<<grid_for(threads, kRealBlock), kRealBlock, 0, sys->ctx->stream>>>(
        sys->cur.pos, sys->cur.charge, sys->cur.mol, v->nbr.as<int>(), v->count.as<int>(),
        v->stride, sys->n, Box3{{sys->box[0], sys->box[1], sys->box[2]},
                                {sys->inv_box[0], sys->inv_box[1], sys->inv_box[2]}},
        a, mode, fx, fy, fz, part, ticket, out);
}

// mode 1 writes (fx, fy, fz), 2 adds to them; part holds 4 doubles per block.
template <bool MIXED>
void launch_real_p(md_system* sys, md_verlet* v, const RealArgs& a, int mode, int tpa, double* fx,
                   double* fy, double* fz, double* part, unsigned* ticket, double* out) {
    switch (tpa) {
        case 32: launch_real_t<32, MIXED>(sys, v, a, mode, fx, fy, fz, part, ticket, out); break;
        case 16: launch_real_t<16, MIXED>(sys, v, a, mode, fx, fy, fz, part, ticket, out); break;
        case 8: launch_real_t<8, MIXED>(sys, v, a, mode, fx, fy, fz, part, ticket, out); break;
        default: launch_real_t<4, MIXED>(sys, v, a, mode, fx, fy, fz, part, ticket, out); break;
    }
}

void launch_real(md_system* sys, md_verlet* v, const RealArgs& a, int mode, int tpa, bool mixed,
                 double* fx, double* fy, double* fz, double* part, unsigned* ticket, double* out) {
    if (mixed) launch_real_p<true>(sys, v, a, mode, tpa, fx, fy, fz, part, ticket, out);
    else launch_real_p<false>(sys, v, a, mode, tpa, fx, fy, fz, part, ticket, out);
}

}  // namespace

}  // namespace mdb

// Result slots inside kResEwald (doubles).
enum {
    kEwReal = 0, kEwRealW, kEwLj, kEwLjW, kEwIntra, kEwIntraW, kEwQ2, kEwRecip, kEwRecipW,
    kEwCount
};

struct md_ewald {
    md_context* ctx = nullptr;
    double cutoff = 10.0;
    int kmax = 5;
    double alpha_in = 0.0;
    double skin = 1.0;
    bool spce = false;
    double sigma_o = 0, epsilon_o = 0;
    int lj_truncation = MD_TRUNCATED;
    md_verlet* list = nullptr;
    double list_box[3] = {0, 0, 0};
    // topology (per original index)
    md_system* topo_sys = nullptr;
    uint64_t topo_version = 0;
    int64_t topo_n = -1;
    mdb::DevBuf partner_off, partner_idx;
    int64_t npartners = 0;
    // k vectors
    double kbox[3] = {0, 0, 0};
    int k_kmax = -1;
    double k_alpha = 0.0;
    mdb::DevBuf ktask, kfac, kcoef;
    int nk = 0, ntask = 0;        // half-space vectors; tasks, whole chunks of them
    double last[kEwCount] = {0};
    double alpha = 0.0;
    mdb::PmeState* pme = nullptr;  // reciprocal term by smooth PME instead of k-vector sums
    bool mixed = false;            // FP32 real-space pair terms (MD_PRECISION_MIXED)
};

namespace mdb {

namespace {

int ewald_topology(md_ewald* ew, md_system* sys) {
    if (ew->topo_sys == sys && ew->topo_version == sys->mol_version && ew->topo_n == sys->n)
        return MD_OK;
    const int64_t n = sys->n;
    std::vector<int64_t> mol(static_cast<size_t>(n));
    if (n > 0) MDB_TRY(md_system_get_molecule_ids(sys, mol.data()));
    // group atoms by molecule (index order within each molecule)
    std::unordered_map<int64_t, std::vector<int>> groups;
    groups.reserve(static_cast<size_t>(n));
    for (int64_t i = 0; i < n; ++i) groups[mol[i]].push_back(static_cast<int>(i));
    std::vector<int> off(static_cast<size_t>(n + 1), 0), idx;
    for (int64_t i = 0; i < n; ++i) off[i + 1] = static_cast<int>(groups[mol[i]].size()) - 1;
    for (int64_t i = 0; i < n; ++i) off[i + 1] += off[i];
    idx.resize(static_cast<size_t>(off[n]));
    for (int64_t i = 0; i < n; ++i) {
        int at = off[i];
        for (int j : groups[mol[i]])
            if (j != i) idx[at++] = j;
    }
    MDB_TRY(ew->partner_off.ensure(sizeof(int) * (n + 1)));
    MDB_TRY(ew->partner_idx.ensure(sizeof(int) * std::max<size_t>(idx.size(), 1)));
    MDB_CUDA(cudaMemcpy(ew->partner_off.ptr, off.data(), sizeof(int) * (n + 1), cudaMemcpyHostToDevice));
    if (!idx.empty())
        MDB_CUDA(cudaMemcpy(ew->partner_idx.ptr, idx.data(), sizeof(int) * idx.size(),
                            cudaMemcpyHostToDevice));
    ew->npartners = static_cast<int64_t>(idx.size());
    ew->topo_sys = sys;
    ew->topo_version = sys->mol_version;
    ew->topo_n = n;
    return MD_OK;
}

// The octant's k vectors (ewald.cpp:112-172: n in [-kmax, kmax]^3, 0 < |n|^2 < kmax^2 + 2,
// which the octant's signs cover) as tasks of kColZ consecutive nz, grouped by nz0; within
// a group nx ascends, and for each nx ny ascends from 0.
int ewald_kvectors(md_ewald* ew, const double box[3], double alpha) {
    if (ew->k_kmax == ew->kmax && ew->k_alpha == alpha && ew->kbox[0] == box[0] &&
        ew->kbox[1] == box[1] && ew->kbox[2] == box[2])
        return MD_OK;
    const int kmax = ew->kmax;
    const double volume = box[0] * box[1] * box[2];
    const double kx0 = 2.0 * kPi / box[0], ky0 = 2.0 * kPi / box[1], kz0 = 2.0 * kPi / box[2];
    const int n2max = kmax * kmax + 2;
    const double coulomb = coulomb_prefactor();
    std::vector<int4> task;
    std::vector<double2> fac;
    int full = 0;  // vectors of the full set
    for (int z0 = 0; z0 <= kmax; z0 += kColZ) {
        for (int nx = 0; nx <= kmax; ++nx) {
            for (int ny = 0; ny <= kmax && nx * nx + ny * ny + z0 * z0 < n2max; ++ny) {
                task.push_back(make_int4(nx, ny, z0, 1));
                for (int nz = z0; nz < z0 + kColZ; ++nz) {
                    const int n2 = nx * nx + ny * ny + nz * nz;
                    if (nz > kmax || n2 == 0 || n2 >= n2max) {
                        fac.push_back(make_double2(0.0, 0.0));
                        continue;
                    }
                    const int signs = (nx ? 2 : 1) * (ny ? 2 : 1) * (nz ? 2 : 1);
                    const double kxv = kx0 * static_cast<double>(nx);
                    const double kyv = ky0 * static_cast<double>(ny);
                    const double kzv = kz0 * static_cast<double>(nz);
                    const double k2 = kxv * kxv + kyv * kyv + kzv * kzv;
                    const double factor =
                        coulomb * (2.0 * kPi / volume) * std::exp(-k2 / (4.0 * alpha * alpha)) / k2;
                    fac.push_back(make_double2(signs * factor, k2));
                    full += signs;
                }
            }
        }
        while (task.size() % kTaskChunk) {
            task.push_back(make_int4(0, 0, z0, 0));
            for (int z = 0; z < kColZ; ++z) fac.push_back(make_double2(0.0, 0.0));
        }
    }
    ew->nk = full / 2;
    ew->ntask = ew->nk > 0 ? static_cast<int>(task.size()) : 0;
    if (ew->ntask > 0) {
        MDB_TRY(ew->ktask.ensure(sizeof(int4) * task.size()));
        MDB_TRY(ew->kfac.ensure(sizeof(double2) * fac.size()));
        MDB_TRY(ew->kcoef.ensure(sizeof(double) * kColSums * task.size()));
        MDB_CUDA(cudaMemcpy(ew->ktask.ptr, task.data(), sizeof(int4) * task.size(), cudaMemcpyHostToDevice));
        MDB_CUDA(cudaMemcpy(ew->kfac.ptr, fac.data(), sizeof(double2) * fac.size(), cudaMemcpyHostToDevice));
    }
    ew->k_kmax = kmax;
    ew->k_alpha = alpha;
    for (int d = 0; d < 3; ++d) ew->kbox[d] = box[d];
    return MD_OK;
}

int ewald_list_gated(md_ewald* ew, md_system* sys, bool checked) {
    if (!checked) MDB_TRY(verlet_check(ew->list, sys));
    return verlet_build(ew->list, sys, true);
}

int ewald_list(md_ewald* ew, md_system* sys) {
    if (ew->list && (ew->list_box[0] != sys->box[0] || ew->list_box[1] != sys->box[1] ||
                     ew->list_box[2] != sys->box[2])) {
        md_verlet_destroy(ew->list);
        ew->list = nullptr;
    }
    if (!ew->list) {
        MDB_TRY(md_verlet_create(ew->ctx, sys->box, ew->cutoff, ew->skin, &ew->list));
        for (int d = 0; d < 3; ++d) ew->list_box[d] = sys->box[d];
    }
    md_verlet* v = ew->list;
    if (!v->sys || v->sys != sys || v->n != sys->n || v->epoch != sys->epoch) {
        MDB_TRY(verlet_build(v, sys, false));
        return MD_OK;
    }
    int f = 0;
    MDB_TRY(md_verlet_needs_rebuild(v, sys, &f));
    if (f) MDB_TRY(verlet_build(v, sys, false));
    return MD_OK;
}

}  // namespace

// k-space forces added to the system's forces (charge = false), or
// dE_recip/dq added to dq (device order); the coefficients must be current.
int recip_force_async(md_ewald* ew, md_system* sys, const KArgs& ka, bool charge, double* dq) {
    md_context* ctx = sys->ctx;
    const int64_t n = sys->n;
    if (n == 0 || ew->ntask == 0) return MD_OK;
    const int per = recip_chunks_per_slice(ctx, n, ew->ntask);
    const int slices = (ew->ntask / kTaskChunk + per - 1) / per;
    void* scratch;
    MDB_TRY(ctx_scratch(ctx, sizeof(double4) * static_cast<size_t>(slices) * n, &scratch));
    const dim3 grid(static_cast<unsigned>((n + kSumBlock - 1) / kSumBlock), static_cast<unsigned>(slices));
    double4* part = static_cast<double4*>(scratch);
    int lanes = 1;
    while (lanes < 32 && lanes < slices) lanes *= 2;
    const unsigned sum_grid = grid_for(lanes * n, kBlock);
    if (charge) {
        k_recip_force<true><<<grid, kSumBlock, 0, ctx->stream>>>(
            sys->cur.pos, sys->cur.charge, n, ka, per, ew->kcoef.as<double>(), part);
        k_recip_sum<true><<<sum_grid, kBlock, 0, ctx->stream>>>(part, slices, lanes, n, nullptr,
                                                               nullptr, nullptr, dq);
    } else {
        k_recip_force<false><<<grid, kSumBlock, 0, ctx->stream>>>(
            sys->cur.pos, sys->cur.charge, n, ka, per, ew->kcoef.as<double>(), part);
        k_recip_sum<false><<<sum_grid, kBlock, 0, ctx->stream>>>(
            part, slices, lanes, n, sys->cur.fx, sys->cur.fy, sys->cur.fz, nullptr);
    }
    ctx->launches += 2;
    MDB_CHECK_LAUNCH();
    return MD_OK;
}

RealArgs real_args_of(const md_ewald* ew, double alpha, bool mixed) {
    RealArgs a;
    a.rc2 = ew->cutoff * ew->cutoff;
    a.alpha = alpha;
    a.coulomb = coulomb_prefactor();
    a.two_alpha_over_sqrt_pi = 2.0 * alpha / std::sqrt(kPi);
    a.neg_alpha2 = -alpha * alpha;
    a.spce_lj = ew->spce ? 1 : 0;
    a.sig2 = ew->sigma_o * ew->sigma_o;
    a.four_eps = 4.0 * ew->epsilon_o;
    a.tf_eps = 24.0 * ew->epsilon_o;
    a.lj_lfs = ew->lj_truncation == MD_LINEAR_FORCE_SHIFT ? 1 : 0;
    a.rc = ew->cutoff;
    // lennard_jones.cpp:32-48
    const double s2 = a.sig2 / a.rc2, s6 = s2 * s2 * s2;
    a.uc = 4.0 * ew->epsilon_o * (s6 * s6 - s6);
    a.dudrc = -(24.0 * ew->epsilon_o * (2.0 * s6 * s6 - s6)) / ew->cutoff;
    // 48 eps (sigma^2 / r^2)^6 and that over r^2 below the largest numbers
    const double top = std::pow(a.sig2, 6.0) * std::max(2.0, 2.0 * a.tf_eps) / (mixed ? 1e37 : 1e307);
    const double line = std::max({1e-15, std::pow(top, 1.0 / 6.0), std::pow(top, 1.0 / 7.0)});
    const float line32 = static_cast<float>(std::min(line, 3e38));
    int64_t bits;
    std::memcpy(&bits, &line, sizeof bits);
    a.quotient_r2 = static_cast<int>(bits >> 32);
    if (mixed) std::memcpy(&a.quotient_r2, &line32, sizeof line32);
    return a;
}

KArgs kargs_of(md_ewald* ew, const md_system* sys) {
    KArgs ka;
    ka.task = ew->ktask.as<int4>();
    ka.fac = ew->kfac.as<double2>();
    ka.ntask = ew->ntask;
    ka.kmax = ew->kmax;
    ka.a = 2.0 * kPi / sys->box[0];
    ka.b = 2.0 * kPi / sys->box[1];
    ka.c = 2.0 * kPi / sys->box[2];
    return ka;
}

// Everything of one evaluation, asynchronously; results land in kResEwald slots.
// mode: 0 energies only, 1 zero + accumulate forces, 2 accumulate onto forces.
// gated: the neighbour list is maintained by device-decided rebuilds (no host
// synchronisation; the list must already be built for this system); checked: the kernel
// that moved the sites has set the list's rebuild flag (ewald_disp_args).
int ewald_eval_async(md_ewald* ew, md_system* sys, int mode, bool gated, bool checked) {
    md_context* ctx = sys->ctx;
    const int64_t n = sys->n;
    double min_len = std::min(sys->box[0], std::min(sys->box[1], sys->box[2]));
    const double alpha = ew->alpha_in > 0.0 ? ew->alpha_in : 5.6 / min_len;  // ewald.cpp:40
    ew->alpha = alpha;
    if (gated) {
        MDB_TRY(ewald_list_gated(ew, sys, checked));
    } else {
        MDB_TRY(ewald_topology(ew, sys));
        if (!ew->pme) MDB_TRY(ewald_kvectors(ew, sys->box, alpha));
        MDB_TRY(ewald_list(ew, sys));
    }
    md_verlet* v = ew->list;
    const RealArgs a = real_args_of(ew, alpha, ew->mixed);
    double* res = ctx_result(ctx, kResEwald);
    const Box3 box{{sys->box[0], sys->box[1], sys->box[2]},
                   {sys->inv_box[0], sys->inv_box[1], sys->inv_box[2]}};
    double* part;
    const int tpa = real_tpa(ctx, n);
    const int64_t real_threads = std::max<int64_t>(n * tpa, 1);
    MDB_TRY(ctx_partials(ctx, 4 * static_cast<size_t>(grid_for(real_threads, kRealBlock)), &part));
    // real space (+ O-O LJ): with forces it writes (mode 1) or adds (mode 2); for
    // energies only it writes into the scratch force sink of a zero-force pass.
    ctx_time_begin(ctx, MD_KERNEL_EWALD_REAL);
    if (mode == 0) {
        // energies only: run the pair pass without touching forces by pointing the
        // sink at scratch (never read back)
        double* sink;
        MDB_TRY(ctx_scratch(ctx, 3 * sizeof(double) * static_cast<size_t>(std::max<int64_t>(n, 1)),
                            reinterpret_cast<void**>(&sink)));
        launch_real(sys, v, a, 1, tpa, ew->mixed, sink, sink + n, sink + 2 * n, part,
                    ctx_counter(ctx, 4), res + kEwReal);
    } else {
        launch_real(sys, v, a, mode, tpa, ew->mixed, sys->cur.fx, sys->cur.fy, sys->cur.fz,
                    part, ctx_counter(ctx, 4), res + kEwReal);
    }
    ctx_time_end(ctx, MD_KERNEL_EWALD_REAL);
    // intramolecular correction
    if (n > 0) {
        k_ewald_intra<<<grid_for(n, kBlock), kBlock, 0, ctx->stream>>>(
            sys->cur.pos, sys->cur.charge, sys->cur.orig, sys->slot, ew->partner_off.as<int>(),
            ew->partner_idx.as<int>(), n, box, a, mode != 0 ? 1 : 0, sys->cur.fx, sys->cur.fy,
            sys->cur.fz, part, ctx_counter(ctx, 5), res + kEwIntra);
    }
    // reciprocal space
    ctx_time_begin(ctx, MD_KERNEL_EWALD_RECIP);
    const KArgs ka = kargs_of(ew, sys);
    if (ew->pme) {
        MDB_TRY(pme_eval_async(ew->pme, sys, alpha, coulomb_prefactor(), mode, res + kEwRecip,
                               ctx_counter(ctx, 12)));
    } else if (ew->ntask > 0 && n > 0) {
        const int tblocks = (ew->ntask + kSumBlock - 1) / kSumBlock;
        // enough site slices to give every SM three blocks
        int64_t slices = std::max<int64_t>(1, (3 * ctx->sm_count) / tblocks);
        slices = std::min<int64_t>(slices, (n + kSiteTile - 1) / kSiteTile);
        const int64_t per = ((n + slices - 1) / slices + kSiteTile - 1) / kSiteTile * kSiteTile;
        slices = (n + per - 1) / per;
        // the slices' sums, like the force pass's after them, live in the context's
        // scratch only until the kernel that adds them
        void* scratch;
        MDB_TRY(ctx_scratch(ctx, sizeof(double) * kColSums * static_cast<size_t>(slices) * ew->ntask,
                            &scratch));
        double* kpart = static_cast<double*>(scratch);
        const size_t smem = sizeof(double2) * 3 * table_axis(ew->kmax) * (kSiteTile + 1);
        if (smem > 48 * 1024)
            MDB_CUDA(cudaFuncSetAttribute(k_structure_factor,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(smem)));
        k_structure_factor<<<dim3(tblocks, static_cast<unsigned>(slices)), kSumBlock, smem, ctx->stream>>>(
            sys->cur.pos, sys->cur.charge, n, ka, per, kpart);
        const int fblocks = kColSums * ew->ntask / 32;
        double* rp;
        MDB_TRY(ctx_partials(ctx, 2 * static_cast<size_t>(fblocks), &rp));
        k_structure_final<<<fblocks, 32 * kFinalGroups, 0, ctx->stream>>>(
            kpart, static_cast<int>(slices), ka, 1.0 / (2.0 * alpha * alpha),
            ew->kcoef.as<double>(), rp, ctx_counter(ctx, 7), res + kEwRecip);
        if (mode != 0) MDB_TRY(recip_force_async(ew, sys, ka, false, nullptr));
    } else {
        MDB_CUDA(cudaMemsetAsync(res + kEwRecip, 0, 2 * sizeof(double), ctx->stream));
    }
    ctx_time_end(ctx, MD_KERNEL_EWALD_RECIP);
    MDB_CHECK_LAUNCH();
    ctx->launches += 5;
    return MD_OK;
}

// The displacement check of the built list, for a kernel of nblocks blocks that moves the sites.
int ewald_disp_args(md_ewald* ew, md_context* ctx, int nblocks, DispArgs* d) {
    double* part;
    MDB_TRY(ctx_partials(ctx, 2 * static_cast<size_t>(nblocks), &part));
    *d = disp_args(ew->list, ctx, part);
    return MD_OK;
}

int ewald_read(md_ewald* ew, md_context* ctx) {
    MDB_TRY(ctx_read_results(ctx, kResEwald, kEwCount, ew->last));
    return MD_OK;
}

}  // namespace mdb

using namespace mdb;

namespace {

int ewald_new(md_context* ctx, double cutoff, int kmax, double alpha, md_ewald** out) {
    if (!ctx || !out) return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_create: NULL argument");
    if (!(cutoff > 0.0) || kmax < 0)
        return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_create: cutoff must be > 0 and kmax >= 0");
    md_ewald* ew = new (std::nothrow) md_ewald();
    if (!ew) return fail(MD_ERR_OUT_OF_MEMORY, "md_ewald_create: host allocation");
    ew->ctx = ctx;
    ew->cutoff = cutoff;
    ew->kmax = kmax;
    ew->alpha_in = alpha;
    *out = ew;
    return MD_OK;
}

void fill_terms(const md_ewald* ew, double terms[4], double* virial) {
    const double coulomb = coulomb_prefactor();
    // ewald.cpp:76: -C alpha / sqrt(pi) * sum q^2
    const double self = -coulomb * ew->alpha / std::sqrt(kPi) * ew->last[kEwQ2];
    if (terms) {
        terms[0] = ew->last[kEwReal];
        terms[1] = ew->last[kEwRecip];
        terms[2] = self;
        terms[3] = ew->last[kEwIntra];
    }
    if (virial) *virial = ew->last[kEwRealW] + ew->last[kEwIntraW] + ew->last[kEwRecipW];
}

}  // namespace

extern "C" {

double md_coulomb_prefactor(void) { return coulomb_prefactor(); }

int md_ewald_create(md_context* ctx, double cutoff, int kmax, double alpha, md_ewald** out) {
    graph_epoch_bump();
    return ewald_new(ctx, cutoff, kmax, alpha, out);
}

int md_ewald_destroy(md_ewald* ew) {
    graph_epoch_bump();
    if (!ew) return MD_OK;
    if (ew->list) md_verlet_destroy(ew->list);
    if (ew->pme) {
        cudaStreamSynchronize(ew->ctx->stream);
        pme_destroy(ew->pme);
    }
    ew->partner_off.release();
    ew->partner_idx.release();
    ew->ktask.release();
    ew->kfac.release();
    ew->kcoef.release();
    delete ew;
    return MD_OK;
}

int md_ewald_set_skin(md_ewald* ew, double skin) {
    graph_epoch_bump();
    if (!ew || !(skin >= 0.0)) return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_set_skin: bad argument");
    ew->skin = skin;
    if (ew->list) {
        md_verlet_destroy(ew->list);
        ew->list = nullptr;
    }
    return MD_OK;
}

int md_ewald_compute(md_ewald* ew, md_system* sys, int mode, double terms[4], double* virial) {
    if (!ew || !sys) return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_compute: NULL argument");
    if (mode < 0 || mode > 2) return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_compute: mode %d", mode);
    if (sys->ctx != ew->ctx) return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_compute: context mismatch");
    MDB_TRY(ewald_eval_async(ew, sys, mode, false, false));
    MDB_TRY(ewald_read(ew, sys->ctx));
    fill_terms(ew, terms, virial);
    return MD_OK;
}

namespace {

// per-atom vectors between the caller's order (n x 3 host) and device double4
int upload_vec(md_system* sys, const double* u, double4* dev_orig, double4* dev) {
    const int64_t n = sys->n;
    std::vector<double4> h(static_cast<size_t>(n));
    for (int64_t o = 0; o < n; ++o) h[o] = make_double4(u[3 * o], u[3 * o + 1], u[3 * o + 2], 0.0);
    MDB_CUDA(cudaMemcpyAsync(dev_orig, h.data(), sizeof(double4) * n, cudaMemcpyHostToDevice,
                             sys->ctx->stream));
    MDB_CUDA(cudaStreamSynchronize(sys->ctx->stream));
    k_to_slot4<<<grid_for(n, kBlock), kBlock, 0, sys->ctx->stream>>>(sys->slot, n, dev_orig, dev);
    return MD_OK;
}

}  // namespace

int md_ewald_set_pme(md_ewald* ew, int kx, int ky, int kz, int order) {
    graph_epoch_bump();
    if (!ew) return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_set_pme: NULL");
    if (kx == 0 && ky == 0 && kz == 0) {  // back to the k-vector sums
        if (ew->pme) {
            cudaStreamSynchronize(ew->ctx->stream);
            pme_destroy(ew->pme);
            ew->pme = nullptr;
        }
        return MD_OK;
    }
    if (order != 4 && order != 6 && order != 8)
        return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_set_pme: order must be 4, 6 or 8");
    const int K[3] = {kx, ky, kz};
    for (int d = 0; d < 3; ++d)
        if (K[d] < 2 * order || K[d] > 4096)
            return fail(MD_ERR_INVALID_ARGUMENT,
                        "md_ewald_set_pme: grid sizes must lie in [2 * order, 4096]");
    mdb::PmeState* s = nullptr;
    MDB_TRY(pme_create(ew->ctx, K, order, &s));
    if (ew->pme) {
        cudaStreamSynchronize(ew->ctx->stream);
        pme_destroy(ew->pme);
    }
    ew->pme = s;
    return MD_OK;
}

int md_ewald_set_precision(md_ewald* ew, int precision) {
    graph_epoch_bump();
    if (!ew || (precision != MD_PRECISION_FP64 && precision != MD_PRECISION_MIXED))
        return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_set_precision: MD_PRECISION_FP64 or _MIXED");
    ew->mixed = precision == MD_PRECISION_MIXED;
    return MD_OK;
}

int md_ewald_pme_grid(const md_ewald* ew, int k[3], int* order) {
    if (!ew || !k || !order) return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_pme_grid: NULL");
    if (!ew->pme) {
        k[0] = k[1] = k[2] = 0;
        *order = 0;
        return MD_OK;
    }
    return pme_grid(ew->pme, k, order);
}

int md_ewald_charge_gradient(md_ewald* ew, md_system* sys, double* dedq) {
    if (!ew || !sys || !dedq) return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_charge_gradient: NULL");
    if (ew->pme)
        return fail(MD_ERR_INVALID_ARGUMENT,
                    "md_ewald_charge_gradient: needs the k-vector reciprocal sum (PME is set)");
    if (sys->ctx != ew->ctx)
        return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_charge_gradient: context mismatch");
    const int64_t n = sys->n;
    if (n == 0) return MD_OK;
    md_context* ctx = sys->ctx;
    // energies (also builds the list, topology, k vectors and S(k))
    MDB_TRY(ewald_eval_async(ew, sys, 0, false, false));
    DevBuf buf;
    MDB_TRY(buf.ensure(2 * sizeof(double) * static_cast<size_t>(n)));
    double* dq = buf.as<double>();
    double* dq_o = dq + n;
    const Box3 box{{sys->box[0], sys->box[1], sys->box[2]},
                   {sys->inv_box[0], sys->inv_box[1], sys->inv_box[2]}};
    const RealArgs a = real_args_of(ew, ew->alpha, false);
    md_verlet* v = ew->list;
    const int g = grid_for(n, kBlock);
    k_ewald_dq<<<g, kBlock, 0, ctx->stream>>>(
        sys->cur.pos, sys->cur.charge, sys->cur.mol, v->nbr.as<int>(), v->count.as<int>(),
        v->stride, sys->cur.orig, sys->slot, ew->partner_off.as<int>(), ew->partner_idx.as<int>(),
        n, box, a, dq);
    MDB_TRY(recip_force_async(ew, sys, kargs_of(ew, sys), true, dq));
    k_to_orig1<<<g, kBlock, 0, ctx->stream>>>(sys->cur.orig, n, dq, dq_o);
    ctx->launches += 3;
    MDB_CHECK_LAUNCH();
    MDB_CUDA(cudaMemcpyAsync(dedq, dq_o, sizeof(double) * n, cudaMemcpyDeviceToHost, ctx->stream));
    MDB_CUDA(cudaStreamSynchronize(ctx->stream));
    buf.release();
    return ctx_check_status(ctx);
}

int md_ewald_real_hvp(md_ewald* ew, md_system* sys, const double* u, double* out) {
    if (!ew || !sys || !u || !out) return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_real_hvp: NULL");
    if (sys->ctx != ew->ctx) return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_real_hvp: context mismatch");
    const int64_t n = sys->n;
    if (n == 0) return MD_OK;
    md_context* ctx = sys->ctx;
    MDB_TRY(ewald_eval_async(ew, sys, 0, false, false));  // list and alpha for this state
    DevBuf buf;
    MDB_TRY(buf.ensure(4 * sizeof(double4) * static_cast<size_t>(n)));
    double4* uo = buf.as<double4>();
    double4* ud = uo + n;
    double4* res = uo + 2 * n;
    double4* res_o = uo + 3 * n;
    MDB_TRY(upload_vec(sys, u, uo, ud));
    const Box3 box{{sys->box[0], sys->box[1], sys->box[2]},
                   {sys->inv_box[0], sys->inv_box[1], sys->inv_box[2]}};
    md_verlet* v = ew->list;
    const int g = grid_for(n, kBlock);
    k_ewald_real_hvp<<<g, kBlock, 0, ctx->stream>>>(sys->cur.pos, sys->cur.charge, sys->cur.mol,
                                                   v->nbr.as<int>(), v->count.as<int>(), v->stride,
                                                   n, box, real_args_of(ew, ew->alpha, false), ud,
                                                   res);
    k_to_orig4<<<g, kBlock, 0, ctx->stream>>>(sys->cur.orig, n, res, res_o);
    ctx->launches += 3;
    MDB_CHECK_LAUNCH();
    std::vector<double4> h(static_cast<size_t>(n));
    MDB_CUDA(cudaMemcpyAsync(h.data(), res_o, sizeof(double4) * n, cudaMemcpyDeviceToHost,
                             ctx->stream));
    MDB_CUDA(cudaStreamSynchronize(ctx->stream));
    buf.release();
    for (int64_t o = 0; o < n; ++o) {
        out[3 * o] = h[o].x;
        out[3 * o + 1] = h[o].y;
        out[3 * o + 2] = h[o].z;
    }
    return ctx_check_status(ctx);
}

int md_ewald_alpha(const md_ewald* ew, double* alpha) {
    if (!ew || !alpha) return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_alpha: NULL");
    *alpha = ew->alpha;
    return MD_OK;
}

int md_ewald_kvector_count(const md_ewald* ew, int* count) {
    if (!ew || !count) return fail(MD_ERR_INVALID_ARGUMENT, "md_ewald_kvector_count: NULL");
    *count = 2 * ew->nk;  // the full set is the half space and its negatives
    return MD_OK;
}

// ------------------------------------------------------------------- SPC/E
int md_spce_create(md_context* ctx, double sigma_o, double epsilon_o, double cutoff, int kmax,
                   double alpha, md_ewald** out) {
    graph_epoch_bump();
    MDB_TRY(ewald_new(ctx, cutoff, kmax, alpha, out));
    (*out)->spce = true;
    (*out)->sigma_o = sigma_o;
    (*out)->epsilon_o = epsilon_o;
    return MD_OK;
}

int md_spce_set_lj_truncation(md_ewald* ew, int truncation) {
    graph_epoch_bump();
    if (!ew || !ew->spce || (truncation != MD_TRUNCATED && truncation != MD_LINEAR_FORCE_SHIFT))
        return fail(MD_ERR_INVALID_ARGUMENT, "md_spce_set_lj_truncation: bad argument");
    ew->lj_truncation = truncation;
    return MD_OK;
}

int md_spce_compute(md_ewald* ew, md_system* sys, int forces, double* energy, double parts[8]) {
    if (!ew || !sys || !ew->spce) return fail(MD_ERR_INVALID_ARGUMENT, "md_spce_compute: not an SPC/E force field");
    if (sys->n % 3 != 0)  // spce_forcefield.cpp:14-17
        return fail(MD_ERR_INVALID_ARGUMENT,
                    "SpceForceField: atom count is not a multiple of 3; expected O,H,H triples");
    MDB_TRY(ewald_eval_async(ew, sys, forces ? 1 : 0, false, false));
    MDB_TRY(ewald_read(ew, sys->ctx));
    double terms[4], vir;
    fill_terms(ew, terms, &vir);
    // dispersion tail of the oxygen subsystem (lennard_jones.cpp:121-135 with n = N/3)
    const double m = static_cast<double>(sys->n / 3);
    const double rho = m / (sys->box[0] * sys->box[1] * sys->box[2]);
    const double sr = ew->sigma_o / ew->cutoff;
    const double sr3 = sr * sr * sr, sr9 = sr3 * sr3 * sr3;
    const double sig3 = ew->sigma_o * ew->sigma_o * ew->sigma_o;
    const double elrc = ew->lj_truncation == MD_LINEAR_FORCE_SHIFT
                            ? 0.0
                            : (8.0 / 3.0) * kPi * m * rho * ew->epsilon_o * sig3 *
                                  ((1.0 / 3.0) * sr9 - sr3);
    const double disp = ew->last[kEwLj];
    // spce_forcefield.cpp:40: disp + elrc + total()
    const double total = disp + elrc + (terms[0] + terms[1] + terms[2] + terms[3]);
    if (energy) *energy = total;
    if (parts) {
        parts[0] = disp;
        parts[1] = elrc;
        parts[2] = terms[0];
        parts[3] = terms[1];
        parts[4] = terms[2];
        parts[5] = terms[3];
        parts[6] = vir + ew->last[kEwLjW];  // atomic virial, no reference counterpart
        parts[7] = total;
    }
    sys->last_energy = total;
    return MD_OK;
}

}  // extern "C"
