// direct_fp64.cu -- plain-FP64 direct O(N^2) passes (the reference drop-in).
//
// Every droplet's pair terms are summed over j = 0..n-1 in ascending order,
// exactly like the reference's serial inner loop, with every expression
// evaluated in the reference's order.  This file is compiled with -fmad=false
// so no multiply-add is contracted: each operation rounds once, and the
// results are bit-identical to the CPU restatement of
//   dem/force_calculator/direct_droplet_force_calculator.py:183-253 (forces)
//   dem/force_calculator/direct_droplet_force_calculator.py:354-411 (convection).
//
// Only the additions are serial, not the terms.  A CTA takes R droplets (rows):
// 256 producer threads evaluate the terms of a tile of j's, side by side, into
// shared memory while one adder thread per (row, component) adds the previous
// tile's terms to its running sum in j order (an FP64 addition has 8 cycles of
// latency, so a chain takes ~10 cycles per j) and stages the next tile's j's.
// One thread per droplet, which this replaces, kept a term's whole latency in
// the chain (~430 ns per j and pass) and left most of the chip idle below
// n ~ 60,000.  The terms use square root, reciprocals and quotients without
// branches (ieee64.cuh), so that a thread has several terms in flight, and the
// six quotients of an Oseen term share one reciprocal.
//
// Bound: the FP64 pipe (59 / 86 operations per pair) at large n, the adders'
// chains and the terms' latency at small n.  Force / convection pass, periodic,
// us, before -> now, events around the pass: n = 500 137 / 310 -> 13 / 13; 2,000 527
// / 1,220 -> 34 / 43; 8,000 2,090 / 4,860 -> 328 / 446; 20,011 5,650 / 12,800 -> 1,800
// / 2,520 (FP64 pipe 68 / 74 % of peak; more resident warps, larger tiles or 512
// producers change that by a few per cent either way).  In a graph, without the
// events' ~6 us: 6.8 / 7.3, 29 / 37, 322 / 439, 1,786 / 2,513.
//
// With the periodic-image correction loaded, the convection kernel adds each
// pair's correction term right after its Stokeslet term and the self term
// after the loop (:413-464), bit-identical to the CPU restatement.  Bound: the
// lines of the correction table that the L1 passes per pair, then the FP64
// pipe (~500 operations per pair).  Four lanes take a component each of the
// cells of one pair after another (corr_four), from a table whose half cells
// are a line each: n = 2,000 7,520 -> 232 us, 8,192 30,800 -> 3,030, 16,384
// 62,200 -> 11,700 (one lane per pair: 550, 7,600, 30,300; four lanes over
// cells of 192 bytes side by side: 319, 4,330, 17,000).
#include "common.cuh"
#include "corr.cuh"
#include "ieee64.cuh"
#include <type_traits>

namespace dem {

enum : int { FORCE64 = 0, OSEEN64 = 1, OSEEN64_CORR = 2 };

constexpr int ORD_P = 256;  // producer threads
constexpr int NV = 6;       // doubles staged per j: x, y, z, r^3, r, - (force) or x, y, z, Fx, Fy, Fz

template <int R, int KIND>
struct OrdShape {
    static constexpr int SUBS = ORD_P / R;                       // j's evaluated side by side per row
    static constexpr int U = SUBS > 32 || KIND == OSEEN64_CORR ? 2 : 4;  // terms per producer thread and tile
    static constexpr int TJ = SUBS * U;                          // j's per tile
    static constexpr int ADD_T = (3 * R + 31) / 32 * 32;         // adder threads: one per (row, component)
    static constexpr int THREADS = ORD_P + ADD_T;
    static constexpr int CTAS = KIND == OSEEN64_CORR ? 2 : 3;    // per SM: 64 - 72 registers (the correction: 96)
    static constexpr int PLANES = KIND == OSEEN64_CORR ? 6 : 3;  // terms per pair
    static constexpr int CS = TJ * R + (R < 16 ? R : 0);         // plane stride (narrow rows: offset banks)
    static constexpr int LOADS = (TJ + ADD_T - 1) / ADD_T;       // staged j's per adder thread
    static constexpr size_t SMEM = sizeof(double) * (2 * PLANES * CS + 2 * NV * TJ);
    static_assert(TJ <= ORD_P, "tile 0 is staged by the first TJ threads");
};

struct Ord64Args {
    int n;
    const double *x, *y, *z, *r;
    const double *fx, *fy, *fz;
    double coeff;  // m_const / eta
    double L, halfL;
    CorrDev corr;
    double *ox, *oy, *oz;
};

struct D3 {
    double x, y, z;
};

// a coordinate: zero or 2^-300 <= |v| < 2^90, so that differences of two are zero or >= 2^-352
__device__ __forceinline__ bool coord_ok(double v) { return v == 0.0 || hi_in(fabs(v), hi_of_pow2(-300), hi_of_pow2(90)); }
__device__ __forceinline__ bool factor_ok(double v) { return hi_in(v, hi_of_pow2(-125), hi_of_pow2(125)); }

// Barrier of the CTA's THREADS threads; whether any of them passed a true value.  The producers and the adders
// reach it from different places, which PTX's barrier allows whole warps, and __syncthreads_or, which wants the
// whole CTA at one call, does not.
template <int THREADS>
__device__ __forceinline__ int cta_any(int v) {
    int any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\t"
        "barrier.cta.red.or.aligned.pred q, 1, %2, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
        : "=r"(any)
        : "r"(v), "n"(THREADS)
        : "memory");
    return any;
}

// ---- pair terms -------------------------------------------------------------
template <bool PER>
__device__ __forceinline__ void image3(double &x, double &y, double &z, double L, double halfL) {
    if (PER) {
        image1(x, L, halfL);
        image1(y, L, halfL);
        image1(z, L, halfL);
    }
}

// The force term of a separation, :183-200 (0 inside the contact cut, :246).  PLAIN: every operand;
// else returns false where the branch-free operations do not apply.
template <bool PLAIN>
__device__ __forceinline__ bool force_term64(double dx, double dy, double dz, double mri3, double rj3, double reach,
                                             D3 &t) {
    const double dx2 = dx * dx, dy2 = dy * dy, dz2 = dz * dz;
    const double r2 = dx2 + dy2 + dz2;
    double M, r_mag;
    bool ok = true;
    if (PLAIN) {
        r_mag = sqrt(r2);
        M = mri3 * rj3 / ipow7(r_mag);
    } else {
        double h;
        r_mag = sqrt_rn(r2, h);
        const double r7 = ipow7(r_mag);
        M = quotient_rn(mri3 * rj3, r7, rcp_rn(r7));
        ok = hi_in(r2, hi_of_pow2(-200), hi_of_pow2(200)) && !low_word_ones(r7);
    }
    const bool keep = r_mag > reach;
    if (!PLAIN) M = keep ? M : 0.0;  // finite operands: the terms become zeros
    // 4 dz^2 and 2 dz^2 are exact: one rounding each with the difference that follows
    const double fxy = M * (__fma_rn(4.0, dz2, -dx2) - dy2);
    t.x = fxy * dx;
    t.y = fxy * dy;
    t.z = M * (__fma_rn(2.0, dz2, -(3 * dx2)) - 3 * dy2) * dz;
    if (PLAIN && !keep) t = D3{0.0, 0.0, 0.0};
    return ok;
}

// The Oseen term of a separation, :382-411.
template <bool PLAIN>
__device__ __forceinline__ bool oseen_term64(double X, double Y, double Z, double Fx, double Fy, double Fz,
                                             double eta, D3 &t) {
    const double XX = X * X, YY = Y * Y, ZZ = Z * Z;
    const double r2 = XX + YY + ZZ;
    double inv_r, xx, yy, zz, xy, xz, yz;
    bool ok = true;
    if (PLAIN) {
        const double rr = sqrt(r2);
        const double r3 = ipow3(rr);
        inv_r = 1 / rr;
        xx = XX / r3;
        yy = YY / r3;
        zz = ZZ / r3;
        xy = (X * Y) / r3;
        xz = (X * Z) / r3;
        yz = (Y * Z) / r3;
    } else {
        double h;
        const double rr = sqrt_rn(r2, h);
        const double r3 = ipow3(rr);
        inv_r = rcp_last(rr, rcp_last(rr, times_pow2(h, 1)));
        const double y3 = rcp_rn(r3);
        xx = quotient_rn(XX, r3, y3);
        yy = quotient_rn(YY, r3, y3);
        zz = quotient_rn(ZZ, r3, y3);
        xy = quotient_rn(X * Y, r3, y3);
        xz = quotient_rn(X * Z, r3, y3);
        yz = quotient_rn(Y * Z, r3, y3);
        ok = hi_in(r2, hi_of_pow2(-200), hi_of_pow2(200)) && !low_word_ones(rr) && !low_word_ones(r3);
    }
    t.x = eta * ((inv_r + xx) * Fx + xy * Fy + xz * Fz);
    t.y = eta * (xy * Fx + (inv_r + yy) * Fy + yz * Fz);
    t.z = eta * (xz * Fx + yz * Fy + (inv_r + zz) * Fz);
    return ok;
}

// corr_pair64 from zero for the pairs of four neighbouring lanes, which have their j in common: lane o takes
// component o of each lane's pair in turn (the last lane o = 2 again, unwritten), so that the four read
// from one line.  Two pairs in flight: 4 unrolled are 15 % slower, one 7 %.  Written to out[q] (component 0 of lane q's pair), its planes `cs` apart.
__device__ __forceinline__ void corr_four(const CorrDev &c, double X, double Y, double Z, double Fx, double Fy,
                                          double Fz, double *out, int cs) {
    const int lane4 = threadIdx.x & 3, o = min(lane4, 2);
    int ax, ay, az;
    double tx, ty, tz;
    corr_axis64(X * c.cL, c.gmin, c.ginv, c.n, ax, tx);
    corr_axis64(Y * c.cL, c.gmin, c.ginv, c.n, ay, ty);
    corr_axis64(Z * c.cL, c.gmin, c.ginv, c.n, az, tz);
    const int m = c.n - 1;
    const int cell1 = (ax * m + ay) * m + az, cell2 = (az * m + ay) * m + ax, cell3 = (ax * m + az) * m + ay;
    const double sx = Fx * c.common, sy = Fy * c.common, sz = Fz * c.common;
    const double2 *const b1 = c.c64 + 2 * o, *const b2 = c.c64 + 2 * (2 - o), *const b3 = c.c64 + 2 * ((3 - o) % 3);
#pragma unroll 2
    for (int q = 0; q < 4; ++q) {
        const double t1 = __shfl_sync(0xffffffffu, tx, q, 4), t2 = __shfl_sync(0xffffffffu, ty, q, 4),
                     t3 = __shfl_sync(0xffffffffu, tz, q, 4);
        double g1[8], g2[8], g3[8];
        corr_ld8(b1 + CORR_CELL64 * (size_t)__shfl_sync(0xffffffffu, cell1, q, 4), g1);
        corr_ld8(b2 + CORR_CELL64 * (size_t)__shfl_sync(0xffffffffu, cell2, q, 4), g2);
        corr_ld8(b3 + CORR_CELL64 * (size_t)__shfl_sync(0xffffffffu, cell3, q, 4), g3);
        const double gz = corr_interp64(g1, t1, t2, t3), gx = corr_interp64(g2, t3, t2, t1),
                     gy = corr_interp64(g3, t1, t3, t2);
        if (lane4 < 3) out[o * cs + q] = 0.0 + (gx * sx + gy * sy + gz * sz);
    }
}

template <int R, bool PER, int KIND>
__global__ void __launch_bounds__(OrdShape<R, KIND>::THREADS, OrdShape<R, KIND>::CTAS) ordered_pass_kernel(const Ord64Args a) {
    using S = OrdShape<R, KIND>;
    extern __shared__ __align__(16) double ord_smem[];
    double *const stage = ord_smem;                 // [2][TJ][NV]
    double *const terms = ord_smem + 2 * NV * S::TJ;  // [2][PLANES][CS]: the term of (j, row) at j * R + row
    const int tid = threadIdx.x;
    const int n = a.n;
    const int row0 = blockIdx.x * R;
    const int ntiles = (n + S::TJ - 1) / S::TJ;

    const double *const src[NV] = {a.x, a.y, a.z, KIND == FORCE64 ? a.r : a.fx, a.fy, a.fz};
    constexpr int NSRC = KIND == FORCE64 ? 4 : 6;
    // Writes droplet j's values to its stage slot (NaN past the end: no fast term); whether it is fit for
    // the branch-free operations.
    auto put = [&](double *slot, double (&v)[NSRC], bool in) {
        if (!in) v[0] = __longlong_as_double(0x7ff8000000000000ll);
        double w3 = v[3], w4 = KIND == FORCE64 ? v[3] : v[NSRC - 2];
        if (KIND == FORCE64) w3 = ipow3(w4);
        slot[0] = v[0], slot[1] = v[1], slot[2] = v[2];
        slot[3] = w3, slot[4] = w4;
        if (KIND != FORCE64) slot[5] = v[NSRC - 1];
        return coord_ok(v[0]) && coord_ok(v[1]) && coord_ok(v[2]) && (KIND != FORCE64 || factor_ok(w3));
    };
    int odd = 0;
    if (tid < S::TJ) {
        double v[NSRC];
#pragma unroll
        for (int w = 0; w < NSRC; ++w) v[w] = tid < n ? src[w][tid] : 0.0;
        odd = !put(stage + NV * tid, v, tid < n) && tid < n;
    }
    odd = __syncthreads_or(odd);

    if (tid < ORD_P) {
        const int row = tid % R, sub = tid / R;
        const int i = row0 + row;
        const int ii = min(i, n - 1);
        const double xi = a.x[ii], yi = a.y[ii], zi = a.z[ii];
        double ri = 0.0, mri3 = 0.0;
        if (KIND == FORCE64) {
            ri = a.r[ii];
            mri3 = a.coeff * ipow3(ri);  // (m_const * r_i**3) is the first product of :189
        }
        const bool row_ok = coord_ok(xi) && coord_ok(yi) && coord_ok(zi) && (KIND != FORCE64 || factor_ok(mri3)) &&
                            (!PER || hi_in(a.L, hi_of_pow2(-300), hi_of_pow2(90)));
        for (int t = 0; t <= ntiles; ++t) {
            if (t < ntiles) {
                const double *const s = stage + (t & 1) * NV * S::TJ + NV * sub;
                double *const o = terms + (t & 1) * S::PLANES * S::CS + sub * R + row;
                // The term of the thread's u-th j, written to its slots; false: the operands need the
                // operators (PLAIN).
                auto term = [&](int u, auto plain) {
                    const double2 *const q = reinterpret_cast<const double2 *>(s + u * S::SUBS * NV);
                    const double2 p0 = q[0], p1 = q[1], p2 = q[2];  // (x, y), (z, r^3 | Fx), (r | Fy, Fz)
                    double *const w = o + u * S::SUBS * R;
                    D3 v;
                    bool ok;
                    double X, Y, Z;
                    if (KIND == FORCE64) {
                        X = p0.x - xi, Y = p0.y - yi, Z = p1.x - zi;
                        image3<PER>(X, Y, Z, a.L, a.halfL);
                        ok = force_term64<decltype(plain)::value>(X, Y, Z, mri3, p1.y, ri + p2.x, v);
                    } else {
                        X = xi - p0.x, Y = yi - p0.y, Z = zi - p1.x;
                        image3<PER>(X, Y, Z, a.L, a.halfL);
                        ok = oseen_term64<decltype(plain)::value>(X, Y, Z, p1.y, p2.x, p2.y, a.coeff, v);
                    }
                    w[0] = v.x;
                    w[S::CS] = v.y;
                    w[2 * S::CS] = v.z;
                    if (KIND == OSEEN64_CORR && !decltype(plain)::value)
                        corr_four(a.corr, X, Y, Z, p1.y, p2.x, p2.y, w - (tid & 3) + 3 * S::CS, S::CS);
                    return ok;
                };
                unsigned redo = row_ok && !odd ? 0u : (1u << S::U) - 1u;
#pragma unroll
                for (int u = 0; u < S::U; ++u) redo |= term(u, std::false_type{}) ? 0u : 1u << u;
                if (KIND == OSEEN64_CORR) __syncwarp();  // the corrections are neighbours' writes
                while (redo) {
                    const int u = __ffs(redo) - 1;
                    redo &= redo - 1;
                    const int j = t * S::TJ + sub + u * S::SUBS;
                    if (j < n && j != i) {
                        term(u, std::true_type{});
                    } else {  // no term: adding +0 leaves a running sum as it is
#pragma unroll
                        for (int p = 0; p < S::PLANES; ++p) o[u * S::SUBS * R + p * S::CS] = 0.0;
                    }
                }
            }
            odd = cta_any<S::THREADS>(0);
        }
    } else {
        const int q = tid - ORD_P;
        const int comp = q / R, row = q % R;
        const bool chain = comp < 3;
        double acc = 0.0;
        for (int t = 0; t <= ntiles; ++t) {
            // tile t + 1: the loads are issued before the sums of tile t - 1, used after them
            const int j0 = (t + 1) * S::TJ;
            double v[S::LOADS][NSRC];
            if (t + 1 < ntiles) {
#pragma unroll
                for (int l = 0; l < S::LOADS; ++l) {
                    const int k = q + l * S::ADD_T, j = j0 + k;
#pragma unroll
                    for (int w = 0; w < NSRC; ++w) v[l][w] = k < S::TJ && j < n ? src[w][j] : 0.0;
                }
            }
            if (t > 0 && chain) {
                const double *p = terms + ((t - 1) & 1) * S::PLANES * S::CS + comp * S::CS + row;
#pragma unroll 16
                for (int k = 0; k < S::TJ; ++k) {
                    acc += p[k * R];
                    if (KIND == OSEEN64_CORR) acc += p[3 * S::CS + k * R];
                }
            }
            odd = 0;
            if (t + 1 < ntiles) {
                double *const s = stage + ((t + 1) & 1) * NV * S::TJ;
#pragma unroll
                for (int l = 0; l < S::LOADS; ++l) {
                    const int k = q + l * S::ADD_T;
                    if (k < S::TJ) odd |= !put(s + NV * k, v[l], j0 + k < n) && j0 + k < n;
                }
            }
            cta_any<S::THREADS>(odd);
        }
        const int i = row0 + row;
        if (chain && i < n) {
            if (KIND == OSEEN64_CORR) acc += a.corr.g_self * (comp == 0 ? a.fx : comp == 1 ? a.fy : a.fz)[i];
            (comp == 0 ? a.ox : comp == 1 ? a.oy : a.oz)[i] = acc;
        }
    }
}

// Launches the pass; a shape that wants more than 48 KB of shared memory (8 rows and more, or the correction) has
// its kernel's limit raised by the context's first call that takes it.  (Raised for all of them when a context was
// created, the driver loaded 18 kernels: 1.6 ms of a process's first context.)
template <int R, bool PER, int KIND>
static int launch_ordered(dem_ctx *ctx, const Ord64Args &a, cudaStream_t s) {
    using S = OrdShape<R, KIND>;
    constexpr unsigned bit = 1u << ((R == 4 ? 0 : R == 8 ? 1 : 2) + 3 * (KIND + 3 * PER));
    if (S::SMEM > 48 * 1024 && !(ctx->ord_smem_set & bit)) {
        const int rc = dem_check_cuda(ctx, cudaFuncSetAttribute(ordered_pass_kernel<R, PER, KIND>,
                                                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM),
                                      "direct_fp64 attributes");
        if (rc) return rc;
        ctx->ord_smem_set |= bit;
    }
    ordered_pass_kernel<R, PER, KIND><<<ceil_div(a.n, R), S::THREADS, S::SMEM, counted(s)>>>(a);
    return DEM_OK;
}

// Rows per CTA.  Few rows per CTA spread a small box over the SMs (one wave: 3 CTAs of 4 rows per SM hold
// 12 n_SM = 1,776 rows); more rows per CTA use the adders' lanes fully.  Force + convection, periodic, us,
// with 4 / 8 / 16 rows: n = 500: 26 / 31 / 36; 1,776: 66 / 69 / 77; 2,500: 140 / 126 / 149; 10,000: 1,516 /
// 1,215 / 1,240; 13,000: 2,526 / 1,891 / 1,921; 16,000: 3,871 / 2,910 / 2,716; 30,000: 12,998 / 9,951 / 9,246
// (32 rows are slower throughout).  With the correction, bound by its gathers, 4 and 8 rows are as fast
// as 16 or faster from n = 4,097 to 16,384.
template <bool PER, int KIND>
static int run_rows(dem_ctx *ctx, const Ord64Args &a, cudaStream_t s) {
    const int sm = ctx->sm_count;
    if (a.n <= 12 * sm) return launch_ordered<4, PER, KIND>(ctx, a, s);
    if constexpr (KIND != OSEEN64_CORR)
        if (a.n > 95 * sm) return launch_ordered<16, PER, KIND>(ctx, a, s);
    return launch_ordered<8, PER, KIND>(ctx, a, s);
}

template <int KIND>
static int run_ordered(dem_ctx *ctx, const char *name, const Ord64Args &a, int periodic, cudaStream_t s) {
    dem_prof_begin(ctx, name, s);
    const int rc = periodic ? run_rows<true, KIND>(ctx, a, s) : run_rows<false, KIND>(ctx, a, s);
    dem_prof_end(ctx, s);
    return rc ? rc : dem_check_launch(ctx, name);
}

int launch_direct_forces_fp64(dem_ctx *ctx, int n, const double *x, const double *y, const double *z,
                              const double *r, double m_const, double L, int periodic, double *fx, double *fy,
                              double *fz, cudaStream_t s) {
    const Ord64Args a{n, x, y, z, r, nullptr, nullptr, nullptr, m_const, L, L * 0.5, CorrDev{}, fx, fy, fz};
    return run_ordered<FORCE64>(ctx, "fp64_force_pass", a, periodic, s);
}

int launch_direct_convection_fp64(dem_ctx *ctx, int n, const double *x, const double *y, const double *z,
                                  const double *fx, const double *fy, const double *fz, double eta, double L,
                                  int periodic, double *vx, double *vy, double *vz, cudaStream_t s) {
    const Ord64Args a{n, x, y, z, nullptr, fx, fy, fz, eta, L, L * 0.5, CorrDev{}, vx, vy, vz};
    return run_ordered<OSEEN64>(ctx, "fp64_convection_pass", a, periodic, s);
}

int launch_direct_convection_fp64_corr(dem_ctx *ctx, const dem_corr *c, int n, const double *x, const double *y,
                                       const double *z, const double *fx, const double *fy, const double *fz,
                                       double eta, double L, int periodic, double *vx, double *vy, double *vz,
                                       cudaStream_t s) {
    const Ord64Args a{n, x, y, z, nullptr, fx, fy, fz, eta, L, L * 0.5, corr_view(c), vx, vy, vz};
    return run_ordered<OSEEN64_CORR>(ctx, "fp64_convection_corr_pass", a, periodic, s);
}

// The operations of ieee64.cuh by themselves, as the terms use them.
__global__ void ieee64_probe_kernel(int n, const double *__restrict__ a, const double *__restrict__ b,
                                    double *__restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double h;
        const double g = sqrt_rn(a[i], h), y = rcp_rn(b[i]);
        out[i] = g;
        out[(size_t)n + i] = rcp_last(g, rcp_last(g, times_pow2(h, 1)));
        out[2 * (size_t)n + i] = y;
        out[3 * (size_t)n + i] = quotient_rn(a[i], b[i], y);
    }
}

}  // namespace dem

extern "C" int dem_ieee64_probe(dem_ctx *ctx, int n, const double *a, const double *b, double *out, void *stream) {
    if (!ctx) return DEM_E_INVALID;
    if (n < 0 || (n > 0 && (!a || !b || !out))) return dem_set_error(ctx, DEM_E_INVALID, "ieee64 probe arguments");
    if (n == 0) return DEM_OK;
    const int grid = min(ceil_div(n, 256), 8 * ctx->sm_count);
    dem::ieee64_probe_kernel<<<grid, 256, 0, counted((cudaStream_t)stream)>>>(n, a, b, out);
    return dem_check_launch(ctx, "ieee64 probe");
}
