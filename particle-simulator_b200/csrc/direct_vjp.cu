// direct_vjp.cu -- adjoint (vector-Jacobian product) of the direct step velocity.
//
// The direct path moves droplet i with (euler_droplet_solver.py:121-125)
//   u_i = F_i / (gamma r_i) + V_i,
//   F_i = m r_i^3 sum_j r_j^3 f(d_ij),  d_ij = mic(x_j - x_i),  cut |d| > r_i + r_j
//         (direct_droplet_force_calculator.py:183-253),
//   V_i = eta sum_{j != i} G(e_ij) F_j,  e_ij = mic(x_i - x_j) = -d_ij,
//         G(e) = I / |e| + e e^T / |e|^3  (:354-411),
// with m = 12 pi eps0 eps_oil E^2.  Given a cotangent lambda on u this file
// computes lambda^T du/dx, lambda^T du/dr (collision cut and periodic wrap
// treated as non-differentiable); lambda^T du/dE = 2 lambda.u / E needs no kernel.
//
// Derivation used by the kernels:
//   * f(d) = P(d) / |d|^7 = grad(phi) / 3 with phi(d) = (|d|^2 - 3 dz^2) / |d|^5,
//     so df/dd = H(d) / 3 with H the (symmetric) Hessian of phi:
//       H = (-3 r^-5 + 15 dz^2 r^-7) I + (15 r^-7 - 105 dz^2 r^-9) d d^T
//           - 6 r^-5 z z^T + 30 dz r^-7 (z d^T + d z^T);
//   * the cotangent reaching the forces is
//       mu_i = lambda_i / (gamma r_i) + eta sum_{j != i} G(x_i - x_j) lambda_j
//     (G is even and symmetric: the Oseen pass applied to lambda);
//   * d(sum_k mu_k.F_k)/dx_i = (m/3) r_i^3 sum_j r_j^3 H(d_ij) (mu_j - mu_i),
//     d(sum_k mu_k.F_k)/dr_i = -3 m r_i^2 sum_j r_j^3 (mu_j - mu_i).f(d_ij);
//   * d(sum_k lambda_k.V_k)/dx_i = eta sum_{j != i} [K(e_ij; lambda_i, F_j) + K(e_ij; lambda_j, F_i)],
//       K(e; a, b) = grad_e(a^T G(e) b) = [(e.b) a + (e.a) b - (a.b) e] / |e|^3 - 3 (a.e)(e.b) e / |e|^5;
//   * d(lambda_i.F_i / (gamma r_i))/dr_i = -lambda_i.F_i / (gamma r_i^2).
// Everything is FP64.  Both O(N^2) passes evaluate every unordered pair once: G is
// even, and a pair's gradient
//   g = (m/3) r_i^3 r_j^3 H(d) (mu_j - mu_i) - eta [K(d; lambda_i, F_j) + K(d; lambda_j, F_i)]
// enters x_i with + and x_j with -, its S = (mu_j - mu_i).f(d) enters r_i as r_j^3 S
// and r_j as r_i^3 S.  With q = dz^2 / r^2, n = mu_j - mu_i, p = d.n / r^2:
//   H n   = r^-5 [(15 q - 3) n + ((15 - 105 q) p + 30 dz nz / r^2) d + (30 dz p - 6 nz) z],
//   n.f   = r^-5 [(5 q - 1) d.n - 2 dz nz];
// with the unit vector e = d / r the powers of r gather in two factors, and the z
// terms join the coefficients of n and e:
//   r^5 (H n)_xy = (15 q - 3) n + a e,  r^5 (H n)_z = (15 q - 9) nz + (a + 30 e.n) ez,
//   a = (15 - 105 q) e.n + 30 ez nz,    r^4 n.f = (5 q - 1) e.n - 2 ez nz.
#include <cmath>

#include "common.cuh"
#include "ieee64.cuh"

namespace dem {

// ---------------------------------------------------------------------------
// Block pairs.  A CTA of W warps takes a pair of blocks (I <= J) of B = 32 W IPT
// droplets.  A lane keeps IPT droplets of I in registers; a warp goes through
// block J 32 droplets at a time, lane l meeting droplet (l + s) mod 32 in step
// s, and the j-side sums travel with their droplet (one shuffle per step), so
// both sides of a pair are added without atomics.  The warps' j-side sums meet
// in shared memory in warp order; every block pair leaves one record per side,
// and the sum kernel adds a droplet's records in block order
// (deterministic).  A diagonal pair (I == J) meets every ordered pair and keeps
// its i side.
//
// Bound: the FP64 pipe, ~102 operations per unordered pair, ~39 in the mu pass
// (before: one thread per droplet and j chunk, every ordered pair); its three-
// operand instructions issue at 75 % of its nominal rate, 67 % in the mu pass.
// Mu / pair pass with their sums, periodic, us, before -> now: n = 2,000 40 / 85 ->
// 30 / 44; 16,384 970 / 3,050 -> 444 / 1,034.
// ---------------------------------------------------------------------------
struct VjpBlocks {
    int nb;           // blocks
    int row0;         // first block row of this launch
    long long item0;  // block pairs before it
};

__host__ __device__ __forceinline__ long long pairs_before(int nb, int row) {
    return (long long)row * nb - (long long)row * (row - 1) / 2;
}

__device__ __forceinline__ void block_pair(const VjpBlocks &b, int &I, int &J) {
    const long long t = b.item0 + blockIdx.x;
    const double h = b.nb + 0.5;
    int i = (int)(h - sqrt(fmax(h * h - 2.0 * (double)t, 0.0)));
    i = max(b.row0, min(i, b.nb - 1));
    while (i > b.row0 && pairs_before(b.nb, i) > t) --i;
    while (i + 1 < b.nb && pairs_before(b.nb, i + 1) <= t) ++i;
    I = i;
    J = i + (int)(t - pairs_before(b.nb, i));
}

template <bool PER>
__device__ __forceinline__ double image64(double d, double L, double halfL) {
    if (PER) image1(d, L, halfL);
    return d;
}

// 1 / sqrt(x) to ~1 ulp: seed y (2^-20), e = 1 - x y^2 and y (1 + e / 2 + 3/8 e^2).  x below infinity.
__device__ __forceinline__ double rsqrt64(double x) {
    const double y = rsqrt_seed(x);
    const double e = fma(-(x * y), y, 1.0);
    return fma(y, fma(0.375, e, 0.5) * e, y);
}

__device__ __forceinline__ double from_next_lane(double v, int lane) {
    return __shfl_sync(0xffffffffu, v, (lane + 1) & 31);
}

// mu pass: u_i = sum_j G(d_ij) lambda_j.  Records: [item][side][3][B].
template <int W, int IPT, bool PER>
__global__ void __launch_bounds__(32 * W) vjp_oseen_kernel(int n, const double *__restrict__ x,
                                                           const double *__restrict__ y, const double *__restrict__ z,
                                                           const double *__restrict__ lx,
                                                           const double *__restrict__ ly,
                                                           const double *__restrict__ lz, double L, double halfL,
                                                           VjpBlocks blocks, double *__restrict__ records) {
    constexpr int B = 32 * W * IPT;
    __shared__ double sj[W][6][32];
    __shared__ double plane[W][3][B];
    int I, J;
    block_pair(blocks, I, J);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double *const src[6] = {x, y, z, lx, ly, lz};
    double xi[IPT], yi[IPT], zi[IPT], ax[IPT], ay[IPT], az[IPT], ux[IPT], uy[IPT], uz[IPT];
    int ii[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int i = I * B + (warp * IPT + k) * 32 + lane;
        ii[k] = i < n ? i : -1;
        xi[k] = i < n ? x[i] : 0.0, yi[k] = i < n ? y[i] : 0.0, zi[k] = i < n ? z[i] : 0.0;
        ax[k] = i < n ? lx[i] : 0.0, ay[k] = i < n ? ly[i] : 0.0, az[k] = i < n ? lz[i] : 0.0;
        ux[k] = uy[k] = uz[k] = 0.0;
    }
    for (int t = 0; t < B / 32; ++t) {
        const int jb = J * B + 32 * t;
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 6; ++c) sj[warp][c][lane] = jb + lane < n ? src[c][jb + lane] : 0.0;
        __syncwarp();
        double vx = 0.0, vy = 0.0, vz = 0.0;
        for (int s = 0; s < 32; ++s) {
            const int jl = (lane + s) & 31, j = jb + jl;
            const double *const q = &sj[warp][0][jl];
            const double xj = q[0], yj = q[32], zj = q[64], bx = q[96], by = q[128], bz = q[160];
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                const double dx = image64<PER>(xj - xi[k], L, halfL), dy = image64<PER>(yj - yi[k], L, halfL),
                             dz = image64<PER>(zj - zi[k], L, halfL);
                const double r2 = dx * dx + dy * dy + dz * dz;
                const double ir = j < n && ii[k] >= 0 && ii[k] != j ? rsqrt64(r2) : 0.0, ir3 = ir * ir * ir;
                const double cj = (dx * bx + dy * by + dz * bz) * ir3;
                const double ci = (dx * ax[k] + dy * ay[k] + dz * az[k]) * ir3;
                ux[k] = fma(bx, ir, fma(dx, cj, ux[k]));
                uy[k] = fma(by, ir, fma(dy, cj, uy[k]));
                uz[k] = fma(bz, ir, fma(dz, cj, uz[k]));
                vx = fma(ax[k], ir, fma(dx, ci, vx));
                vy = fma(ay[k], ir, fma(dy, ci, vy));
                vz = fma(az[k], ir, fma(dz, ci, vz));
            }
            vx = from_next_lane(vx, lane);
            vy = from_next_lane(vy, lane);
            vz = from_next_lane(vz, lane);
        }
        plane[warp][0][32 * t + lane] = vx;
        plane[warp][1][32 * t + lane] = vy;
        plane[warp][2][32 * t + lane] = vz;
    }
    double *const o = records + (size_t)blockIdx.x * 6 * B;
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int p = (warp * IPT + k) * 32 + lane;
        o[p] = ux[k];
        o[B + p] = uy[k];
        o[2 * B + p] = uz[k];
    }
    if (I == J) return;
    __syncthreads();
    for (int p = threadIdx.x; p < 3 * B; p += 32 * W) {
        const int c = p / B, k = p % B;
        double v = plane[0][c][k];
#pragma unroll
        for (int w = 1; w < W; ++w) v += plane[w][c][k];
        o[3 * B + p] = v;
    }
}

struct VjpArgs {
    int n;
    const double *x, *y, *z, *r;
    const double *fx, *fy, *fz;  // forces at this state
    const double *lx, *ly, *lz;  // lambda: cotangent on u
    double *mx, *my, *mz;        // mu: cotangent on F
    double m_const, eta, stokes, L, halfL;
    double *gx, *gy, *gz, *gr;
};

// Pair terms.  Records: [item][side][4][B]: the gradient's three components (i side +, j side - g) and
// sum of r_other^3 S.
template <int W, int IPT, bool PER>
__global__ void __launch_bounds__(32 * W) vjp_pair_kernel(const VjpArgs a, VjpBlocks blocks,
                                                          double *__restrict__ records) {
    constexpr int B = 32 * W * IPT;
    __shared__ double sj[W][14][32];
    __shared__ double plane[W][4][B];
    int I, J;
    block_pair(blocks, I, J);
    const int n = a.n;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double *const src[13] = {a.x, a.y, a.z, a.r, a.mx, a.my, a.mz, a.lx, a.ly, a.lz, a.fx, a.fy, a.fz};
    double v[IPT][13], wi[IPT];
    double gx[IPT], gy[IPT], gz[IPT], gs[IPT];
    int ii[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int i = I * B + (warp * IPT + k) * 32 + lane;
        ii[k] = i < n ? i : -1;
#pragma unroll
        for (int c = 0; c < 13; ++c) v[k][c] = i < n ? src[c][i] : 0.0;
        wi[k] = ipow3(v[k][3]);
        gx[k] = gy[k] = gz[k] = gs[k] = 0.0;
    }
    const double m3 = a.m_const / 3.0;
    for (int t = 0; t < B / 32; ++t) {
        const int jb = J * B + 32 * t;
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 13; ++c) sj[warp][c][lane] = jb + lane < n ? src[c][jb + lane] : 0.0;
        sj[warp][13][lane] = jb + lane < n ? ipow3(a.r[jb + lane]) : 0.0;
        __syncwarp();
        double hx = 0.0, hy = 0.0, hz = 0.0, hs = 0.0;  // droplet j's side: - sum g, sum r_i^3 S
        for (int s = 0; s < 32; ++s) {
            const int jl = (lane + s) & 31, j = jb + jl;
            const double *const q = &sj[warp][0][jl];
            const double wj = q[13 * 32];
            const double ljx = q[7 * 32], ljy = q[8 * 32], ljz = q[9 * 32];
            const double fjx = q[10 * 32], fjy = q[11 * 32], fjz = q[12 * 32];
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                const double lix = v[k][7], liy = v[k][8], liz = v[k][9], fix = v[k][10], fiy = v[k][11], fiz = v[k][12];
                const double dx = image64<PER>(q[0] - v[k][0], a.L, a.halfL),
                             dy = image64<PER>(q[32] - v[k][1], a.L, a.halfL),
                             dz = image64<PER>(q[64] - v[k][2], a.L, a.halfL);
                const double r2 = dx * dx + dy * dy + dz * dz;
                const double ir = j < n && ii[k] >= 0 && ii[k] != j ? rsqrt64(r2) : 0.0;
                const double ex = dx * ir, ey = dy * ir, ez = dz * ir, ir2 = ir * ir;
                // force terms, inside the contact cut of the forward pass (|d| = r2 / |d|) none
                const double c4 = r2 * ir > v[k][3] + q[3 * 32] ? ir2 * ir2 : 0.0;
                const double nx = q[4 * 32] - v[k][4], ny = q[5 * 32] - v[k][5], nz = q[6 * 32] - v[k][6];
                const double en = ex * nx + ey * ny + ez * nz, qz = ez * ez, t = ez * nz;
                const double a1 = fma(30.0, t, fma(-105.0, qz, 15.0) * en);
                const double S = c4 * fma(-2.0, t, fma(5.0, qz, -1.0) * en);
                const double wf = (m3 * wi[k]) * wj * (c4 * ir);
                // Oseen terms
                const double dl = ex * lix + ey * liy + ez * liz, ef = ex * fjx + ey * fjy + ez * fjz;
                const double el = ex * ljx + ey * ljy + ez * ljz, df = ex * fix + ey * fiy + ez * fiz;
                const double ab = lix * fjx + liy * fjy + liz * fjz + ljx * fix + ljy * fiy + ljz * fiz;
                const double kf = -a.eta * ir2;
                const double kd = kf * fma(-3.0, fma(dl, ef, el * df), -ab);
                const double kdl = kf * dl, kef = kf * ef, kel = kf * el, kdf = kf * df;
                // along n, along e, and the z components of both
                const double wn = wf * fma(15.0, qz, -3.0), we = fma(wf, a1, kd);
                const double wnz = wf * fma(15.0, qz, -9.0), wez = fma(wf, fma(30.0, en, a1), kd);
                const double tx = fma(wn, nx, fma(we, ex, fma(kef, lix, fma(kdl, fjx, fma(kdf, ljx, kel * fix)))));
                const double ty = fma(wn, ny, fma(we, ey, fma(kef, liy, fma(kdl, fjy, fma(kdf, ljy, kel * fiy)))));
                const double tz = fma(wnz, nz, fma(wez, ez, fma(kef, liz, fma(kdl, fjz, fma(kdf, ljz, kel * fiz)))));
                gx[k] += tx;
                gy[k] += ty;
                gz[k] += tz;
                gs[k] = fma(wj, S, gs[k]);
                hx -= tx;
                hy -= ty;
                hz -= tz;
                hs = fma(wi[k], S, hs);
            }
            hx = from_next_lane(hx, lane);
            hy = from_next_lane(hy, lane);
            hz = from_next_lane(hz, lane);
            hs = from_next_lane(hs, lane);
        }
        plane[warp][0][32 * t + lane] = hx;
        plane[warp][1][32 * t + lane] = hy;
        plane[warp][2][32 * t + lane] = hz;
        plane[warp][3][32 * t + lane] = hs;
    }
    double *const o = records + (size_t)blockIdx.x * 8 * B;
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int p = (warp * IPT + k) * 32 + lane;
        o[p] = gx[k];
        o[B + p] = gy[k];
        o[2 * B + p] = gz[k];
        o[3 * B + p] = gs[k];
    }
    if (I == J) return;
    __syncthreads();
    for (int p = threadIdx.x; p < 4 * B; p += 32 * W) {
        const int c = p / B, k = p % B;
        double w = plane[0][c][k];
#pragma unroll
        for (int ww = 1; ww < W; ++ww) w += plane[ww][c][k];
        o[4 * B + p] = w;
    }
}

// What the block pairs read for the droplets' own arrays: finite coordinates no farther out than that a squared
// distance stays finite (the terms of a pair so far apart are below 2^-500 of any other's), and radii whose cube does:
// the zero factor of a cut pair must not meet an infinity.
__global__ void vjp_admit_kernel(const VjpArgs a, double *__restrict__ adm) {
    const int n = a.n;
    const double *const src[3] = {a.x, a.y, a.z};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double v = src[c][i];
            adm[c * (size_t)n + i] = fabs(v) < INFINITY ? fmin(fmax(v, -0x1p510), 0x1p510) : v;
        }
        adm[3 * (size_t)n + i] = fmin(a.r[i], 0x1p341);
    }
}

// sums[c][i] (+)= droplet i's records of block rows [row0, row1), in block order; the last rows' launch writes the
// results: mu_i = eta sum_i + lambda_i / (gamma r_i), for the pair pass in mu_pairs (zeros where r_i is zero, whose
// weight r_i^3 outdoes the quotient, or not a number, which cuts every pair), or the gradients.
template <int NC>
__global__ void vjp_sum_kernel(const VjpArgs a, int B, int nb, int row0, int row1, const double *__restrict__ records,
                               double *__restrict__ sums, double *__restrict__ mu_pairs) {
    const int n = a.n;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)NC * n) return;
    const int c = (int)(t / n), i = (int)(t % n), b = i / B, k = i % B;
    double v = row0 ? sums[t] : 0.0;
    // 16 loads in flight, added in order
    auto add = [&](long long item, int I, int end, int step, int less, int side) {
        const size_t stride = (size_t)2 * NC * B;
        const double *p = records + (size_t)item * stride + (size_t)(side * NC + c) * B + k;
        for (; I < end; I += 16) {
            double w[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                w[q] = I + q < end ? *p : 0.0;
                if (I + q + 1 < end) p += (size_t)(step - less * (I + q)) * stride;
            }
#pragma unroll
            for (int q = 0; q < 16; ++q)
                if (I + q < end) v += w[q];
        }
    };
    add(b - row0, row0, min(b, row1), nb - 1, 1, 1);  // j side of (I, b): the next row's item is nb - I - 1 further
    if (b >= row0 && b < row1) add(pairs_before(nb, b) - pairs_before(nb, row0), b, nb, 1, 0, 0);  // i side of (b, J)
    if (row1 < nb) {
        sums[t] = v;
        return;
    }
    const double ri = a.r[i];
    if (NC == 3) {
        const double w = 1.0 / (a.stokes * ri);
        const double mu = a.eta * v + w * (c == 0 ? a.lx : c == 1 ? a.ly : a.lz)[i];
        (c == 0 ? a.mx : c == 1 ? a.my : a.mz)[i] = mu;
        mu_pairs[t] = fabs(w) < INFINITY ? mu : 0.0;
    } else if (c < 3) {
        (c == 0 ? a.gx : c == 1 ? a.gy : a.gz)[i] = v;
    } else {
        const double lf = a.lx[i] * a.fx[i] + a.ly[i] * a.fy[i] + a.lz[i] * a.fz[i];
        a.gr[i] = -3.0 * a.m_const * ri * ri * v - lf / (a.stokes * ri * ri);
    }
}

constexpr int VJP_OWN = 11;  // workspace doubles per droplet: sums (4), admitted x, y, z, r, and mu

struct VjpShape {
    int warps, ipt, B, nb;
    int rows;      // block rows per launch
    size_t bytes;  // records of one launch, the sums and what the pairs read
};

static size_t record_bytes(const VjpShape &s) {
    return (size_t)pairs_before(s.nb, s.rows) * sizeof(double) * 8 * s.B;
}

// Block rows per launch whose records stay below `budget` (at least one).
static void fit_rows(VjpShape &s, int n, size_t budget) {
    s.rows = s.nb;
    while (s.rows > 1 && record_bytes(s) > budget) s.rows = (s.rows + 1) / 2;
    s.bytes = record_bytes(s) + sizeof(double) * VJP_OWN * n;
}

// Records of a launch stay below this; a larger n goes through its block rows in several launches.
constexpr size_t VJP_RECORD_BYTES = size_t(2) << 30;

// Blocks of 32 droplets fill the SMs with a small box's block pairs, blocks of 64 (two droplets per lane
// share the loads and shuffles) are faster from n ~ 2,000 on, and two such warps on a block of 128, with
// half the records and reads per pair, once its larger grains leave no last wave.  Both passes, periodic,
// us, with 32 / 64 / 128: n = 1,000: 45 / 64 / -; 2,000: 73 / 68 / 102; 8,192: - / 407 / 449; 10,000: - / 603 /
// 609; 11,000: - / 734 / 714; 16,384: 1,792 / 1,529 / 1,470; 40,000: - / 8,689 / 8,578; 65,536: - / 23,247 /
// 22,738 (four warps of one droplet per lane 9,268 and 24,636, four of two 8,698 and 22,985).
static VjpShape vjp_shape(int n) {
    VjpShape s;
    s.warps = n > 10500 ? 2 : 1;
    s.ipt = n >= 2000 ? 2 : 1;
    s.B = 32 * s.warps * s.ipt;
    s.nb = ceil_div(n, s.B);
    fit_rows(s, n, VJP_RECORD_BYTES);
    return s;
}

template <int W, int IPT>
static void launch_rows(int nb, const VjpArgs &a, bool per, bool pair, int row0, int row1, double *records,
                        cudaStream_t s) {
    const VjpBlocks b{nb, row0, pairs_before(nb, row0)};
    const unsigned grid = (unsigned)(pairs_before(nb, row1) - b.item0);
    if (pair) {
        if (per)
            vjp_pair_kernel<W, IPT, true><<<grid, 32 * W, 0, counted(s)>>>(a, b, records);
        else
            vjp_pair_kernel<W, IPT, false><<<grid, 32 * W, 0, counted(s)>>>(a, b, records);
    } else {
        if (per)
            vjp_oseen_kernel<W, IPT, true>
                <<<grid, 32 * W, 0, counted(s)>>>(a.n, a.x, a.y, a.z, a.lx, a.ly, a.lz, a.L, a.halfL, b, records);
        else
            vjp_oseen_kernel<W, IPT, false>
                <<<grid, 32 * W, 0, counted(s)>>>(a.n, a.x, a.y, a.z, a.lx, a.ly, a.lz, a.L, a.halfL, b, records);
    }
}

// One O(N^2) pass: mu (into a.mx, ... and own + 8 n) or the pair terms (into the gradients).  a: the caller's arrays.
static void vjp_pass(const VjpShape &sh, const VjpArgs &a, bool per, bool pair, double *records, double *own,
                     cudaStream_t s) {
    const size_t n = (size_t)a.n;
    double *const sums = own, *const adm = own + 4 * n, *const mu = own + 8 * n;
    VjpArgs p = a;  // as the pairs read them
    p.x = adm, p.y = adm + n, p.z = adm + 2 * n, p.r = adm + 3 * n;
    p.mx = mu, p.my = mu + n, p.mz = mu + 2 * n;
    for (int row0 = 0; row0 < sh.nb; row0 += sh.rows) {
        const int row1 = min(sh.nb, row0 + sh.rows);
        if (sh.warps == 2)
            launch_rows<2, 2>(sh.nb, p, per, pair, row0, row1, records, s);
        else if (sh.ipt == 2)
            launch_rows<1, 2>(sh.nb, p, per, pair, row0, row1, records, s);
        else
            launch_rows<1, 1>(sh.nb, p, per, pair, row0, row1, records, s);
        if (pair)
            vjp_sum_kernel<4><<<ceil_div(4LL * a.n, 128), 128, 0, counted(s)>>>(a, sh.B, sh.nb, row0, row1, records, sums,
                                                                               nullptr);
        else
            vjp_sum_kernel<3><<<ceil_div(3LL * a.n, 128), 128, 0, counted(s)>>>(a, sh.B, sh.nb, row0, row1, records, sums,
                                                                               mu);
    }
}

int launch_direct_vjp(dem_ctx *ctx, int n, const double *x, const double *y, const double *z, const double *r,
                      const double *fx, const double *fy, const double *fz, const double *lx, const double *ly,
                      const double *lz, double m_const, double eta, double stokes, double L, int periodic,
                      double *mx, double *my, double *mz, double *gx, double *gy, double *gz, double *gr,
                      cudaStream_t s) {
    if (n == 0) return DEM_OK;
    VjpShape sh = vjp_shape(n);
    // the context's partial sums, [splits][3][capacity]: the droplets' own, then the records; where the device has no
    // room for them, fewer block rows per launch (the same sums in the same order)
    auto ensure = [&] {
        return dem_ensure_partials(ctx, ceil_div((int64_t)(sh.bytes / sizeof(double)), 3LL * ctx->capacity));
    };
    int rc = ensure();
    while (rc && sh.rows > 1) {
        fit_rows(sh, n, record_bytes(sh) / 2);
        rc = ensure();
    }
    if (rc) return rc;
    double *own = ctx->partial, *records = own + VJP_OWN * (size_t)n;
    const VjpArgs a{n, x, y, z, r, fx, fy, fz, lx, ly, lz, mx, my, mz, m_const, eta, stokes, L, 0.5 * L, gx, gy, gz, gr};
    dem_prof_begin(ctx, "vjp_mu_pass", s);
    vjp_admit_kernel<<<min(ceil_div(n, 256), 8 * ctx->sm_count), 256, 0, counted(s)>>>(a, own + 4 * (size_t)n);
    vjp_pass(sh, a, periodic != 0, false, records, own, s);
    dem_prof_end(ctx, s);
    if ((rc = dem_check_launch(ctx, "vjp mu"))) return rc;
    dem_prof_begin(ctx, "vjp_pass", s);
    vjp_pass(sh, a, periodic != 0, true, records, own, s);
    dem_prof_end(ctx, s);
    return dem_check_launch(ctx, "vjp pair pass");
}

}  // namespace dem
