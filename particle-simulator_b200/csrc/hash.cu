// hash.cu -- spatial-hash collision detection with the reference's exact
// cell, hash and distance semantics, producing the sorted unique pair set.
//
// dem/collision_detector/spatial_hash_collision_detector.py:
//   _hash_cell :74-76, _assign_cells :79-112, _prefix_sum :115-123,
//   _scatter_particles :126-132, _detect_collisions :135-229, detect :233-316.
//
// The reference compares a droplet i with every j > i in the hash buckets of the
// 27 cells around its own, cells of twice the LARGEST radius: ~120 candidates per
// droplet for lognormal radii at 2 % volume fraction, of which one in 250 touches
// something.  Its pair set is {touching pairs} intersected with {pairs whose
// bucket the 27 cells reach}; the second condition is a property of two droplets
// alone, so it is checked for touching pairs only and these are found on a search
// grid of their own (hashed cells of 4.5 MEAN radii, smaller in dense boxes):
//   1. maximum and mean radius; the last CTA derives both grids
//   2. search cell of every droplet, rank in its bucket (atomics)
//   3. bucket starts (any order: one CTA-wide scan and one atomic per CTA)
//   4. FP32 records in bucket order
//   5. per droplet i: the search cells within 2 r_i (i is the pair's larger droplet,
//      ties by index, so this covers the contact distance); candidates pass an FP32
//      far test, then the reference's contact test in FP64, then the reachability
//      test: list of pairs, pairs per row, raw hits
//   6. exclusive scan of the row counts, pairs into their rows, rows sorted by rank
//      (more pairs than the list holds: found again, straight into the output's rows)
// A droplet reads ~6 cells and ~2 candidates at 2 % volume fraction.
// Memory roofline: the chain is bounded by HBM and latency, not arithmetic.  Its
// algorithmic bytes per detection are 32 N + 8 K (N droplets, K pairs): position and
// radius read once, 8 B per pair written.  Kernels, periodic, before (27 buckets per
// droplet) -> now: N = 2^20 769 -> 235 us (the search 580 -> 125, bound by L2
// latency), N = 2,000 123 -> 54, of which most are gaps between short kernels.
// Dense boxes are bounded by the tests' instructions.  A whole detection, equal
// radii, periodic, us, before -> now, N = 100,000: volume fraction 0.3 (1.2 pairs
// per droplet) 328 -> 222, 0.6 386 -> 239, 2 545 -> 347, 7 1,205 -> 689; N = 400,000:
// 0.3 730 -> 464, 0.6 864 -> 540, 2 1,225 -> 824, 5 2,098 -> 1,605.  Past about 25
// pairs per droplet the list no longer holds them: the kernels alone, at 28, N =
// 100,000 1,098 -> 1,011, 400,000 2,816 -> 3,423.
// The contact test is the same IEEE expression as the reference's (this file is
// compiled with -fmad=false) and does not depend on the order of the two droplets,
// so the pair set is bit-identical to the reference's np.unique output.
#include <algorithm>
#include <climits>
#include <cmath>

#include "common.cuh"
#include "scan.cuh"

namespace dem {

struct HashParams {
    double cell;
    int32_t grid;
    int32_t valid;
};

__device__ __forceinline__ unsigned long long ordered_bits(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double from_ordered_bits(unsigned long long o) {
    const unsigned long long b = (o >> 63) ? (o & 0x7fffffffffffffffull) : ~o;
    return __longlong_as_double((long long)b);
}

__global__ void max_kernel(int n, const double *__restrict__ r, unsigned long long *__restrict__ slot) {
    unsigned long long m = 0ull;  // below every ordered value
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned long long o = ordered_bits(r[i]);
        m = o > m ? o : m;
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, m, off);
        m = t > m ? t : m;
    }
    if ((threadIdx.x & 31) == 0) atomicMax(slot, m);
}

// even_cells = 0: the reference's grid, cell = 2 max r and grid = ceil(L / cell)
// (a periodic box whose side is not a whole number of cells gets a partial last
// cell, across which touching pairs one cell apart are not compared -- the
// reference's pair set, kept bit-exact).  even_cells = 1 (the generator's own
// use): grid = floor(L / (2 max r)) whole cells of side L / grid >= 2 max r, so
// every touching pair is compared across the periodic faces too.
__device__ __forceinline__ HashParams hash_params(double max_radius, double L, int even_cells) {
    double cell = 2.0 * max_radius;  // :258
    HashParams p;
    p.valid = cell > 0 ? 1 : 0;  // :259-260
    double g = p.valid ? (even_cells ? floor(L / cell) : ceil(L / cell)) : 1.0;
    if (!(g >= 1.0)) g = 1.0;
    if (g > 1073741824.0) g = 1073741824.0;
    if (even_cells && p.valid) cell = L / g;
    p.cell = cell;
    p.grid = (int32_t)g;  // :262
    return p;
}

__global__ void hash_params_kernel(const unsigned long long *__restrict__ slot, double L, HashParams *__restrict__ hp) {
    *hp = hash_params(from_ordered_bits(*slot), L, 0);
}

__device__ __forceinline__ int32_t hash_cell(int32_t ix, int32_t iy, int32_t iz, int32_t mask) {
    const uint32_t h = ((uint32_t)ix * 73856093u) ^ ((uint32_t)iy * 19349663u) ^ ((uint32_t)iz * 83492791u);
    return (int32_t)(h & (uint32_t)mask);
}

__device__ __forceinline__ int32_t floor_mod(int32_t a, int32_t m) {
    if ((uint32_t)a < (uint32_t)m) return a;
    const int32_t q = a % m;
    return q < 0 ? q + m : q;
}

// floor_mod(a, m) for a in [-1, m] (a neighbour of a periodic cell coordinate)
__device__ __forceinline__ int32_t wrap1(int32_t a, int32_t m) {
    a += a < 0 ? m : 0;
    return a >= m ? a - m : a;
}

__device__ __forceinline__ int32_t cell_coord(double p, double cell, int32_t grid, bool periodic) {
    int32_t v = (int32_t)floor(p / cell);
    if (periodic) return floor_mod(v, grid);
    return v < 0 ? 0 : (v >= grid ? grid - 1 : v);
}

__global__ void assign_kernel(int n, const double *__restrict__ x, const double *__restrict__ y,
                              const double *__restrict__ z, const HashParams *__restrict__ hp, int periodic,
                              int32_t mask, int32_t *__restrict__ cell_hash, int32_t *__restrict__ bucket_count) {
    const HashParams p = *hp;
    if (!p.valid) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int32_t ix = cell_coord(x[i], p.cell, p.grid, periodic);
        const int32_t iy = cell_coord(y[i], p.cell, p.grid, periodic);
        const int32_t iz = cell_coord(z[i], p.cell, p.grid, periodic);
        const int32_t h = hash_cell(ix, iy, iz, mask);
        cell_hash[i] = h;
        atomicAdd(&bucket_count[h], 1);
    }
}

__global__ void scatter_kernel(int n, const int32_t *__restrict__ cell_hash, const HashParams *__restrict__ hp,
                               int32_t *__restrict__ cursor, int32_t *__restrict__ sorted_idx) {
    if (!hp->valid) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int32_t slot = atomicAdd(&cursor[cell_hash[i]], 1);
        sorted_idx[slot] = i;
    }
}

// The reference's contact test sqrt(d2) <= s (s = r_i + r_j, the root correctly
// rounded), decided from d2 alone unless d2 lies within a relative 2^-45 of s^2.
// With s2 = RN(s * s): d2 > s2 (1 + 2^-45) implies sqrt(d2) > s (1 + 2^-47), above
// s + ulp(s) / 2, so the rounded root exceeds s; d2 <= s2 (1 - 2^-45) implies
// d2 < s^2, so the rounded root is <= s.  Both need s > 0 and s2 normal and
// finite (the relative bounds), else, and inside the band, the square root decides.
__device__ __forceinline__ bool contact_rn(double d2, double s) {
    const double s2 = s * s;
    const bool normal = s > 0.0 && s2 >= 0x1p-960 && s2 <= 0x1p+960;
    if (normal && d2 > s2 * (1.0 + 0x1p-45)) return false;
    if (normal && d2 <= s2 * (1.0 - 0x1p-45)) return true;
    return sqrt(d2) <= s;
}

// Visits every candidate j > i of droplet i (the distinct buckets of its 27
// neighbour cells) and calls f(j) for those in contact (the allocation-free
// detector).
template <typename F>
__device__ __forceinline__ void for_each_contact(int i, const double *__restrict__ x, const double *__restrict__ y,
                                                 const double *__restrict__ z, const double *__restrict__ r,
                                                 const HashParams &p, int periodic, double L, double halfL,
                                                 int32_t mask, int n, const int32_t *__restrict__ bstart,
                                                 const int32_t *__restrict__ sorted_idx, F &&f) {
    const double xi = x[i], yi = y[i], zi = z[i], ri = r[i];
    const int32_t cx = cell_coord(xi, p.cell, p.grid, periodic);
    const int32_t cy = cell_coord(yi, p.cell, p.grid, periodic);
    const int32_t cz = cell_coord(zi, p.cell, p.grid, periodic);
    auto candidate = [&](int32_t s, int m) {
        const int32_t j = sorted_idx[s];
        if (!(i < j)) return;
        double dx = x[j] - xi, dy = y[j] - yi, dz = z[j] - zi;
        if (periodic) {
            dx = mic64(dx, L, halfL);
            dy = mic64(dy, L, halfL);
            dz = mic64(dz, L, halfL);
        }
        if (contact_rn(dx * dx + dy * dy + dz * dz, ri + r[j])) f(j, m);  // dist <= r_i + r_j
    };
    // Neighbour cell c = 9 (di + 1) + 3 (dj + 1) + (dk + 1): its bucket, or -1 outside an open box.
    auto cell_hash = [&](int c) -> int32_t {
        int32_t nx = cx + c / 9 - 1, ny = cy + (c / 3) % 3 - 1, nz = cz + c % 3 - 1;
        if (periodic) {  // cx, cy, cz lie in [0, grid): one step wraps (= floor_mod)
            nx = wrap1(nx, p.grid);
            ny = wrap1(ny, p.grid);
            nz = wrap1(nz, p.grid);
        } else if (nx < 0 || ny < 0 || nz < 0 || nx >= p.grid || ny >= p.grid || nz >= p.grid) {
            return -1;
        }
        return hash_cell(nx, ny, nz, mask);
    };
    // Usual case: the 27 cells map to distinct buckets (kept in registers: static indices).
    {
        int32_t h[27];
#pragma unroll
        for (int c = 0; c < 27; ++c) h[c] = cell_hash(c);
        bool dup = false;
#pragma unroll
        for (int c = 1; c < 27; ++c)
#pragma unroll
            for (int m = 0; m < c; ++m) dup |= h[c] >= 0 && h[c] == h[m];
        if (!dup) {
            for (int c = 0; c < 27; ++c) {
                const int32_t hc = cell_hash(c);
                if (hc < 0) continue;
                const int32_t start = bstart[hc];
                int32_t end = bstart[hc + 1];
                if (end > n) end = n;  // :199-201
                for (int32_t s = start; s < end; ++s) candidate(s, 1);
            }
            return;
        }
    }
    // Tiny grids or colliding buckets: a bucket seen from several cells is
    // scanned once, its contacts counted with that multiplicity.
    int32_t hs[27];
    int nh = 0;
    int mult[27];
    for (int di = -1; di <= 1; ++di)
        for (int dj = -1; dj <= 1; ++dj)
            for (int dk = -1; dk <= 1; ++dk) {
                int32_t nx = cx + di, ny = cy + dj, nz = cz + dk;
                if (periodic) {
                    nx = floor_mod(nx, p.grid);
                    ny = floor_mod(ny, p.grid);
                    nz = floor_mod(nz, p.grid);
                } else if (nx < 0 || ny < 0 || nz < 0 || nx >= p.grid || ny >= p.grid || nz >= p.grid) {
                    continue;
                }
                const int32_t h = hash_cell(nx, ny, nz, mask);
                int q = 0;
                while (q < nh && hs[q] != h) ++q;
                if (q == nh) {
                    hs[nh] = h;
                    mult[nh] = 1;
                    ++nh;
                } else {
                    ++mult[q];
                }
            }
    for (int q = 0; q < nh; ++q) {
        const int32_t start = bstart[hs[q]];
        int32_t end = bstart[hs[q] + 1];
        if (end > n) end = n;  // :199-201
        for (int32_t s = start; s < end; ++s) candidate(s, mult[q]);
    }
}

__global__ void count_pairs_kernel(int n, const double *__restrict__ x, const double *__restrict__ y,
                                   const double *__restrict__ z, const double *__restrict__ r,
                                   const HashParams *__restrict__ hp, int periodic,
                                   double L, int32_t mask, const int32_t *__restrict__ bstart,
                                   const int32_t *__restrict__ sorted_idx, int32_t *__restrict__ pair_count,
                                   unsigned long long *__restrict__ raw) {
    const HashParams p = *hp;
    unsigned long long local_raw = 0;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int i = p.valid ? sorted_idx[t] : t;  // bucket order (the buckets are filled when valid)
        int32_t c = 0;
        if (p.valid) {
            for_each_contact(i, x, y, z, r, p, periodic, L, 0.5 * L, mask, n, bstart, sorted_idx,
                             [&](int32_t, int m) {
                                 ++c;
                                 local_raw += (unsigned long long)m;
                             });
        }
        pair_count[i] = c;
    }
    if (local_raw) atomicAdd(raw, local_raw);
}

__global__ void write_pairs_kernel(int n, const double *__restrict__ x, const double *__restrict__ y,
                                   const double *__restrict__ z, const double *__restrict__ r,
                                   const HashParams *__restrict__ hp, int periodic, double L, int32_t mask,
                                   const int32_t *__restrict__ bstart, const int32_t *__restrict__ sorted_idx,
                                   const int64_t *__restrict__ offset, int32_t *__restrict__ pairs, int64_t cap,
                                   int64_t *__restrict__ counts, uint32_t *err) {
    const HashParams p = *hp;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        counts[0] = p.valid ? offset[n] : 0;
        if (p.valid && offset[n] > cap) raise_device_error(err, DEM_DEVERR_PAIR_OVERFLOW);
    }
    if (!p.valid) return;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int i = sorted_idx[t];  // bucket order, as in count_pairs_kernel
        const int64_t o0 = offset[i], o1 = offset[i + 1];
        // the row's slots that fit in the buffer: all of them, except in the one row that the
        // capacity cuts (o0 < cap < o1), and none in the rows after it
        const int64_t m = (o1 < cap ? o1 : cap) - o0;
        if (m <= 0) continue;
        // ascending j within the row of droplet i: each j found is inserted into the sorted run
        // pairs[o0 .. o0 + len); once the run holds m entries the largest drops out, so a cut row
        // keeps its m smallest j and the buffer holds the lexicographically first cap pairs
        int64_t len = 0;
        for_each_contact(i, x, y, z, r, p, periodic, L, 0.5 * L, mask, n, bstart, sorted_idx, [&](int32_t j, int) {
            int64_t q;
            if (len < m) {
                pairs[2 * (o0 + len)] = i;
                q = len++;
            } else {
                if (j >= pairs[2 * (o0 + m - 1) + 1]) return;
                q = m - 1;
            }
            while (q > 0 && pairs[2 * (o0 + q - 1) + 1] > j) {
                pairs[2 * (o0 + q) + 1] = pairs[2 * (o0 + q - 1) + 1];
                --q;
            }
            pairs[2 * (o0 + q) + 1] = j;
        });
    }
}

// ---------------------------------------------------------------------------
// The search of the context entry point
// ---------------------------------------------------------------------------
struct SearchParams {
    HashParams hash;   // the reference's cells
    double inv_h;      // search cells per unit length
    double r_max;
    int32_t m;         // search cells per axis, cyclic (a periodic box); 0: unbounded; 1: one cell holds everything
};

// Words of the workspace that a detection zeroes: these, the bucket counts, the row counts.
struct SearchMisc {
    unsigned long long max_bits;  // maximum radius (ordered bits)
    float r_sum;                  // of the positive radii
    unsigned int done;            // CTAs of radius_kernel that have finished
    unsigned int next_slot;       // slots given out to buckets
    unsigned int found;           // pairs in the list, modulo 2^32 (the scan of the row counts has the pairs' number)
    unsigned int pad[2];
};
static_assert(sizeof(SearchMisc) == 4 * SEARCH_MISC_WORDS, "ctx.cu sizes the workspace by this");

// Search cells: 4.5 mean radii, so that a mean droplet's reach (2 r) covers (4 / 4.5 + 1)^3 ~ 6.7 cells and a cell
// holds ~0.4 droplets at 2 % volume fraction; in dense boxes 1.3 mean distances (2 droplets per cell) down to one
// mean radius, which leaves fewer candidates outside the reach.  Detection, equal radii, periodic, us, with 4.5
// mean radii / this: N = 400,000, volume fraction 0.3: 503 / 483, 0.6: 1,241 / 1,033, 2: 3,344 / 2,127; N = 2^20 at
// 0.02: 369 / 374 (1 or 1.7 mean distances: within 3 %; all before the list could lie in the output).  Not below
// half the largest radius (whose droplet then searches at most 10^3 cells) nor above 4.5 of it.  Periodic boxes:
// whole cells, at most 1,024 per axis (cell_id tells the cells of one search apart).
// One cell for everything where distance does not decide: cells without a finite size (an infinite radius, whose
// droplet touches droplets at any distance; L = 0, negative or not finite) and radii below 2^-500 (the contact
// test's squares underflow: droplets many radii apart pass it).
__global__ void radius_kernel(int n, const double *__restrict__ r, double L, double spaced, int periodic, int even_cells,
                              SearchMisc *__restrict__ misc, SearchParams *__restrict__ out) {
    __shared__ bool last;
    unsigned long long m = 0ull;  // below every ordered value
    float sum = 0.f;
#pragma unroll 4
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double v = r[i];
        const unsigned long long o = ordered_bits(v);
        m = o > m ? o : m;
        sum += v > 0.0 ? (float)v : 0.f;
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, m, off);
        m = t > m ? t : m;
        sum += __shfl_xor_sync(0xffffffffu, sum, off);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&misc->max_bits, m);
        atomicAdd(&misc->r_sum, sum);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&misc->done, 1u) + 1u == gridDim.x;
    __syncthreads();
    if (!last || threadIdx.x != 0) return;
    __threadfence();
    SearchParams p;
    p.hash = hash_params(from_ordered_bits(*(volatile unsigned long long *)&misc->max_bits), L, even_cells);
    const double r_max = from_ordered_bits(*(volatile unsigned long long *)&misc->max_bits);
    const double mean = (double)*(volatile float *)&misc->r_sum / n;
    double h = fmax(fmax(fmin(spaced, 4.5 * mean), mean), 0.5 * r_max);
    h = h <= 4.5 * r_max ? h : 4.5 * r_max;
    p.r_max = r_max;
    p.m = 0;
    p.inv_h = 1.0 / h;
    if (periodic) {
        const double cells = floor(L / h);
        p.m = cells >= 1024.0 ? 1024 : cells >= 1.0 ? (int32_t)cells : 1;
        p.inv_h = p.m / L;
    }
    if (!(p.inv_h > 0.0 && p.inv_h < INFINITY && r_max >= 0x1p-500)) {
        p.m = 1;
        p.inv_h = 0.0;
    }
    *out = p;
}

__device__ __forceinline__ int32_t search_floor(double v) {  // floor, kept within +-2^30
    return (int32_t)fmin(fmax(floor(v), -0x1p30), 0x1p30);
}
__device__ __forceinline__ int32_t search_coord(double v, const SearchParams &p) {
    const int32_t c = search_floor(v * p.inv_h);
    return p.m ? floor_mod(c, p.m) : c;
}
__device__ __forceinline__ uint32_t search_bucket(int32_t cx, int32_t cy, int32_t cz, uint32_t mask) {
    uint32_t h = (uint32_t)cx * 0x9E3779B1u ^ (uint32_t)cy * 0x85EBCA77u ^ (uint32_t)cz * 0xC2B2AE3Du;
    h ^= h >> 15;
    return (h * 0x2C1B3C6Du >> 7) & mask;
}
// Tells the cells of one droplet's search apart: their coordinates differ by less than 512 per axis (open
// boxes: at most 10) or are the distinct residues below 1,024 of a periodic box.
__device__ __forceinline__ int32_t cell_id(int32_t cx, int32_t cy, int32_t cz) {
    return (int32_t)((uint32_t)cx + ((uint32_t)cy << 10) + ((uint32_t)cz << 20));
}

__global__ void search_assign_kernel(int n, const double *__restrict__ x, const double *__restrict__ y,
                                     const double *__restrict__ z, const SearchParams *__restrict__ sp, uint32_t mask,
                                     int32_t *__restrict__ count, int4 *__restrict__ key) {
    const SearchParams p = *sp;
    if (!p.hash.valid) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int32_t cx = search_coord(x[i], p), cy = search_coord(y[i], p), cz = search_coord(z[i], p);
        const uint32_t b = search_bucket(cx, cy, cz, mask);
        key[i] = make_int4((int)b, atomicAdd(&count[b], 1), cell_id(cx, cy, cz), 0);
    }
}

// bucket[b] = (first slot, droplets): the CTA scans its buckets and takes its slots with one atomic, so
// buckets of different CTAs follow one another in any order.
constexpr int SB_T = 256, SB_ITEMS = 8;
__global__ void __launch_bounds__(SB_T) search_starts_kernel(uint32_t buckets, const int32_t *__restrict__ count,
                                                             SearchMisc *__restrict__ misc,
                                                             const SearchParams *__restrict__ sp,
                                                             int2 *__restrict__ bucket) {
    if (!sp->hash.valid) return;
    __shared__ int wsum[SB_T / 32], base;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t first = (blockIdx.x * SB_T + threadIdx.x) * SB_ITEMS;
    int c[SB_ITEMS], own = 0;
#pragma unroll
    for (int k = 0; k < SB_ITEMS; ++k) {
        c[k] = first + k < buckets ? count[first + k] : 0;
        own += c[k];
    }
    int inc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    if (threadIdx.x == 0) {
        int total = 0;
        for (int k = 0; k < SB_T / 32; ++k) {
            const int v = wsum[k];
            wsum[k] = total;
            total += v;
        }
        base = (int)atomicAdd(&misc->next_slot, (unsigned int)total);
    }
    __syncthreads();
    int at = base + wsum[w] + inc - own;
#pragma unroll
    for (int k = 0; k < SB_ITEMS; ++k) {
        if (first + k < buckets) bucket[first + k] = make_int2(at, c[k]);
        at += c[k];
    }
}

__global__ void search_scatter_kernel(int n, const double *__restrict__ x, const double *__restrict__ y,
                                      const double *__restrict__ z, const double *__restrict__ r,
                                      const SearchParams *__restrict__ sp, const int4 *__restrict__ key,
                                      const int2 *__restrict__ bucket, float4 *__restrict__ rec) {
    if (!sp->hash.valid) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int4 k = key[i];
        const size_t s = bucket[k.x].x + k.y;
        rec[2 * s] = make_float4((float)x[i], (float)y[i], (float)z[i], (float)r[i]);
        rec[2 * s + 1] = make_float4(__int_as_float(i), __int_as_float(k.z), 0.f, 0.f);
    }
}

struct SearchArgs {
    int n;
    const double *x, *y, *z, *r;
    const SearchParams *sp;
    int periodic;
    double L, halfL;
    int32_t hash_mask;   // the reference's table
    uint32_t mask;       // search buckets - 1
    const int2 *bucket;
    const float4 *rec;   // per slot: (x, y, z, r), (droplet, cell id, -, -)
    SearchMisc *misc;
    int32_t *row_count;
    int32_t *list;       // pairs (i, j) in any order, list_cap of them
    uint32_t list_cap;
    int2 *tmp;           // the list's pairs in rows: tmp_cap pairs, or (rows' j only) 2 tmp_cap int32
    uint32_t tmp_cap;
    int2 *cut;           // the row that the capacity cuts, when the list does not hold all pairs: n pairs
    unsigned long long *raw;
};

// How many of the 27 cells around droplet i's cell map to droplet j's bucket (:160-201): 0 when the
// reference does not compare i with j > i.
__device__ __noinline__ int reference_hits(const SearchArgs &a, const HashParams &p, int i, int j) {
    const bool per = a.periodic;
    const int32_t cx = cell_coord(a.x[i], p.cell, p.grid, per), cy = cell_coord(a.y[i], p.cell, p.grid, per),
                  cz = cell_coord(a.z[i], p.cell, p.grid, per);
    const int32_t hj = hash_cell(cell_coord(a.x[j], p.cell, p.grid, per), cell_coord(a.y[j], p.cell, p.grid, per),
                                 cell_coord(a.z[j], p.cell, p.grid, per), a.hash_mask);
    uint32_t hx[3], hy[3], hz[3];  // hash_cell's products of the three neighbours per axis
    bool in[3][3];                 // inside the grid (a periodic one: always)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        int32_t nx = cx + d - 1, ny = cy + d - 1, nz = cz + d - 1;
        if (per) nx = wrap1(nx, p.grid), ny = wrap1(ny, p.grid), nz = wrap1(nz, p.grid);
        hx[d] = (uint32_t)nx * 73856093u, hy[d] = (uint32_t)ny * 19349663u, hz[d] = (uint32_t)nz * 83492791u;
        in[d][0] = (uint32_t)nx < (uint32_t)p.grid, in[d][1] = (uint32_t)ny < (uint32_t)p.grid, in[d][2] = (uint32_t)nz < (uint32_t)p.grid;
    }
    int hits = 0;
#pragma unroll
    for (int c = 0; c < 27; ++c)
        hits += in[c / 9][0] && in[c / 3 % 3][1] && in[c % 3][2] &&
                (int32_t)((hx[c / 9] ^ hy[c / 3 % 3] ^ hz[c % 3]) & (uint32_t)a.hash_mask) == hj;
    return hits;
}

// The reference's contact test of two droplets (:203-219).
__device__ __forceinline__ bool in_contact(const SearchArgs &a, int i, int j) {
    double dx = a.x[j] - a.x[i], dy = a.y[j] - a.y[i], dz = a.z[j] - a.z[i];
    if (a.periodic) {
        dx = mic64(dx, a.L, a.halfL);
        dy = mic64(dy, a.L, a.halfL);
        dz = mic64(dz, a.L, a.halfL);
    }
    return contact_rn(dx * dx + dy * dy + dz * dz, a.r[i] + a.r[j]);  // dist <= r_i + r_j
}

// FP32 record q of a droplet, its radius widened for far_apart: by 2^-17 (max |x_i| + L) plus 2^-18 of the radii
// sum, far more than FP32 rounding of either record can account for.  A margin below 2^-100 turns the far
// test off.
__device__ __forceinline__ float4 widened(float4 q, double L) {
    const float marg = 0x1p-17f * (fmaxf(fabsf(q.x), fmaxf(fabsf(q.y), fabsf(q.z))) + fabsf((float)L));
    q.w = marg >= 0x1p-100f ? q.w * (1.f + 0x1p-18f) + marg : INFINITY;
    return q;
}
// Clearly not in contact (c: the candidate's record).  The per-axis distance is bounded below by the smaller of
// |d| and ||d| - L|, which covers either image the FP64 test may take; NaNs and overflowed bounds fail the
// comparison and go to the FP64 test, so every pair that test accepts is still found.
__device__ __forceinline__ bool far_apart(const float4 &q, const float4 &c, bool periodic, float Lf) {
    float ax = fabsf(c.x - q.x), ay = fabsf(c.y - q.y), az = fabsf(c.z - q.z);
    if (periodic) {
        ax = fminf(ax, fabsf(ax - Lf));
        ay = fminf(ay, fabsf(ay - Lf));
        az = fminf(az, fabsf(az - Lf));
    }
    const float s = fmaf(c.w, 1.f + 0x1p-18f, q.w);
    return fmaf(ax, ax, fmaf(ay, ay, az * az)) > s * s;
}

// The search cells within `reach` of a coordinate, per axis: first cell and how many (periodic: wrapped, each
// cell once).  `slack` covers the rounding of v and of the cell coordinates.  A coordinate that is not finite
// touches nothing (unless a radius is infinite: one cell).
struct Span {
    int32_t first, len;
};
__device__ __forceinline__ Span span_of(double v, double reach, double slack, const SearchParams &p) {
    if (p.m == 1) return {0, 1};
    if (!(fabs(v) < INFINITY)) return {0, 0};
    const double wide = reach * (1.0 + 0x1p-18) + slack;
    const int32_t lo = search_floor((v - wide) * p.inv_h), hi = search_floor((v + wide) * p.inv_h);
    const long long len = (long long)hi - lo + 1;
    if (!p.m) return {lo, (int32_t)len};  // len <= ~20: cells are at least half the largest radius
    return len >= p.m ? Span{0, p.m} : Span{floor_mod(lo, p.m), (int32_t)len};
}
// From an FP32 coordinate (rounded by 2^-24 of itself), unless that is coarse against the cells or the cells
// are near FP32's subnormal range.
__device__ __forceinline__ Span span_of32(float v, const double *__restrict__ exact, int i, double reach, double L,
                                          const SearchParams &p) {
    const double slack = 0x1p-20 * (fabs((double)v) + (p.m ? fabs(L) : 0.0));
    if (slack * p.inv_h < 0.125 && p.inv_h < 0x1p100) return span_of((double)v, reach, slack, p);
    const double e = exact[i];
    return span_of(e, reach, 1e-14 * (fabs(e) + (p.m ? fabs(L) : 0.0)), p);
}
__device__ __forceinline__ int32_t span_cell(const Span &s, int k, const SearchParams &p) {
    const int32_t c = s.first + k;
    return p.m && c >= p.m ? c - p.m : c;
}

// `group` <= 32 droplets (bucket order, from slot t0 on) per warp.  Their search cells form one list, 32 of which
// the warp looks up at a time, and the droplets found in them another, of which it tests 32 at a time: a droplet
// has 1 to 27 cells, rarely thousands, and 0 to a few candidates in each, so loops per lane would mostly wait for
// the longest lane's loads (436 us at N = 2^20; this form 125).  Pairs that pass the far test queue up in turn, and
// settle(touching, i, j), i < j, takes 32 of them: the contact test and its caller's reachability test, ~1,500
// instructions, run with full warps.
struct SearchWarp {
    float4 q[32];              // widened record
    float r[32];               // radius
    int i[32];                 // droplet
    Span span[3][32];
    int first[32];             // the droplet's first entry in the list of cells
    int2 queue[64];            // candidates: slot, (cell id)
    unsigned char owner[64];   // and whose
    int2 near[64];             // pairs to settle
};

template <typename Settle>
__device__ __forceinline__ void search_warp(const SearchArgs &a, const SearchParams &p, SearchWarp &sh, int t0, int group,
                                            Settle &&settle) {
    const int lane = threadIdx.x & 31, t = t0 + lane;
    const unsigned lt = (1u << lane) - 1u;
    const float Lf = (float)a.L;
    int cells = 0;
    if (lane < group && t < a.n) {
        const float4 q = a.rec[2 * (size_t)t];
        const int i = __float_as_int(a.rec[2 * (size_t)t + 1].x);
        sh.q[lane] = widened(q, a.L);
        sh.r[lane] = q.w;
        sh.i[lane] = i;
        // The partner's radius is at most this droplet's (by the FP32 order), so 2 r covers the contact
        // distance; where FP32 radii are not normal numbers their order says nothing and r_max bounds it.
        const double reach = q.w > 0x1p-100f && q.w < 0x1p100f ? 2.0 * q.w : a.r[i] + p.r_max;
        if (reach >= 0.0) {  // (a pair of negative radii never touches)
            const Span sx = span_of32(q.x, a.x, i, reach, a.L, p), sy = span_of32(q.y, a.y, i, reach, a.L, p),
                       sz = span_of32(q.z, a.z, i, reach, a.L, p);
            sh.span[0][lane] = sx;
            sh.span[1][lane] = sy;
            sh.span[2][lane] = sz;
            cells = sx.len * sy.len * sz.len;
        }
    }
    int end = cells;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += v;
    }
    const int total = __shfl_sync(0xffffffffu, end, 31);
    sh.first[lane] = end - cells;
    __syncwarp();

    // Entry e of the list of cells: its owner, its cell's id and bucket.
    auto look_up = [&](int e, int &owner, int &id) -> int2 {
        if (e >= total) return make_int2(0, 0);
        int lo = 0;
#pragma unroll
        for (int step = 16; step; step >>= 1)  // the last lane whose first entry is <= e (an empty lane shares the next one's)
            if (lo + step < 32 && sh.first[lo + step] <= e) lo += step;
        owner = lo;
        const Span sx = sh.span[0][lo], sy = sh.span[1][lo], sz = sh.span[2][lo];
        const int k = e - sh.first[lo], kxy = k / sz.len;
        const int32_t cz = span_cell(sz, k - kxy * sz.len, p), kx = kxy / sy.len;
        const int32_t cy = span_cell(sy, kxy - kx * sy.len, p), cx = span_cell(sx, kx, p);
        id = cell_id(cx, cy, cz);
        return a.bucket[search_bucket(cx, cy, cz, a.mask)];
    };
    int near = 0;
    auto settle_near = [&](int k) {
        const int2 e = lane < k ? sh.near[lane] : make_int2(0, 0);
        settle(lane < k && in_contact(a, e.x, e.y), e.x, e.y);
    };
    // The first `k` <= 32 queued candidates: the smaller droplets (ties: the smaller index) of their cells.
    auto test = [&](int k) {
        bool hit = false;
        int i = 0, j = 0;
        if (lane < k) {
            const int2 c = sh.queue[lane];
            const int o = sh.owner[lane];
            const float4 q = a.rec[2 * (size_t)c.x], r = a.rec[2 * (size_t)c.x + 1];
            i = sh.i[o];
            j = __float_as_int(r.x);
            const bool smaller = q.w < sh.r[o] || (q.w == sh.r[o] && j < i);
            hit = smaller && __float_as_int(r.y) == c.y && !far_apart(sh.q[o], q, a.periodic, Lf);
        }
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        if (!hits) return;
        if (hit) sh.near[near + __popc(hits & lt)] = make_int2(min(i, j), max(i, j));
        near += __popc(hits);
        __syncwarp();
        if (near < 32) return;
        settle_near(32);
        near -= 32;
        const int2 rest = sh.near[32 + lane];
        __syncwarp();
        if (lane < near) sh.near[lane] = rest;
        __syncwarp();
    };
    int queued = 0;
    int owner = 0, id = 0;
    int2 b = look_up(lane, owner, id);
    for (int e = lane; e - lane < total; e += 32) {
        int next_owner = 0, next_id = 0;
        const int2 next = look_up(e + 32, next_owner, next_id);  // in flight while this round's are queued
        for (int k = 0; __any_sync(0xffffffffu, k < b.y); ++k) {
            const unsigned live = __ballot_sync(0xffffffffu, k < b.y);
            if (k < b.y) {
                const int at = queued + __popc(live & lt);
                sh.queue[at] = make_int2(b.x + k, id);
                sh.owner[at] = (unsigned char)owner;
            }
            queued += __popc(live);
            __syncwarp();
            if (queued >= 32) {
                test(32);
                queued -= 32;
                const int2 c = sh.queue[32 + lane];
                const unsigned char o = sh.owner[32 + lane];
                __syncwarp();
                sh.queue[lane] = c;
                sh.owner[lane] = o;
                __syncwarp();
            }
        }
        b = next;
        owner = next_owner;
        id = next_id;
    }
    test(queued);
    if (near) settle_near(near);
    __syncwarp();  // the warp's next droplets may take its place
}

// The pairs into the list (as many as it holds), pairs per row, raw hits.
constexpr int SP_WARPS = 4;
__global__ void __launch_bounds__(32 * SP_WARPS) search_pairs_kernel(const __grid_constant__ SearchArgs a, int group) {
    __shared__ SearchWarp sh[SP_WARPS];
    const SearchParams p = *a.sp;
    if (!p.hash.valid) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long raw = 0;
    search_warp(a, p, sh[w], (blockIdx.x * SP_WARPS + w) * group, group, [&](bool touching, int i, int j) {
        const int hits = touching ? reference_hits(a, p.hash, i, j) : 0;
        raw += hits;
        if (hits) atomicAdd(&a.row_count[i], 1);
        const unsigned found = __ballot_sync(0xffffffffu, hits > 0);
        unsigned at = 0;
        if (lane == 0 && found) at = atomicAdd(&a.misc->found, (unsigned)__popc(found));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(found & ((1u << lane) - 1u));
        if (hits && at < a.list_cap) {
            a.list[2 * (size_t)at] = i;
            a.list[2 * (size_t)at + 1] = j;
        }
    });
    if (raw) atomicAdd(a.raw, raw);
}

// The row that the capacity cuts (n when it cuts none): some of its pairs lie below `cap`, some above.
__device__ __forceinline__ int cut_row(const int64_t *__restrict__ offset, int n, int64_t cap) {
    if (offset[n] <= cap) return n;
    int lo = 0, hi = n;  // offset[lo] <= cap < offset[hi]
    while (hi - lo > 1) {
        const int mid = lo + (hi - lo) / 2;
        if (offset[mid] <= cap)
            lo = mid;
        else
            hi = mid;
    }
    return offset[lo] < cap ? lo : n;
}

// The pairs into their rows (any order within a row): those of the list into `tmp`, their j only where `tmp` has no
// room for pairs.  More pairs than the list holds: they are searched again, straight into the output (j only), and
// the row that the capacity cuts into `cut`.
constexpr int PL_WARPS = 8;
__global__ void __launch_bounds__(32 * PL_WARPS) place_pairs_kernel(const __grid_constant__ SearchArgs a, int group,
                                                                    const int64_t *__restrict__ offset, int32_t *pairs,
                                                                    int64_t cap) {
    __shared__ SearchWarp sh[PL_WARPS];
    const SearchParams p = *a.sp;
    if (!p.hash.valid) return;
    const int64_t total = offset[a.n];
    if (total <= (int64_t)a.list_cap) {
        int32_t *const tmp_j = reinterpret_cast<int32_t *>(a.tmp);
        for (int64_t q = blockIdx.x * blockDim.x + threadIdx.x; q < total; q += gridDim.x * blockDim.x) {
            const int i = a.list[2 * q], j = a.list[2 * q + 1];
            const int64_t at = offset[i] + atomicSub(&a.row_count[i], 1) - 1;
            if (total <= (int64_t)a.tmp_cap)
                a.tmp[at] = make_int2(i, j);
            else
                tmp_j[at] = j;
        }
        return;
    }
    const int w = threadIdx.x >> 5, warps = gridDim.x * PL_WARPS;
    for (int64_t t0 = (int64_t)(blockIdx.x * PL_WARPS + w) * group; t0 < a.n; t0 += (int64_t)warps * group)
        search_warp(a, p, sh[w], (int)t0, group, [&](bool touching, int i, int j) {
            if (!touching || offset[i] >= cap || !reference_hits(a, p.hash, i, j)) return;
            const int64_t o0 = offset[i], at = o0 + atomicSub(&a.row_count[i], 1) - 1;
            if (offset[i + 1] <= cap)
                pairs[2 * at + 1] = j;
            else
                a.cut[at - o0] = make_int2(i, j);
        });
}

// Row i: its j's (STRIDE apart) in ascending order, as pairs, to `to`; STRIDE 2: they are the second entries there.
// By one thread: up to 8; by a warp: up to 128 from registers, more as a bitonic sort in place whose comparators all
// put the smaller value first (entries past the end would be the largest: left out).
constexpr int ROW_THREAD = 8, ROW_REGS = 4;
template <int STRIDE>
__device__ __forceinline__ void sort_row_thread(const int32_t *from, int len, int i, int32_t *to) {
    int v[ROW_THREAD];
#pragma unroll
    for (int k = 0; k < ROW_THREAD; ++k) v[k] = k < len ? from[STRIDE * k] : INT_MAX;
#pragma unroll
    for (int k = 0; k < ROW_THREAD; ++k) {
        int rank = 0;
#pragma unroll
        for (int q = 0; q < ROW_THREAD; ++q) rank += v[q] < v[k];
        if (k < len) {
            to[2 * rank] = i;
            to[2 * rank + 1] = v[k];
        }
    }
}
template <int STRIDE>
__device__ __forceinline__ void sort_row_warp(int32_t *from, int64_t len, int i, int32_t *to, int lane) {
    if (len <= 32 * ROW_REGS) {
        int v[ROW_REGS], rank[ROW_REGS];
#pragma unroll
        for (int k = 0; k < ROW_REGS; ++k) {
            v[k] = 32 * k + lane < len ? from[STRIDE * (32 * k + lane)] : INT_MAX;
            rank[k] = 0;
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < ROW_REGS; ++q) {
            if (32 * q >= len) break;
            for (int l = 0; l < 32; ++l) {
                const int other = __shfl_sync(0xffffffffu, v[q], l);
#pragma unroll
                for (int k = 0; k < ROW_REGS; ++k) rank[k] += other < v[k];
            }
        }
#pragma unroll
        for (int k = 0; k < ROW_REGS; ++k)
            if (32 * k + lane < len) {
                to[2 * rank[k]] = i;
                to[2 * rank[k] + 1] = v[k];
            }
        __syncwarp();
        return;
    }
    auto order = [&](int64_t x, int64_t y) {
        if (y >= len) return;
        const int32_t u = from[STRIDE * x], v = from[STRIDE * y];
        if (u > v) {
            from[STRIDE * x] = v;
            from[STRIDE * y] = u;
        }
    };
    for (int64_t size = 2; size < 2 * len; size <<= 1) {
        const int64_t whole = (len + size - 1) / size * size;
        for (int64_t t = lane; 2 * t < whole; t += 32) {  // blocks of `size`: ends inwards
            const int64_t first = 2 * t / size * size, k = t % (size / 2);
            order(first + k, first + size - 1 - k);
        }
        __syncwarp();
        for (int64_t step = size / 4; step > 0; step >>= 1) {
            for (int64_t t = lane; 2 * t < whole; t += 32) {
                const int64_t x = 2 * t - (t & (step - 1));
                order(x, x + step);
            }
            __syncwarp();
        }
    }
    for (int64_t t = lane; t < len; t += 32) {
        to[2 * t] = i;
        if (STRIDE == 1) to[2 * t + 1] = from[t];
    }
    __syncwarp();
}

// The rows that end at or before `cap`, from `tmp` (STRIDE 1) or in the output itself.
template <int STRIDE>
__device__ __forceinline__ void sort_rows(int n, const int64_t *__restrict__ offset, int32_t *from, int32_t *pairs, int64_t cap) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31, warps = gridDim.x * blockDim.x >> 5;
    const int per = min(32, max(1, (n + warps - 1) / warps));  // rows per warp and round
    for (int64_t i0 = (int64_t)(tid >> 5) * per; i0 < n; i0 += (int64_t)warps * per) {
        const int64_t i = i0 + lane;
        int64_t o0 = 0, o1 = 0;
        if (lane < per && i < n) o0 = offset[i], o1 = offset[i + 1];
        const int64_t len = o1 <= cap ? o1 - o0 : 0;
        if (len > 0 && len <= ROW_THREAD) sort_row_thread<STRIDE>(from + STRIDE * o0, (int)len, (int)i, pairs + 2 * o0);
        for (unsigned m = __ballot_sync(0xffffffffu, len > ROW_THREAD); m; m &= m - 1) {
            const int l = __ffs(m) - 1;
            const int64_t at = __shfl_sync(0xffffffffu, o0, l);
            sort_row_warp<STRIDE>(from + STRIDE * at, __shfl_sync(0xffffffffu, len, l), (int)(i0 + l), pairs + 2 * at, lane);
        }
    }
}

// The rows sorted by j; entries at or past `cap` are dropped, so the buffer holds the lexicographically first
// cap pairs.  Pairs in `tmp` go to their rank in their row, a thread each; else the rows are sorted, and the row
// that the capacity cuts comes from `cut`.
__global__ void __launch_bounds__(256) write_rows_kernel(const __grid_constant__ SearchArgs a, const int64_t *__restrict__ offset,
                                                         int32_t *pairs, int64_t cap, int64_t *__restrict__ counts,
                                                         uint32_t *err) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, threads = gridDim.x * blockDim.x;
    const bool valid = a.sp->hash.valid;
    const int64_t total = valid ? offset[a.n] : 0;
    if (tid == 0) {
        counts[0] = total;
        if (total > cap) raise_device_error(err, DEM_DEVERR_PAIR_OVERFLOW);
    }
    if (!valid) return;
    // Entry e of a row of `len` entries to its place from `to` on.
    auto place = [&](const int2 &e, const int2 *row, int64_t len, int64_t to) {
        for (int64_t w = 0; w < len; ++w) to += row[w].y < e.y;
        if (to < cap) {
            pairs[2 * to] = e.x;
            pairs[2 * to + 1] = e.y;
        }
    };
    const bool listed = total <= (int64_t)a.list_cap;
    if (listed && total <= (int64_t)a.tmp_cap) {
        for (int64_t q = tid; q < total; q += threads) {
            const int2 e = a.tmp[q];
            const int64_t o0 = offset[e.x];
            place(e, a.tmp + o0, offset[e.x + 1] - o0, o0);
        }
    } else if (listed) {
        sort_rows<1>(a.n, offset, reinterpret_cast<int32_t *>(a.tmp), pairs, cap);
    } else {
        const int cut = cut_row(offset, a.n, cap);
        if (cut < a.n) {
            const int64_t len = offset[cut + 1] - offset[cut];
            for (int64_t q = tid; q < len; q += threads) place(a.cut[q], a.cut, len, offset[cut]);
        }
        sort_rows<2>(a.n, offset, pairs + 1, pairs, cap);
    }
}

// DirectCollisionFrequency.compute, pbm/collision_frequency/direct_collision_freq.py:17-41, on the
// detected pairs: matrix[b_i][b_j] += 1 and matrix[b_j][b_i] += 1 for every pair.
__global__ void pair_bin_kernel(const int32_t *__restrict__ pairs, const int64_t *__restrict__ num_pairs,
                                int64_t cap, const int32_t *__restrict__ bins, int nbins,
                                unsigned int *__restrict__ matrix) {
    const int64_t k = min(num_pairs[0], cap);
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < k; p += (int64_t)gridDim.x * blockDim.x) {
        const int bi = bins[pairs[2 * p]], bj = bins[pairs[2 * p + 1]];
        atomicAdd(&matrix[bi * nbins + bj], 1u);
        atomicAdd(&matrix[bj * nbins + bi], 1u);
    }
}

int launch_hash_detect(dem_ctx *ctx, int n, const double *x, const double *y, const double *z, const double *r,
                       double L, int periodic, int table_size, int32_t *pairs, int64_t cap, int64_t *counts,
                       cudaStream_t s, int even_cells) {
    // the limit from when the table was scanned (now a mask only, and the row counts are): 2^25 buckets, 2^24 droplets
    if (table_size > (int64_t)SCAN_MAX_BLOCKS * SCAN_TILE)
        return dem_set_error(ctx, DEM_E_CAPACITY, "scan: too many elements");
    int rc = dem_check_cuda(ctx, cudaMemsetAsync(counts, 0, 2 * sizeof(int64_t), s), "memset");
    if (rc || n == 0) return rc;
    const uint32_t buckets = search_buckets(n);
    // zeroed together: misc, row counts, bucket counts
    SearchMisc *misc = reinterpret_cast<SearchMisc *>(ctx->search_zero);
    int32_t *row_count = ctx->search_zero + SEARCH_MISC_WORDS, *bucket_count = row_count + n;
    SearchParams *sp = reinterpret_cast<SearchParams *>(ctx->dscratch + 2);
    static_assert(sizeof(SearchParams) <= 6 * sizeof(double), "dscratch[2..7]");
    rc = dem_check_cuda(ctx, cudaMemsetAsync(misc, 0, sizeof(int32_t) * (SEARCH_MISC_WORDS + (size_t)n + buckets), s),
                        "memset");
    if (rc) return rc;
    const int grid = max(1, min(ceil_div(n, 256), 8 * ctx->sm_count));
    dem_prof_begin(ctx, "hash_detect", s);
    radius_kernel<<<max(1, min(ceil_div(n, 1024), 4 * ctx->sm_count)), 256, 0, counted(s)>>>(
        n, r, L, 1.3 * L / std::cbrt((double)n), periodic, even_cells, misc, sp);
    search_assign_kernel<<<grid, 256, 0, counted(s)>>>(n, x, y, z, sp, buckets - 1, bucket_count, ctx->search_key);
    search_starts_kernel<<<ceil_div(buckets, SB_T * SB_ITEMS), SB_T, 0, counted(s)>>>(buckets, bucket_count, misc, sp,
                                                                                     ctx->search_bucket);
    search_scatter_kernel<<<grid, 256, 0, counted(s)>>>(n, x, y, z, r, sp, ctx->search_key, ctx->search_bucket,
                                                        ctx->search_rec);
    if ((rc = dem_check_launch(ctx, "hash search grid"))) return rc;
    SearchArgs a{};
    a.n = n;
    a.x = x;
    a.y = y;
    a.z = z;
    a.r = r;
    a.sp = sp;
    a.periodic = periodic;
    a.L = L;
    a.halfL = 0.5 * L;
    a.hash_mask = table_size - 1;
    a.mask = buckets - 1;
    a.bucket = ctx->search_bucket;
    a.rec = ctx->search_rec;
    a.misc = misc;
    a.row_count = row_count;
    // The list lies in the output where that is the larger place (every listed pair's final place is there, too), else
    // at the workspace's end.  Its rows take the workspace before it, from the search's own arrays on (no longer
    // needed when the list holds all pairs).
    const int64_t list_cap = ctx->search_list_cap;
    const bool out = cap > list_cap;
    const int64_t room = (char *)(ctx->search_list + (out ? 2 : 1) * list_cap) - (char *)ctx->search_key;
    a.list = out ? pairs : reinterpret_cast<int32_t *>(ctx->search_list + list_cap);
    a.list_cap = (uint32_t)std::min<int64_t>({out ? cap : list_cap, room / 4, INT_MAX});
    a.tmp = reinterpret_cast<int2 *>(ctx->search_key);
    a.tmp_cap = (uint32_t)std::min<int64_t>(room / 8, INT_MAX);
    a.cut = ctx->search_list;
    a.raw = reinterpret_cast<unsigned long long *>(counts + 1);
    // few droplets: fewer per warp, so that ~8 warps per SM share the search (N = 2,000: 14.7 -> 7.6 us with 4)
    int group = 32;
    while (group > 4 && ceil_div(n, group) < 8 * ctx->sm_count) group >>= 1;
    search_pairs_kernel<<<ceil_div(n, group * SP_WARPS), 32 * SP_WARPS, 0, counted(s)>>>(a, group);
    if ((rc = dem_check_launch(ctx, "hash search"))) return rc;
    rc = exclusive_scan<int32_t, int64_t>(ctx, row_count, ctx->pair_offset, n, s);
    if (rc) return rc;
    const int pgrid = max(1, min(ceil_div(n, group * PL_WARPS), 2 * ctx->sm_count));
    // At most 32 droplets' pairs per warp, whatever `group` is: its CTAs hold as much of an SM as a pass's do, and a pass
    // that starts beside it (the solver's speculative step) is spread over the SMs that they leave.  N = 2,000, FP64: with
    // 63 CTAs every eighth convection pass took 54 us, with 8 all take 38.6; found again, 40 pairs per droplet, 178 -> 521
    // (768 with the reference's buckets).  Three CTAs per SM, all that are resident: with two, N = 100,000 and 400,000 at
    // 28 pairs per droplet took 1,266 and 3,915 us, not 1,011 and 3,423.
    place_pairs_kernel<<<max(1, min(ceil_div(n, 32 * PL_WARPS), 3 * ctx->sm_count)), 32 * PL_WARPS, 0, counted(s)>>>(
        a, group, ctx->pair_offset, pairs, cap);
    write_rows_kernel<<<pgrid, 256, 0, counted(s)>>>(a, ctx->pair_offset, pairs, cap, counts, ctx->d_err);
    dem_prof_end(ctx, s);
    return dem_check_launch(ctx, "hash write");
}

}  // namespace dem

// ===========================================================================
// Allocation-free variant of the spatial-hash detector.
//
// Some callers cannot call cudaMalloc at the time they detect collisions: a
// host application that hands the library a fixed device-memory budget up
// front and forbids later allocations, a control loop that must not take the
// device-wide synchronisation and latency jitter of cudaMalloc/cudaFree
// between steps, or code that runs while another component owns the CUDA
// allocator.  For them dem_hash_detect_noalloc needs no context and allocates
// nothing: its workspace (bucket table, per-droplet hashes, bucket members,
// per-droplet pair counts and offsets, scan totals) is the file-scope device
// array below, sized for at most NOALLOC_MAX_N droplets and a hash table of at
// most NOALLOC_MAX_TABLE buckets.  Every GPU that loads the library keeps this
// array (about 2.9 MB) until the process exits.
// ===========================================================================
#include <mutex>

namespace dem {

constexpr int NOALLOC_MAX_N = 65536;
constexpr int NOALLOC_MAX_TABLE = 131072;  // next power of two >= 2 * NOALLOC_MAX_N
constexpr int NOALLOC_MAX_DEVICES = 64;

constexpr size_t na_align(size_t b) { return (b + 255) & ~size_t(255); }
constexpr size_t NA_CELL = 0;                                                      // int32[MAX_N]
constexpr size_t NA_SORTED = NA_CELL + na_align(sizeof(int32_t) * NOALLOC_MAX_N);    // int32[MAX_N]
constexpr size_t NA_PCOUNT = NA_SORTED + na_align(sizeof(int32_t) * NOALLOC_MAX_N);  // int32[MAX_N + 1]
constexpr size_t NA_POFF = NA_PCOUNT + na_align(sizeof(int32_t) * (NOALLOC_MAX_N + 1));       // int64[MAX_N + 1]
constexpr size_t NA_BCOUNT = NA_POFF + na_align(sizeof(int64_t) * (NOALLOC_MAX_N + 1));       // int32[MAX_TABLE]
constexpr size_t NA_BSTART = NA_BCOUNT + na_align(sizeof(int32_t) * NOALLOC_MAX_TABLE);       // int32[MAX_TABLE + 1]
constexpr size_t NA_BCURSOR = NA_BSTART + na_align(sizeof(int32_t) * (NOALLOC_MAX_TABLE + 1));  // int32[MAX_TABLE]
constexpr size_t NA_SUMS = NA_BCURSOR + na_align(sizeof(int32_t) * NOALLOC_MAX_TABLE);  // int64[SCAN_MAX_BLOCKS + 1]
constexpr size_t NA_MISC = NA_SUMS + na_align(sizeof(int64_t) * (SCAN_MAX_BLOCKS + 1));  // max slot, params, err
constexpr size_t NA_BYTES = NA_MISC + 256;

static __device__ __align__(256) unsigned char g_noalloc_scratch[NA_BYTES];

struct NoallocDevice {
    unsigned char *scratch = nullptr;  // device address of g_noalloc_scratch on this device
    int sm_count = 0;
};
static NoallocDevice g_noalloc_dev[NOALLOC_MAX_DEVICES];
static std::mutex g_noalloc_mutex;

// Once per device, with that device current: the device address of the array.
// (In host code g_noalloc_scratch names a host-side stand-in, not device memory.)
static int noalloc_setup(NoallocDevice &out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return DEM_E_CUDA;
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return DEM_E_INVALID;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    NoallocDevice &d = g_noalloc_dev[dev];
    if (!d.scratch) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return DEM_E_CUDA;
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return DEM_E_CUDA;
        d.sm_count = sms > 0 ? sms : 1;
        d.scratch = static_cast<unsigned char *>(p);
    }
    out = d;
    return DEM_OK;
}

}  // namespace dem

extern "C" int dem_hash_detect_noalloc(int n, const double *x, const double *y, const double *z, const double *r,
                                       double L, int periodic, int table_size, int32_t *pairs,
                                       int64_t pair_capacity, int64_t *counts, void *stream) {
    using namespace dem;
    if (n < 0 || n > NOALLOC_MAX_N) return DEM_E_CAPACITY;
    if (table_size < 1 || table_size > NOALLOC_MAX_TABLE || (table_size & (table_size - 1))) return DEM_E_CAPACITY;
    if (!counts || pair_capacity < 0 || (pair_capacity > 0 && !pairs)) return DEM_E_INVALID;
    if (n > 0 && (!x || !y || !z || !r)) return DEM_E_INVALID;
    NoallocDevice d;
    int rc = noalloc_setup(d);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    unsigned char *base = d.scratch;
    int32_t *cell_hash = reinterpret_cast<int32_t *>(base + NA_CELL);
    int32_t *sorted_idx = reinterpret_cast<int32_t *>(base + NA_SORTED);
    int32_t *pair_count = reinterpret_cast<int32_t *>(base + NA_PCOUNT);
    int64_t *pair_offset = reinterpret_cast<int64_t *>(base + NA_POFF);
    int32_t *bucket_count = reinterpret_cast<int32_t *>(base + NA_BCOUNT);
    int32_t *bucket_start = reinterpret_cast<int32_t *>(base + NA_BSTART);
    int32_t *bucket_cursor = reinterpret_cast<int32_t *>(base + NA_BCURSOR);
    void *sums = base + NA_SUMS;
    unsigned long long *slot = reinterpret_cast<unsigned long long *>(base + NA_MISC);
    HashParams *hp = reinterpret_cast<HashParams *>(base + NA_MISC + 16);
    uint32_t *err = reinterpret_cast<uint32_t *>(base + NA_MISC + 64);
    const int32_t mask = table_size - 1;
    const int grid = max(1, min(ceil_div(n, 256), 8 * d.sm_count));
    // the array keeps the previous call's contents: reset what must start at zero
    if (cudaMemsetAsync(base + NA_MISC, 0, 256, s) != cudaSuccess) return DEM_E_CUDA;
    if (cudaMemsetAsync(counts, 0, 2 * sizeof(int64_t), s) != cudaSuccess) return DEM_E_CUDA;
    if (cudaMemsetAsync(bucket_count, 0, sizeof(int32_t) * table_size, s) != cudaSuccess) return DEM_E_CUDA;
    if (n == 0) return DEM_OK;
    max_kernel<<<grid, 256, 0, counted(s)>>>(n, r, slot);
    hash_params_kernel<<<1, 1, 0, counted(s)>>>(slot, L, hp);
    assign_kernel<<<grid, 256, 0, counted(s)>>>(n, x, y, z, hp, periodic, mask, cell_hash, bucket_count);
    if (cudaGetLastError() != cudaSuccess) return DEM_E_CUDA;
    if (exclusive_scan_into<int32_t, int32_t>(bucket_count, bucket_start, table_size, static_cast<int32_t *>(sums),
                                              s) != cudaSuccess)
        return DEM_E_CUDA;
    if (cudaMemcpyAsync(bucket_cursor, bucket_start, sizeof(int32_t) * table_size, cudaMemcpyDeviceToDevice, s) !=
        cudaSuccess)
        return DEM_E_CUDA;
    scatter_kernel<<<grid, 256, 0, counted(s)>>>(n, cell_hash, hp, bucket_cursor, sorted_idx);
    const int dgrid = ceil_div(n, 128);
    count_pairs_kernel<<<dgrid, 128, 0, counted(s)>>>(n, x, y, z, r, hp, periodic, L, mask,
                                                             bucket_start, sorted_idx, pair_count,
                                                             reinterpret_cast<unsigned long long *>(counts + 1));
    if (cudaGetLastError() != cudaSuccess) return DEM_E_CUDA;
    if (exclusive_scan_into<int32_t, int64_t>(pair_count, pair_offset, n, static_cast<int64_t *>(sums), s) !=
        cudaSuccess)
        return DEM_E_CUDA;
    write_pairs_kernel<<<dgrid, 128, 0, counted(s)>>>(n, x, y, z, r, hp, periodic, L, mask,
                                                             bucket_start, sorted_idx, pair_offset, pairs,
                                                             pair_capacity, counts, err);
    return cudaGetLastError() == cudaSuccess ? DEM_OK : DEM_E_CUDA;
}

extern "C" int dem_pair_bin_matrix(dem_ctx *ctx, const int32_t *pairs, const int64_t *num_pairs, int64_t pair_capacity,
                                   const int32_t *bins, int nbins, uint32_t *matrix, void *stream) {
    if (!ctx || nbins < 1 || !matrix || !num_pairs || pair_capacity < 0) return DEM_E_INVALID;
    if (pair_capacity > 0 && (!pairs || !bins)) return DEM_E_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    int rc = dem_check_cuda(ctx, cudaMemsetAsync(matrix, 0, sizeof(uint32_t) * nbins * nbins, s), "memset");
    if (rc || pair_capacity == 0) return rc;
    const int grid = (int)std::min<int64_t>((pair_capacity + 255) / 256, 8LL * ctx->sm_count);
    dem::pair_bin_kernel<<<grid, 256, 0, counted(s)>>>(pairs, num_pairs, pair_capacity, bins, nbins, matrix);
    return dem_check_launch(ctx, "pair bin matrix");
}
