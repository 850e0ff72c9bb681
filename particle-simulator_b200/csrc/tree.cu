// tree.cu -- flat Barnes-Hut octree (reference drop-in), FP64.
//
// Restates FlatOctree (dem/octree/flat_tree.py:36-1630, dem/octree/octree_node.py)
// on the device with the same tree, node numbering and arithmetic:
//   build            :180-246  level by level; the serial subdivision loop
//                              (:309-354) becomes a scan over the level's nodes
//                              (the first k candidates in node order get
//                              children, k limited by the node pool exactly as
//                              the serial `base + 8 > max_nodes` test does)
//   leaf slots       :371-397  leaves in node order, particles ascending inside
//   next pointers    :400-463  per level, top-down
//   R^3 aggregates   :469-554  leaves in particle order, parents in octant order
//   force walk       :783-894  stackless walk, MAC s^2 < theta^2 D^2
//   force moments    :696-777  sum F and P_ab = sum x_a F_b
//   velocity walks   :1000-1280 (Stokeslet) and :1326-1588 (total velocity)
// Every walk visits nodes in the reference's order and accumulates in the
// reference's order; the file is compiled with -fmad=false, so forces and
// velocities are bit-identical to the reference expressions in IEEE binary64.
#include <vector>

#include "common.cuh"
#include "corr.cuh"
#include "scan.cuh"

constexpr int WALK_T = 128;  // threads per CTA of the walks
constexpr size_t WALK_REC_BYTES = 64, WALK_DIP_BYTES = 96;

struct dem_tree {
    dem_ctx *ctx = nullptr;  // must outlive the tree while kernels run; destroy does not touch it
    int device = 0;
    int cap = 0, max_nodes = 0;
    int n = 0, node_count = 0, parent_count = 0, leaf_slot_count = 0, pool_exhausted = 0;
    double L = 0;
    int periodic = 0;
    std::vector<int> level_off;
    // nodes
    double *mn = nullptr, *mx = nullptr;   // [3][M]
    double *R3 = nullptr;                  // [4][M]: sum, x, y, z
    double *maxr = nullptr;                // [M]
    double *fs = nullptr;                  // [12][M]: F(3), P_ab(9)
    int32_t *first_child = nullptr, *next = nullptr, *leaf_start = nullptr, *count = nullptr;
    int32_t *child_cnt = nullptr;          // [M][8]
    int32_t *parents = nullptr, *parent_fc = nullptr;
    int32_t *flag = nullptr, *rank = nullptr;  // [M + 1]
    int32_t *fill = nullptr;               // [M]
    // particles
    double *p = nullptr;                   // [4][N]: x, y, z, r
    double *pf = nullptr;                  // [3][N]: forces of the last force walk
    int32_t *part_node = nullptr, *part_oct = nullptr, *leaf_idx = nullptr;
    // walk records (walk_records_kernel) and droplets in leaf-slot order
    char *rec_f = nullptr, *rec_v = nullptr, *rec_d = nullptr;  // [M]
    double2 *slot_p = nullptr, *slot_f = nullptr;               // [N][2]: (x, y), (z, r); (Fx, Fy), (Fz, -)
    int32_t *roots = nullptr;              // [2]: where the force / velocity walk starts
    bool built = false;                    // the last build completed
    bool vel_records = false;              // rec_v / rec_d belong to this build
    int32_t *h_total = nullptr;            // pinned
    const dem_corr *corr = nullptr;        // periodic-image correction (borrowed), or none
};

namespace dem {

// Plain view of the tree passed to the kernels by value.
struct TreeDev {
    int cap, max_nodes, n, node_count, periodic;
    double L;
    double *mn, *mx, *R3, *maxr, *fs;
    int32_t *first_child, *next, *leaf_start, *count, *child_cnt, *parents, *parent_fc, *flag, *rank, *fill;
    double *p, *pf;
    int32_t *part_node, *part_oct, *leaf_idx;
    char *rec_f, *rec_v, *rec_d;
    double2 *slot_p, *slot_f;
    int32_t *roots;
    uint32_t *err;
};

static TreeDev view(const dem_tree *t) {
    TreeDev v;
    v.cap = t->cap;
    v.max_nodes = t->max_nodes;
    v.n = t->n;
    v.node_count = t->node_count;
    v.periodic = t->periodic;
    v.L = t->L;
    v.mn = t->mn;
    v.mx = t->mx;
    v.R3 = t->R3;
    v.maxr = t->maxr;
    v.fs = t->fs;
    v.first_child = t->first_child;
    v.next = t->next;
    v.leaf_start = t->leaf_start;
    v.count = t->count;
    v.child_cnt = t->child_cnt;
    v.parents = t->parents;
    v.parent_fc = t->parent_fc;
    v.flag = t->flag;
    v.rank = t->rank;
    v.fill = t->fill;
    v.p = t->p;
    v.pf = t->pf;
    v.part_node = t->part_node;
    v.part_oct = t->part_oct;
    v.leaf_idx = t->leaf_idx;
    v.rec_f = t->rec_f;
    v.rec_v = t->rec_v;
    v.rec_d = t->rec_d;
    v.slot_p = t->slot_p;
    v.slot_f = t->slot_f;
    v.roots = t->roots;
    v.err = t->ctx->d_err;
    return v;
}

__device__ __forceinline__ double node_size(const double *mn, const double *mx, int M, int k) {
    const double dx = mx[k] - mn[k], dy = mx[M + k] - mn[M + k], dz = mx[2 * M + k] - mn[2 * M + k];
    const double m = dx >= dy ? dx : dy;  // ti.max
    return m >= dz ? m : dz;
}

__device__ __forceinline__ void node_center(const double *mn, const double *mx, const double *R3, int M, int k,
                                            double &cx, double &cy, double &cz) {
    if (R3[k] > 0.0) {
        const double inv = 1.0 / R3[k];
        cx = R3[M + k] * inv;
        cy = R3[2 * M + k] * inv;
        cz = R3[3 * M + k] * inv;
    } else {
        cx = (mn[k] + mx[k]) * 0.5;
        cy = (mn[M + k] + mx[M + k]) * 0.5;
        cz = (mn[2 * M + k] + mx[2 * M + k]) * 0.5;
    }
}

// ---------------------------------------------------------------------------
// build
// ---------------------------------------------------------------------------
__global__ void tree_init_kernel(TreeDev t, int n, double L, const double *__restrict__ x,
                                 const double *__restrict__ y, const double *__restrict__ z,
                                 const double *__restrict__ r) {
    const int M = t.max_nodes, N = t.cap;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        t.p[i] = x[i];
        t.p[N + i] = y[i];
        t.p[2 * N + i] = z[i];
        t.p[3 * N + i] = r[i];
        t.part_node[i] = 0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // _init_root_kernel :249-270
        for (int a = 0; a < 3; ++a) {
            t.mn[a * M] = 0.0;
            t.mx[a * M] = L;
        }
        t.first_child[0] = -1;
        t.next[0] = -1;
        t.leaf_start[0] = -1;
        t.count[0] = n;
        for (int a = 0; a < 4; ++a) t.R3[a * M] = 0.0;
        t.fs[0] = t.fs[M] = t.fs[2 * M] = 0.0;
    }
}

__global__ void zero_child_cnt_kernel(int32_t *child_cnt, int ls, int le) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < (le - ls) * 8; k += gridDim.x * blockDim.x)
        child_cnt[(size_t)ls * 8 + k] = 0;
}

// _level_assign_octants :284-306 (octree_node.py:84-95).  In the first two levels many lanes of a warp fall into one
// octant and count as one: atomics on 8 or 64 counters took 16 and 24 us at N = 100,003, 4 and 15 now (64 nodes:
// 15 either way).
constexpr int FEW_NODES = 8;
__global__ void assign_octants_kernel(TreeDev t, int n, int ls, int le) {
    const int M = t.max_nodes, N = t.cap;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int node = t.part_node[i];
        if (node >= ls && node < le) {
            const double cx = (t.mn[node] + t.mx[node]) * 0.5;
            const double cy = (t.mn[M + node] + t.mx[M + node]) * 0.5;
            const double cz = (t.mn[2 * M + node] + t.mx[2 * M + node]) * 0.5;
            int o = 0;
            if (t.p[i] >= cx) o |= 1;
            if (t.p[N + i] >= cy) o |= 2;
            if (t.p[2 * N + i] >= cz) o |= 4;
            t.part_oct[i] = o;
            if (le - ls <= FEW_NODES) {
                const unsigned peers = __match_any_sync(__activemask(), node * 8 + o);
                if ((peers & ((1u << (threadIdx.x & 31)) - 1u)) == 0)
                    atomicAdd(&t.child_cnt[(size_t)node * 8 + o], __popc(peers));
            } else {
                atomicAdd(&t.child_cnt[(size_t)node * 8 + o], 1);
            }
        }
    }
}

__global__ void subdivide_flags_kernel(TreeDev t, int ls, int le, int mpl) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < le - ls; k += gridDim.x * blockDim.x) {
        const int node = ls + k;
        t.flag[k] = (t.first_child[node] < 0 && t.count[node] > mpl) ? 1 : 0;
    }
}

// _level_subdivide_and_alloc :309-354 for the first `sub` candidates: a thread per child, so that neighbouring
// lanes fill neighbouring entries of the node arrays (a thread per parent: 152 us over the levels of N = 100,003, one droplet
// per leaf; 44 now)
__global__ void subdivide_kernel(TreeDev t, int ls, int le, int sub, int node_count, int parent_count) {
    const int M = t.max_nodes;
    const long long width = 8LL * (le - ls), stride = (long long)gridDim.x * blockDim.x;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < width; e += stride) {
        const int k = (int)(e >> 3), o = (int)(e & 7);
        if (!t.flag[k]) continue;
        const int q = t.rank[k];
        if (q >= sub) continue;
        const int node = ls + k;
        const int base = node_count + 8 * q, child = base + o;
        if (o == 0) {
            t.first_child[node] = base;
            t.parents[parent_count + q] = node;
            t.parent_fc[parent_count + q] = base;
        }
        for (int a = 0; a < 3; ++a) {
            const double lo = t.mn[a * M + node], hi = t.mx[a * M + node], c = (lo + hi) * 0.5;
            const bool up = (o >> a) & 1;
            t.mn[a * M + child] = up ? c : lo;
            t.mx[a * M + child] = up ? hi : c;
        }
        t.first_child[child] = -1;  // init_node, octree_node.py:117-154
        t.next[child] = -1;
        t.leaf_start[child] = -1;
        t.count[child] = t.child_cnt[(size_t)node * 8 + o];
        for (int a = 0; a < 4; ++a) t.R3[a * M + child] = 0.0;
        t.maxr[child] = 0.0;
        for (int a = 0; a < 12; ++a) t.fs[a * M + child] = 0.0;
    }
}

// _level_scatter :357-366
__global__ void level_scatter_kernel(TreeDev t, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int node = t.part_node[i];
        if (node >= 0 && t.first_child[node] >= 0) t.part_node[i] = t.first_child[node] + t.part_oct[i];
    }
}

__global__ void leaf_flags_kernel(TreeDev t, int nc) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nc; k += gridDim.x * blockDim.x) {
        t.flag[k] = (t.first_child[k] < 0 && t.count[k] > 0) ? t.count[k] : 0;
        t.fill[k] = 0;
    }
}

// _finalize_leaves_alloc :371-385 (slots in node order)
__global__ void leaf_start_kernel(TreeDev t, int nc) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nc; k += gridDim.x * blockDim.x)
        if (t.first_child[k] < 0 && t.count[k] > 0) t.leaf_start[k] = t.rank[k];
}

// _finalize_leaves_scatter :388-397
__global__ void leaf_scatter_kernel(TreeDev t, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int node = t.part_node[i];
        if (node >= 0 && t.first_child[node] < 0) {
            const int l0 = t.leaf_start[node];
            if (l0 >= 0) t.leaf_idx[l0 + atomicAdd(&t.fill[node], 1)] = i;
        }
    }
}

// particles of a leaf in ascending index order (the reference fills leaves serially)
__global__ void leaf_sort_kernel(TreeDev t, int nc) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nc; k += gridDim.x * blockDim.x) {
        if (!(t.first_child[k] < 0 && t.count[k] > 1 && t.leaf_start[k] >= 0)) continue;
        int32_t *a = t.leaf_idx + t.leaf_start[k];
        const int c = t.count[k];
        for (int u = 1; u < c; ++u) {
            const int32_t v = a[u];
            int w = u - 1;
            while (w >= 0 && a[w] > v) {
                a[w + 1] = a[w];
                --w;
            }
            a[w + 1] = v;
        }
    }
}

// _build_next_pointers_pass1 :400-415
__global__ void next_pass1_kernel(TreeDev t, int a, int b) {
    for (int i = a + blockIdx.x * blockDim.x + threadIdx.x; i < b; i += gridDim.x * blockDim.x) {
        const int parent = t.parents[i], base = t.parent_fc[i];
        const int pn = t.next[parent];
        for (int o = 0; o < 8; ++o) t.next[base + o] = (o == 7) ? pn : base + o + 1;
    }
}

// _build_next_pointers_pass2 :418-446
__global__ void next_pass2_kernel(TreeDev t, int a, int b) {
    for (int i = a + blockIdx.x * blockDim.x + threadIdx.x; i < b; i += gridDim.x * blockDim.x) {
        const int parent = t.parents[i], base = t.parent_fc[i];
        if (t.count[parent] == 0) {
            t.first_child[parent] = t.next[parent];
            continue;
        }
        int first = -1, last = -1;
        for (int j = 0; j < 8; ++j) {
            const int c = base + j;
            if (t.count[c] > 0) {
                if (first < 0) {
                    first = last = c;
                } else {
                    t.next[last] = c;
                    last = c;
                }
            }
        }
        if (last >= 0) {
            t.next[last] = t.next[parent];
            t.first_child[parent] = first;
        }
    }
}

// _init_leaf_r3 :470-511
__global__ void leaf_r3_kernel(TreeDev t, int nc) {
    const int M = t.max_nodes, N = t.cap;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nc; k += gridDim.x * blockDim.x) {
        double s = 0, wx = 0, wy = 0, wz = 0, mr = 0;
        if (t.first_child[k] < 0 && t.count[k] > 0 && t.leaf_start[k] >= 0) {
            const int l0 = t.leaf_start[k], c = t.count[k];
            for (int q = 0; q < c; ++q) {
                const int i = t.leaf_idx[l0 + q];
                if (i >= 0) {
                    const double ri = t.p[3 * N + i];
                    const double r3 = ipow3(ri);
                    s += r3;
                    wx += t.p[i] * r3;
                    wy += t.p[N + i] * r3;
                    wz += t.p[2 * N + i] * r3;
                    if (ri > mr) mr = ri;
                }
            }
        }
        t.R3[k] = s;
        t.R3[M + k] = wx;
        t.R3[2 * M + k] = wy;
        t.R3[3 * M + k] = wz;
        t.maxr[k] = mr;
        t.fs[k] = t.fs[M + k] = t.fs[2 * M + k] = 0.0;
    }
}

// _sweep_r3_level :514-542
__global__ void sweep_r3_kernel(TreeDev t, int a, int b) {
    const int M = t.max_nodes;
    for (int i = a + blockIdx.x * blockDim.x + threadIdx.x; i < b; i += gridDim.x * blockDim.x) {
        const int parent = t.parents[i], base = t.parent_fc[i];
        double s = 0, wx = 0, wy = 0, wz = 0, mr = 0;
        for (int j = 0; j < 8; ++j) {
            const int c = base + j;
            if (t.count[c] > 0) {
                s += t.R3[c];
                wx += t.R3[M + c];
                wy += t.R3[2 * M + c];
                wz += t.R3[3 * M + c];
                if (t.maxr[c] > mr) mr = t.maxr[c];
            }
        }
        t.R3[parent] = s;
        t.R3[M + parent] = wx;
        t.R3[2 * M + parent] = wy;
        t.R3[3 * M + parent] = wz;
        t.maxr[parent] = mr;
    }
}

// _init_leaf_forces(_from_fields) :556-627, :696-766
__global__ void leaf_forces_kernel(TreeDev t, int nc, const double *__restrict__ fx, const double *__restrict__ fy,
                                   const double *__restrict__ fz) {
    const int M = t.max_nodes, N = t.cap;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nc; k += gridDim.x * blockDim.x) {
        double s[3] = {0, 0, 0}, P[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        if (t.first_child[k] < 0 && t.count[k] > 0 && t.leaf_start[k] >= 0) {
            const int l0 = t.leaf_start[k], c = t.count[k];
            for (int q = 0; q < c; ++q) {
                const int i = t.leaf_idx[l0 + q];
                if (i >= 0) {
                    const double f[3] = {fx[i], fy[i], fz[i]};
                    const double xx[3] = {t.p[i], t.p[N + i], t.p[2 * N + i]};
                    s[0] += f[0];
                    s[1] += f[1];
                    s[2] += f[2];
                    for (int u = 0; u < 3; ++u)
                        for (int v = 0; v < 3; ++v) P[3 * u + v] += xx[u] * f[v];
                }
            }
        }
        for (int u = 0; u < 3; ++u) t.fs[u * M + k] = s[u];
        for (int u = 0; u < 9; ++u) t.fs[(3 + u) * M + k] = P[u];
    }
}

// _sweep_forces_level :629-672: moment blockIdx.y of a parent per thread, children in order (N = 100,003: 103 us for
// all levels with a thread's twelve sums per parent, 29 now)
__global__ void sweep_forces_kernel(TreeDev t, int a, int b) {
    double *const fs = t.fs + (size_t)blockIdx.y * t.max_nodes;
    for (int i = a + blockIdx.x * blockDim.x + threadIdx.x; i < b; i += gridDim.x * blockDim.x) {
        const int base = t.parent_fc[i];
        double acc = 0;
        for (int j = 0; j < 8; ++j) {
            const int c = base + j;
            if (t.count[c] > 0) acc += fs[c];
        }
        fs[t.parents[i]] = acc;
    }
}

// ---------------------------------------------------------------------------
// Walk records.  A walk visits a node through one 64-byte record (two loads): the size
// squared and the centre (the same expressions the reference evaluates at every
// visit, :466-520, evaluated once), what the accepted node needs, and two links
// that leave out the nodes the walk passes over without a term (empty, R^3 sum
// below 1e-30 :861, squared force sum below 1e-60 :1155; half the nodes of a tree
// of one droplet per leaf): the first of its children that is not passed over
// (or what follows them), and the next node when it is done.  Links: -1 the end;
// child <= -2 marks a leaf whose first slot is -2 - child.
// ---------------------------------------------------------------------------
struct __align__(32) ForceRec {
    double s2, cx, cy, cz, r3;
    int32_t child, next, count, pad[3];
};
struct __align__(32) VelRec {
    double s2, cx, cy, cz;
    int32_t child, next;
    double fx, fy, fz;
};
// Dipole D_ab = P_ab - c_a F_b about the centre (:1215-1230) and its trace.
struct __align__(32) DipRec {
    double d[9], tr, pad[2];
};
static_assert(sizeof(ForceRec) == WALK_REC_BYTES && sizeof(VelRec) == WALK_REC_BYTES && sizeof(DipRec) == WALK_DIP_BYTES,
              "the tree's allocation");

// Half a record or one droplet: 32 bytes (so aligned) in one 256-bit load.
struct Half {
    double a, b, c, d;
};
__device__ __forceinline__ Half half_at(const void *p, int k) {
    Half h;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(h.a), "=d"(h.b), "=d"(h.c), "=d"(h.d)
        : "l"((const char *)p + 32 * (size_t)k));
    return h;
}

template <bool FORCE>
__device__ __forceinline__ bool passed_over(const TreeDev &t, int k) {
    if (t.count[k] == 0) return true;
    if (FORCE) return t.R3[k] < 1e-30;
    const size_t M = t.max_nodes;
    const double fx = t.fs[k], fy = t.fs[M + k], fz = t.fs[2 * M + k];
    return fx * fx + fy * fy + fz * fz < 1e-60;
}

// The first node from k on that has a term or is opened (a walk that met k, or any node it passes over).
template <bool FORCE>
__device__ __forceinline__ int first_kept(const TreeDev &t, int k) {
    for (int steps = 0; k >= 0 && passed_over<FORCE>(t, k); k = t.next[k])
        if (++steps > t.node_count) return -1;  // broken links: the walk's own bound reports them
    return k;
}

template <bool FORCE>
__global__ void walk_records_kernel(TreeDev t, int nc, int32_t *__restrict__ root) {
    const int M = t.max_nodes;
    if (blockIdx.x == 0 && threadIdx.x == 0) *root = first_kept<FORCE>(t, 0);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nc; k += gridDim.x * blockDim.x) {
        if (passed_over<FORCE>(t, k)) continue;  // no walk loads its record
        const double s = node_size(t.mn, t.mx, M, k);
        double cx, cy, cz;
        node_center(t.mn, t.mx, t.R3, M, k, cx, cy, cz);
        const int fc = t.first_child[k];
        const int child = fc < 0 ? -2 - t.leaf_start[k] : first_kept<FORCE>(t, fc);
        const int next = first_kept<FORCE>(t, t.next[k]);
        if (FORCE) {
            ForceRec *const o = reinterpret_cast<ForceRec *>(t.rec_f) + k;
            *o = ForceRec{s * s, cx, cy, cz, t.R3[k], child, next, t.count[k], {0, 0, 0}};
        } else {
            const double Fx = t.fs[k], Fy = t.fs[M + k], Fz = t.fs[2 * (size_t)M + k];
            reinterpret_cast<VelRec *>(t.rec_v)[k] = VelRec{s * s, cx, cy, cz, child, next, Fx, Fy, Fz};
            const double *P = t.fs + 3 * (size_t)M;
            DipRec d;
            const double c[3] = {cx, cy, cz}, F[3] = {Fx, Fy, Fz};
#pragma unroll
            for (int q = 0; q < 9; ++q) d.d[q] = P[(size_t)q * M + k] - c[q / 3] * F[q % 3];
            d.tr = d.d[0] + d.d[4] + d.d[8];
            reinterpret_cast<DipRec *>(t.rec_d)[k] = d;
        }
    }
}

// Droplets (x, y, z, r) in leaf-slot order; with fx: their forces.
__global__ void slot_droplets_kernel(TreeDev t, int n) {
    const size_t N = t.cap;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const int j = t.leaf_idx[s];
        t.slot_p[2 * (size_t)s] = make_double2(t.p[j], t.p[N + j]);
        t.slot_p[2 * (size_t)s + 1] = make_double2(t.p[2 * N + j], t.p[3 * N + j]);
    }
}
__global__ void slot_forces_kernel(TreeDev t, int n, const double *__restrict__ fx, const double *__restrict__ fy,
                                   const double *__restrict__ fz) {
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const int j = t.leaf_idx[s];
        t.slot_f[2 * (size_t)s] = make_double2(fx[j], fy[j]);
        t.slot_f[2 * (size_t)s + 1] = make_double2(fz[j], 0.0);
    }
}

// The walks.  One thread per target, in leaf-slot order (a permutation of all n particles: every particle
// ends in a leaf), so the lanes of a warp walk neighbouring targets along nearly the same path; each
// target's sums are its own thread's, in the reference's order, whatever order the targets are taken in.
// A lane first goes on to its next term -- an accepted node or a pair of a leaf -- and the warp then
// evaluates the lanes' terms together (a node's and a pair's force have the same form).
//
// Bound: latency (a visit's record, a chain of FP64 operations) and divergence (13 of 32 lanes active on
// average): 21 warps per SM are all there is at N = 100,000.  N = 100,003, one droplet per leaf, open, force /
// total-velocity walk: 2.00 / 3.54 ms with 11 to 23 scattered loads and a division per visit, half of the
// visits on empty nodes; 1.24 / 2.13 ms with records, links past those nodes and terms taken together, 1.19 /
// 1.96 with 256-bit loads (a diverged warp's loads pass the L1 a line at a time: two per visit instead of
// four); 16 droplets per leaf, periodic: 11.5 / 15.0 -> 5.5 / 7.6.  CTAs of 32 threads: 2 % faster there with
// one droplet per leaf, 5 to 10 % slower at N = 2,000.
// (Loading the next node's record before a term is evaluated: 1.39 / 2.22, the loads wait all the same.)
template <bool PER>
__device__ __forceinline__ void image64x3(double &dx, double &dy, double &dz, double L, double halfL) {
    if (PER) {
        dx = mic64(dx, L, halfL);
        dy = mic64(dy, L, halfL);
        dz = mic64(dz, L, halfL);
    }
}

// _compute_forces_kernel :783-894
template <bool PER>
__global__ void __launch_bounds__(WALK_T) force_walk_kernel(TreeDev t, double m_const, double theta_sq,
                                                            double *__restrict__ fx, double *__restrict__ fy,
                                                            double *__restrict__ fz) {
    const int N = t.cap, n = t.n;
    const double L = t.L, halfL = 0.5 * t.L;
    const char *const rec = t.rec_f;
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= n) return;
    const int i = t.leaf_idx[slot];
    const double2 pa = t.slot_p[2 * (size_t)slot], pb = t.slot_p[2 * (size_t)slot + 1];
    const double xi = pa.x, yi = pa.y, zi = pb.x, ri = pb.y;
    const double mri3 = m_const * ipow3(ri);
    double Fx = 0, Fy = 0, Fz = 0;
    int node = t.roots[0], k = 0, kend = 0;
    int steps = 0;  // every node is visited at most once; more means broken links
    while (true) {
        double dx, dy, dz, d_sq, w;
        bool term = false;
        while (k < kend || node >= 0) {
            if (k < kend) {
                const int s = k++;
                if (s == slot) continue;
                const Half q = half_at(t.slot_p, s);
                dx = q.a - xi, dy = q.b - yi, dz = q.c - zi;
                image64x3<PER>(dx, dy, dz, L, halfL);
                d_sq = dx * dx + dy * dy + dz * dz;
                const double r_sum = ri + q.d;
                if (!(d_sq >= r_sum * r_sum)) continue;
                w = ipow3(q.d);
                term = true;
                break;
            }
            if (++steps > t.node_count + 1) {
                raise_device_error(t.err, DEM_DEVERR_NODE_OVERFLOW);
                node = -1;
                break;
            }
            const Half q = half_at(rec, 2 * node), l = half_at(rec, 2 * node + 1);  // size^2, centre | R^3, links, count
            const int child = __double2loint(l.b), next = __double2hiint(l.b);
            if (child <= -2) {
                k = -2 - child;
                kend = k + __double2loint(l.c);
                node = next;
                continue;
            }
            dx = q.b - xi, dy = q.c - yi, dz = q.d - zi;
            image64x3<PER>(dx, dy, dz, L, halfL);
            d_sq = dx * dx + dy * dy + dz * dz;
            if (q.a < theta_sq * d_sq && d_sq > 0.0) {
                w = l.a;
                node = next;
                term = true;
                break;
            }
            node = child;
        }
        if (!term) break;
        const double rr = sqrt(d_sq);
        const double r7 = d_sq * d_sq * d_sq * rr;
        const double factor = mri3 * w / r7;
        const double dx2 = dx * dx, dy2 = dy * dy, dz2 = dz * dz;
        const double ang = 4.0 * dz2 - dx2 - dy2;
        Fx += factor * dx * ang;
        Fy += factor * dy * ang;
        Fz += factor * dz * (2.0 * dz2 - 3.0 * dx2 - 3.0 * dy2);
    }
    fx[i] = Fx;
    fy[i] = Fy;
    fz[i] = Fz;
    t.pf[i] = Fx;
    t.pf[N + i] = Fy;
    t.pf[2 * (size_t)N + i] = Fz;
}

// _compute_stokeslet_kernel :1000-1280 (stokes <= 0) and
// _compute_total_velocity_kernel :1326-1588 (stokes > 0); with CORR the
// periodic-image correction after every leaf pair (:1070-1131) and accepted
// node (:1171-1213), and the self term of the Stokeslet walk (:1271-1276).
template <bool PER, bool CORR>
__global__ void __launch_bounds__(WALK_T) velocity_walk_kernel(TreeDev t, const double *__restrict__ Fx_,
                                                               const double *__restrict__ Fy_,
                                                               const double *__restrict__ Fz_, double eta,
                                                               double theta_sq, double stokes, CorrDev corr,
                                                               double *__restrict__ vx, double *__restrict__ vy,
                                                               double *__restrict__ vz) {
    const int N = t.cap, n = t.n;
    const double L = t.L, halfL = 0.5 * t.L;
    const char *const rec = t.rec_v;
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= n) return;
    const int i = t.leaf_idx[slot];
    const double2 pa = t.slot_p[2 * (size_t)slot], pb = t.slot_p[2 * (size_t)slot + 1];
    const double xi = pa.x, yi = pa.y, zi = pb.x, ri = pb.y;
    double ux = 0, uy = 0, uz = 0;
    if (stokes > 0) {
        const double inv_stokes_r = 1.0 / (stokes * ri);
        ux = t.pf[i] * inv_stokes_r;
        uy = t.pf[N + i] * inv_stokes_r;
        uz = t.pf[2 * (size_t)N + i] * inv_stokes_r;
    }
    int node = t.roots[1], k = 0, kend = 0;
    int steps = 0;
    while (true) {
        double dx, dy, dz, d_sq, Fx, Fy, Fz;
        int accepted = -1;
        bool term = false;
        while (k < kend || node >= 0) {
            if (k < kend) {
                const int s = k++;
                if (s == slot) continue;
                const Half q = half_at(t.slot_p, s);
                dx = xi - q.a, dy = yi - q.b, dz = zi - q.c;
                image64x3<PER>(dx, dy, dz, L, halfL);
                d_sq = dx * dx + dy * dy + dz * dz;
                const double r_sum = ri + q.d;
                if (!(d_sq >= r_sum * r_sum)) continue;
                const Half f = half_at(t.slot_f, s);
                Fx = f.a, Fy = f.b, Fz = f.c;
                term = true;
                break;
            }
            if (++steps > t.node_count + 1) {
                raise_device_error(t.err, DEM_DEVERR_NODE_OVERFLOW);
                node = -1;
                break;
            }
            const Half q = half_at(rec, 2 * node), l = half_at(rec, 2 * node + 1);  // size^2, centre | links, force
            const int child = __double2loint(l.a), next = __double2hiint(l.a);
            if (child <= -2) {
                k = -2 - child;
                kend = k + t.count[node];
                node = next;
                continue;
            }
            dx = xi - q.b, dy = yi - q.c, dz = zi - q.d;
            image64x3<PER>(dx, dy, dz, L, halfL);
            d_sq = dx * dx + dy * dy + dz * dz;
            if (q.a < theta_sq * d_sq && d_sq > 0.0) {
                Fx = l.b, Fy = l.c, Fz = l.d;
                accepted = node;
                node = next;
                term = true;
                break;
            }
            node = child;
        }
        if (!term) break;
        const double rr = sqrt(d_sq);
        const double inv_r = 1.0 / rr;
        const double inv_r2 = inv_r * inv_r;
        const double dot = dx * Fx + dy * Fy + dz * Fz;
        const double coeff = eta * inv_r;
        ux += coeff * (Fx + dx * inv_r2 * dot);
        uy += coeff * (Fy + dy * inv_r2 * dot);
        uz += coeff * (Fz + dz * inv_r2 * dot);
        if (CORR) corr_pair64(corr, dx, dy, dz, Fx, Fy, Fz, ux, uy, uz);
        if (accepted >= 0) {  // dipole correction :1215-1265, R^3-weighted centre (same as get_center)
            const Half d0 = half_at(t.rec_d, 3 * accepted), d1 = half_at(t.rec_d, 3 * accepted + 1),
                       d2 = half_at(t.rec_d, 3 * accepted + 2);
            const double D[9] = {d0.a, d0.b, d0.c, d0.d, d1.a, d1.b, d1.c, d1.d, d2.a};
            const double rx = dx, ry = dy, rz = dz;
            const double Ux = D[0] * rx + D[3] * ry + D[6] * rz;
            const double Uy = D[1] * rx + D[4] * ry + D[7] * rz;
            const double Uz = D[2] * rx + D[5] * ry + D[8] * rz;
            const double wx = D[0] * rx + D[1] * ry + D[2] * rz;
            const double wy = D[3] * rx + D[4] * ry + D[5] * rz;
            const double wz = D[6] * rx + D[7] * ry + D[8] * rz;
            const double s_tr = d2.b;
            const double q = rx * wx + ry * wy + rz * wz;
            const double inv_r3 = inv_r * inv_r2;
            const double inv_r5 = inv_r3 * inv_r2;
            ux += eta * (inv_r3 * (Ux - wx - s_tr * rx) + 3.0 * rx * q * inv_r5);
            uy += eta * (inv_r3 * (Uy - wy - s_tr * ry) + 3.0 * ry * q * inv_r5);
            uz += eta * (inv_r3 * (Uz - wz - s_tr * rz) + 3.0 * rz * q * inv_r5);
        }
    }
    if (CORR && !(stokes > 0)) {  // self term, Stokeslet walk only
        ux += corr.g_self * Fx_[i];
        uy += corr.g_self * Fy_[i];
        uz += corr.g_self * Fz_[i];
    }
    vx[i] = ux;
    vy[i] = uy;
    vz[i] = uz;
}

// TreeCollisionFrequency._count_collisions, pbm/collision_frequency/tree_collision_freq.py:62-135:
// every pair j > i with |MIC(x_j - x_i)|^2 <= (r_i + r_j)^2 adds 1 to matrix[b_i][b_j]
// and to matrix[b_j][b_i]; a node is skipped when the squared distance from x_i to
// its box exceeds (r_i + max radius in the node)^2, the box distance taken per
// axis as the gap to the nearer face and, when periodic, replaced by L - gap
// when the gap exceeds L/2 (:137-175), as the reference does.
template <bool PER>
__global__ void collision_walk_kernel(TreeDev t, const int32_t *__restrict__ bins, int nbins,
                                      unsigned int *__restrict__ matrix) {
    const int M = t.max_nodes, N = t.cap, n = t.n;
    const double L = t.L, halfL = 0.5 * t.L;
    // targets in leaf-slot order, as in force_walk_kernel (the counts are integers: any order)
    for (int slot = blockIdx.x * blockDim.x + threadIdx.x; slot < n; slot += gridDim.x * blockDim.x) {
        const int i = t.leaf_idx[slot];
        const double xi = t.p[i], yi = t.p[N + i], zi = t.p[2 * N + i], ri = t.p[3 * N + i];
        const int bi = bins[i];
        int node = 0, steps = 0;
        while (node >= 0) {
            if (++steps > t.node_count + 1) {
                raise_device_error(t.err, DEM_DEVERR_NODE_OVERFLOW);
                break;
            }
            const int cnt = t.count[node];
            if (cnt == 0) {
                node = t.next[node];
                continue;
            }
            if (t.first_child[node] < 0) {
                const int l0 = t.leaf_start[node];
                for (int k = 0; k < cnt; ++k) {
                    const int j = t.leaf_idx[l0 + k];
                    if (j >= 0 && j > i) {
                        double dx = t.p[j] - xi, dy = t.p[N + j] - yi, dz = t.p[2 * N + j] - zi;
                        if (PER) {
                            dx = mic64(dx, L, halfL);
                            dy = mic64(dy, L, halfL);
                            dz = mic64(dz, L, halfL);
                        }
                        const double dist_sq = dx * dx + dy * dy + dz * dz;
                        const double contact = ri + t.p[3 * N + j];
                        if (dist_sq <= contact * contact) {
                            const int bj = bins[j];
                            atomicAdd(&matrix[bi * nbins + bj], 1u);
                            atomicAdd(&matrix[bj * nbins + bi], 1u);
                        }
                    }
                }
                node = t.next[node];
                continue;
            }
            const double max_contact = ri + t.maxr[node];
            double g[3];
            const double p3[3] = {xi, yi, zi};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const double lo = t.mn[a * (size_t)M + node], hi = t.mx[a * (size_t)M + node];
                double d = 0.0;
                if (p3[a] < lo)
                    d = lo - p3[a];
                else if (p3[a] > hi)
                    d = p3[a] - hi;
                if (PER && L > 0.0 && d > halfL) d = L - d;
                g[a] = d;
            }
            const double min_dist_sq = g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
            node = min_dist_sq > max_contact * max_contact ? t.next[node] : t.first_child[node];
        }
    }
}

__global__ void copy_nodes_kernel(TreeDev t, int nc, int32_t *count, int32_t *first_child, int32_t *next,
                                  int32_t *leaf_start, double *r3, double *fs) {
    const int M = t.max_nodes;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nc; k += gridDim.x * blockDim.x) {
        if (count) count[k] = t.count[k];
        if (first_child) first_child[k] = t.first_child[k];
        if (next) next[k] = t.next[k];
        if (leaf_start) leaf_start[k] = t.leaf_start[k];
        if (r3)
            for (int a = 0; a < 4; ++a) r3[4 * (size_t)k + a] = t.R3[a * M + k];
        if (fs)
            for (int a = 0; a < 12; ++a) fs[12 * (size_t)k + a] = t.fs[a * M + k];
    }
}

static int grid_for(dem_ctx *ctx, int64_t work) { return (int)max(1LL, min((long long)ceil_div(work, 256), 16LL * ctx->sm_count)); }

}  // namespace dem

using namespace dem;

static int tree_free(dem_tree *t) {
    void *ptrs[] = {t->mn,       t->mx,   t->R3,       t->maxr,      t->fs,   t->first_child, t->next,
                    t->leaf_start, t->count, t->child_cnt, t->parents, t->parent_fc, t->flag, t->rank,
                    t->fill,     t->p,    t->pf,       t->part_node, t->part_oct, t->leaf_idx,
                    t->rec_f,    t->rec_v, t->rec_d,   t->slot_p,    t->slot_f,   t->roots};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    if (t->h_total) cudaFreeHost(t->h_total);
    return DEM_OK;
}

extern "C" {

int dem_tree_create(dem_ctx *ctx, int capacity, int max_nodes, dem_tree **out) {
    if (!ctx || !out || capacity < 1 || max_nodes < 1) return DEM_E_INVALID;
    *out = nullptr;
    dem_tree *t = new dem_tree();
    t->ctx = ctx;
    t->device = ctx->device;
    t->cap = capacity;
    t->max_nodes = max_nodes;
    const size_t M = (size_t)max_nodes, N = (size_t)capacity;
    cudaSetDevice(ctx->device);
    cudaError_t e = cudaSuccess;
#define ALLOC(f, T, k) \
    if (e == cudaSuccess) e = cudaMalloc((void **)&t->f, sizeof(T) * (k))
    ALLOC(mn, double, 3 * M);
    ALLOC(mx, double, 3 * M);
    ALLOC(R3, double, 4 * M);
    ALLOC(maxr, double, M);
    ALLOC(fs, double, 12 * M);
    ALLOC(first_child, int32_t, M);
    ALLOC(next, int32_t, M);
    ALLOC(leaf_start, int32_t, M);
    ALLOC(count, int32_t, M);
    ALLOC(child_cnt, int32_t, 8 * M);
    ALLOC(parents, int32_t, M);
    ALLOC(parent_fc, int32_t, M);
    ALLOC(flag, int32_t, M + 1);
    ALLOC(rank, int32_t, M + 1);
    ALLOC(fill, int32_t, M);
    ALLOC(p, double, 4 * N);
    ALLOC(pf, double, 3 * N);
    ALLOC(part_node, int32_t, N);
    ALLOC(part_oct, int32_t, N);
    ALLOC(leaf_idx, int32_t, N);
    ALLOC(rec_f, char, WALK_REC_BYTES * M);
    ALLOC(rec_v, char, WALK_REC_BYTES * M);
    ALLOC(rec_d, char, WALK_DIP_BYTES * M);
    ALLOC(slot_p, double2, 2 * N);
    ALLOC(slot_f, double2, 2 * N);
    ALLOC(roots, int32_t, 2);
#undef ALLOC
    if (e == cudaSuccess) e = cudaMallocHost((void **)&t->h_total, sizeof(int32_t) * 2);
    if (e != cudaSuccess) {
        tree_free(t);
        delete t;
        return dem_check_cuda(ctx, e, "tree allocation");
    }
    *out = t;
    return DEM_OK;
}

void dem_tree_destroy(dem_tree *t) {
    if (!t) return;
    cudaSetDevice(t->device);
    tree_free(t);
    delete t;
}

int dem_tree_build(dem_tree *t, int n, const double *x, const double *y, const double *z, const double *r, double L,
                   int periodic, int mpl, void *stream) {
    if (!t) return DEM_E_INVALID;
    dem_ctx *ctx = t->ctx;
    if (n < 0) return dem_set_error(ctx, DEM_E_INVALID, "n must be >= 0");
    if (n > t->cap)
        return dem_set_error(ctx, DEM_E_CAPACITY, "Number of particles (" + std::to_string(n) +
                                                      ") exceeds allocated capacity (" + std::to_string(t->cap) + ")");
    cudaSetDevice(ctx->device);
    cudaStream_t s = (cudaStream_t)stream;
    t->n = n;
    t->L = L;
    t->periodic = periodic ? 1 : 0;
    t->node_count = 1;
    t->parent_count = 0;
    t->pool_exhausted = 0;
    t->built = t->vel_records = false;
    t->level_off.clear();
    dem_prof_begin(ctx, "tree_build", s);
    tree_init_kernel<<<grid_for(ctx, max(n, 1)), 256, 0, counted(s)>>>(view(t), n, L, x, y, z, r);
    int ls = 0, le = 1;
    for (int level = 0; level < 40; ++level) {
        const int pc_before = t->parent_count;
        const int width = le - ls;
        zero_child_cnt_kernel<<<grid_for(ctx, 8LL * width), 256, 0, counted(s)>>>(t->child_cnt, ls, le);
        assign_octants_kernel<<<grid_for(ctx, max(n, 1)), 256, 0, counted(s)>>>(view(t), n, ls, le);
        subdivide_flags_kernel<<<grid_for(ctx, width), 256, 0, counted(s)>>>(view(t), ls, le, mpl);
        int rc = exclusive_scan<int32_t, int32_t>(ctx, t->flag, t->rank, width, s);
        if (rc) return rc;
        rc = dem_check_cuda(ctx, cudaMemcpyAsync(t->h_total, t->rank + width, sizeof(int32_t), cudaMemcpyDeviceToHost, s),
                            "tree build");
        if (!rc) rc = dem_check_cuda(ctx, cudaStreamSynchronize(s), "tree build");
        if (rc) return rc;
        const int total = t->h_total[0];
        const int room = (t->max_nodes - t->node_count) / 8;
        const int sub = total < room ? total : (room > 0 ? room : 0);
        if (sub < total) t->pool_exhausted = 1;
        if (sub > 0) {
            subdivide_kernel<<<grid_for(ctx, 8LL * width), 256, 0, counted(s)>>>(view(t), ls, le, sub, t->node_count, t->parent_count);
            t->node_count += 8 * sub;
            t->parent_count += sub;
        }
        level_scatter_kernel<<<grid_for(ctx, max(n, 1)), 256, 0, counted(s)>>>(view(t), n);
        ls = le;
        le = t->node_count;
        if (t->parent_count > pc_before) t->level_off.push_back(pc_before);
        if (sub == 0) break;
    }
    const int nc = t->node_count;
    leaf_flags_kernel<<<grid_for(ctx, nc), 256, 0, counted(s)>>>(view(t), nc);
    int rc = exclusive_scan<int32_t, int32_t>(ctx, t->flag, t->rank, nc, s);
    if (rc) return rc;
    leaf_start_kernel<<<grid_for(ctx, nc), 256, 0, counted(s)>>>(view(t), nc);
    leaf_scatter_kernel<<<grid_for(ctx, max(n, 1)), 256, 0, counted(s)>>>(view(t), n);
    leaf_sort_kernel<<<grid_for(ctx, nc), 256, 0, counted(s)>>>(view(t), nc);
    const int nl = (int)t->level_off.size();
    auto lev_end = [&](int l) { return l + 1 < nl ? t->level_off[l + 1] : t->parent_count; };
    for (int l = 0; l < nl; ++l)
        next_pass1_kernel<<<grid_for(ctx, lev_end(l) - t->level_off[l]), 256, 0, counted(s)>>>(view(t), t->level_off[l], lev_end(l));
    for (int l = 0; l < nl; ++l)
        next_pass2_kernel<<<grid_for(ctx, lev_end(l) - t->level_off[l]), 256, 0, counted(s)>>>(view(t), t->level_off[l], lev_end(l));
    leaf_r3_kernel<<<grid_for(ctx, nc), 256, 0, counted(s)>>>(view(t), nc);
    for (int l = nl - 1; l >= 0; --l)
        sweep_r3_kernel<<<grid_for(ctx, lev_end(l) - t->level_off[l]), 256, 0, counted(s)>>>(view(t), t->level_off[l], lev_end(l));
    rc = dem_check_cuda(ctx, cudaMemcpyAsync(t->h_total + 1, t->rank + nc, sizeof(int32_t), cudaMemcpyDeviceToHost, s),
                        "tree build");
    if (!rc) rc = dem_check_cuda(ctx, cudaStreamSynchronize(s), "tree build");
    if (rc) return rc;
    t->leaf_slot_count = t->h_total[1];
    walk_records_kernel<true><<<grid_for(ctx, nc), 256, 0, counted(s)>>>(view(t), nc, t->roots);
    slot_droplets_kernel<<<grid_for(ctx, max(n, 1)), 256, 0, counted(s)>>>(view(t), n);
    dem_prof_end(ctx, s);
    rc = dem_check_launch(ctx, "tree build");
    t->built = rc == DEM_OK;
    return rc;
}

int dem_tree_forces(dem_tree *t, double m_const, double theta_sq, double *fx, double *fy, double *fz, void *stream) {
    if (!t || !fx || !fy || !fz) return DEM_E_INVALID;
    if (t->n == 0) return DEM_OK;
    if (!t->built) return dem_set_error(t->ctx, DEM_E_INVALID, "the tree's build did not complete");
    cudaStream_t s = (cudaStream_t)stream;
    dem_prof_begin(t->ctx, "tree_force_walk", s);
    const int grid = ceil_div(t->n, WALK_T);
    if (t->periodic)
        force_walk_kernel<true><<<grid, WALK_T, 0, counted(s)>>>(view(t), m_const, theta_sq, fx, fy, fz);
    else
        force_walk_kernel<false><<<grid, WALK_T, 0, counted(s)>>>(view(t), m_const, theta_sq, fx, fy, fz);
    dem_prof_end(t->ctx, s);
    return dem_check_launch(t->ctx, "tree force walk");
}

// The velocity walk's records from the node force sums.
static void velocity_records(dem_tree *t, cudaStream_t s) {
    walk_records_kernel<false><<<grid_for(t->ctx, t->node_count), 256, 0, counted(s)>>>(view(t), t->node_count, t->roots + 1);
    t->vel_records = true;
}

int dem_tree_propagate_forces(dem_tree *t, const double *fx, const double *fy, const double *fz, void *stream) {
    if (!t) return DEM_E_INVALID;
    dem_ctx *ctx = t->ctx;
    cudaStream_t s = (cudaStream_t)stream;
    const int N = t->cap, nc = t->node_count;
    if (!fx) {
        fx = t->pf;
        fy = t->pf + N;
        fz = t->pf + 2 * (size_t)N;
    }
    leaf_forces_kernel<<<grid_for(ctx, nc), 256, 0, counted(s)>>>(view(t), nc, fx, fy, fz);
    const int nl = (int)t->level_off.size();
    for (int l = nl - 1; l >= 0; --l) {
        const int a = t->level_off[l], b = l + 1 < nl ? t->level_off[l + 1] : t->parent_count;
        sweep_forces_kernel<<<dim3(grid_for(ctx, b - a), 12), 256, 0, counted(s)>>>(view(t), a, b);
    }
    if (t->built) velocity_records(t, s);  // the links of a tree without a build lead anywhere
    return dem_check_launch(ctx, "tree propagate forces");
}

int dem_tree_velocity(dem_tree *t, const double *fx, const double *fy, const double *fz, double eta_const,
                      double theta_sq, double stokes_factor, double *vx, double *vy, double *vz, void *stream) {
    if (!t || !vx || !vy || !vz) return DEM_E_INVALID;
    if (t->n == 0) return DEM_OK;
    if (!t->built) return dem_set_error(t->ctx, DEM_E_INVALID, "the tree's build did not complete");
    const int N = t->cap;
    if (!fx) {
        fx = t->pf;
        fy = t->pf + N;
        fz = t->pf + 2 * (size_t)N;
    }
    cudaStream_t s = (cudaStream_t)stream;
    if (!t->vel_records) velocity_records(t, s);  // no forces propagated on this tree: its links, the sums as they are
    dem_prof_begin(t->ctx, "tree_velocity_walk", s);
    const int grid = ceil_div(t->n, WALK_T);
    const TreeDev tv = view(t);
    slot_forces_kernel<<<grid_for(t->ctx, t->n), 256, 0, counted(s)>>>(tv, t->n, fx, fy, fz);
    if (t->corr) {
        const CorrDev cv = corr_view(t->corr);
        if (t->periodic)
            velocity_walk_kernel<true, true><<<grid, WALK_T, 0, counted(s)>>>(tv, fx, fy, fz, eta_const, theta_sq,
                                                                           stokes_factor, cv, vx, vy, vz);
        else
            velocity_walk_kernel<false, true><<<grid, WALK_T, 0, counted(s)>>>(tv, fx, fy, fz, eta_const, theta_sq,
                                                                            stokes_factor, cv, vx, vy, vz);
    } else {
        const CorrDev none{};
        if (t->periodic)
            velocity_walk_kernel<true, false><<<grid, WALK_T, 0, counted(s)>>>(tv, fx, fy, fz, eta_const, theta_sq,
                                                                            stokes_factor, none, vx, vy, vz);
        else
            velocity_walk_kernel<false, false><<<grid, WALK_T, 0, counted(s)>>>(tv, fx, fy, fz, eta_const, theta_sq,
                                                                             stokes_factor, none, vx, vy, vz);
    }
    dem_prof_end(t->ctx, s);
    return dem_check_launch(t->ctx, "tree velocity walk");
}

int dem_tree_set_correction(dem_tree *t, const dem_corr *corr) {
    if (!t) return DEM_E_INVALID;
    if (corr && corr->ctx && corr->ctx->device != t->device)
        return dem_set_error(t->ctx, DEM_E_INVALID, "correction grid lives on another device");
    t->corr = corr;
    return DEM_OK;
}

int dem_tree_stats(const dem_tree *t, int64_t *out) {
    if (!t || !out) return DEM_E_INVALID;
    out[0] = t->node_count;
    out[1] = t->parent_count;
    out[2] = t->leaf_slot_count;
    out[3] = t->max_nodes;
    out[4] = (int64_t)t->level_off.size();
    out[5] = t->n;
    out[6] = t->pool_exhausted;
    out[7] = t->cap;
    return DEM_OK;
}

int dem_tree_nodes(dem_tree *t, int32_t *count, int32_t *first_child, int32_t *next, int32_t *leaf_start, double *r3,
                   double *fs, void *stream) {
    if (!t) return DEM_E_INVALID;
    const int nc = t->node_count;
    copy_nodes_kernel<<<grid_for(t->ctx, nc), 256, 0, counted((cudaStream_t)stream)>>>(view(t), nc, count, first_child, next,
                                                                             leaf_start, r3, fs);
    return dem_check_launch(t->ctx, "tree nodes");
}

int dem_tree_collision_matrix(dem_tree *t, const int32_t *bins, int nbins, uint32_t *matrix, void *stream) {
    if (!t || nbins < 1 || !matrix || (t->n > 0 && !bins)) return DEM_E_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    int rc = dem_check_cuda(t->ctx, cudaMemsetAsync(matrix, 0, sizeof(uint32_t) * nbins * nbins, s), "memset");
    if (rc || t->n == 0) return rc;
    const int grid = ceil_div(t->n, 128);
    dem_prof_begin(t->ctx, "tree_collision_walk", s);
    if (t->periodic)
        collision_walk_kernel<true><<<grid, 128, 0, counted(s)>>>(view(t), bins, nbins, matrix);
    else
        collision_walk_kernel<false><<<grid, 128, 0, counted(s)>>>(view(t), bins, nbins, matrix);
    dem_prof_end(t->ctx, s);
    return dem_check_launch(t->ctx, "tree collision walk");
}

int dem_tree_leaf_indices(dem_tree *t, int32_t *out, void *stream) {
    if (!t || !out) return DEM_E_INVALID;
    if (t->n == 0) return DEM_OK;
    return dem_check_cuda(t->ctx,
                          cudaMemcpyAsync(out, t->leaf_idx, sizeof(int32_t) * t->n, cudaMemcpyDeviceToDevice,
                                          (cudaStream_t)stream),
                          "leaf indices");
}

}  // extern "C"
