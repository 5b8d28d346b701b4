// build.cu — device construction of the leaf order, neighbour, stencil,
// hanging-node and ghost tables of a leaf set.
//
// Replaces, for the GPU path, what the reference rebuilds after every
// change of the tree: idneighbor (src/neighbor.F90:399-449), the leaf lists
// of IDgrid (src/solution.F90:593-693), and the per-call stencil search of
// parent_value_weno / child_value_weno / search_cell_5 / WLSI_US_WENO's
// geometry (src/XuanGua.F90:45-356), which the reference redoes inside
// every stage for every hanging face.
#include <cub/cub.cuh>

#include "handle.cuh"
#include "scan.cuh"
#include "topo.cuh"

namespace fdm {

#define FDM_ATAN_BIAS 1.000000013351432e-10   /* REAL(4) 1e-10, src/XuanGua.F90:40 */
#define FDM_PI_REF 3.1415926535897932

enum BuildErr { BE_PARTITION = 0, BE_NULLNB = 1, BE_OVERFLOW = 2, BE_ROOT = 3, BE_LEVEL = 4, BE_INDEX = 5 };

static inline int nblk(int64_t n, int t) { return (int)((n + t - 1) / t); }

// get_direction (src/XuanGua.F90:33-43): 45-degree sector 1..8 (1 = east,
// counter-clockwise) of (xx,yy) seen from (x,y).
__device__ __noinline__ int get_direction_atan(double dx, double dy) {
    const double angle = (atan2(dy, dx) + FDM_ATAN_BIAS) * 180.0 / FDM_PI_REF;
    const int f = (int)floor((angle + 22.5) / 45.0 + 8);
    return ((f % 8) + 8) % 8 + 1;
}
// The sector follows from |dy| against tan(22.5) |dx| and tan(67.5) |dx|
// except next to a sector boundary: a relative margin of 1e-9 on the
// tangent keeps the point more than 3.5e-10 rad from the boundary, which
// is more than the 1e-10 rad shift of the bias plus the rounding of atan2
// and of the angle arithmetic, so the sector is the one the formula above
// gives; the points within the margin (and dx = dy = 0) take the formula.
__device__ __forceinline__ int get_direction(double xx, double yy, double x, double y) {
    const double dx = xx - x;
    const double dy = yy - y;
    const double a = fabs(dx), b = fabs(dy);
    constexpr double T1 = 0.41421356237309503, T2 = 2.414213562373095;   // tan(22.5), tan(67.5)
    constexpr double LO = 1.0 - 1e-9, HI = 1.0 + 1e-9;
    if (b < a * (T1 * LO)) return dx > 0.0 ? 1 : 5;
    if (b > a * (T2 * HI)) return dy > 0.0 ? 3 : 7;
    if (b > a * (T1 * HI) && b < a * (T2 * LO)) return dx > 0.0 ? (dy > 0.0 ? 2 : 8) : (dy > 0.0 ? 4 : 6);
    return get_direction_atan(dx, dy);
}

// ------------------------------------------------------------ classify
constexpr unsigned long long LEAF_INTERIOR = 1ull, LEAF_GHOST = 1ull << 32;
__global__ void k_classify(const uint64_t *__restrict__ lkey, int64_t NL, Geometry G,
                           unsigned long long *kind, int8_t *cross, int32_t *err) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= NL) return;
    const int64_t total = (int64_t)G.m * G.n;
    const uint64_t key = lkey[k];
    const int lvl = (int)(key & 15u);
    const int64_t root = (int64_t)(key >> 34);
    const uint64_t pos = key_pos(key);
    if (root >= total) { atomicExch(err + BE_ROOT, 1); return; }
    if (lvl >= MAXLVL_TAB - 1) atomicExch(err + BE_LEVEL, 1);
    if (pos & (span_of_level(lvl) - 1)) atomicExch(err + BE_PARTITION, 1);
    const uint64_t prev_end = k == 0 ? 0ull : key_pos(lkey[k - 1]) + span_of_level((int)(lkey[k - 1] & 15u));
    if (pos != prev_end) atomicExch(err + BE_PARTITION, 1);
    if (k == NL - 1 && pos + span_of_level(lvl) != ((uint64_t)total << 30)) atomicExch(err + BE_PARTITION, 1);
    const int c = root_cross(G, root);
    cross[k] = (int8_t)c;
    // halo leaves of a strip take ghost slots (not advanced, not filled)
    const bool halo = root_in_halo(G, root);
    // interior leaf in the low word, ghost in the high one: one scan counts both
    kind[k] = c == 0 && !halo ? LEAF_INTERIOR : c == -5 && !halo ? 0ull : LEAF_GHOST;
}

// slots (interior leaves, ghosts, corners, each in key order; before: the
// interior leaves and ghosts before each leaf) and centres
__global__ void k_slots(int64_t NL, int64_t NI, int64_t NG, const uint64_t *__restrict__ lkey, Geometry G,
                        const unsigned long long *__restrict__ kind, const unsigned long long *__restrict__ before,
                        int32_t *lslot, int32_t *slot_leaf, double *cx, double *cy) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= NL) return;
    const unsigned long long c = kind[k], p = before[k];
    const int64_t bi = (int64_t)(p & 0xffffffffull), bg = (int64_t)(p >> 32);
    const int32_t s = (int32_t)(c == LEAF_INTERIOR ? bi : c == LEAF_GHOST ? NI + bg : NI + NG + (k - bi - bg));
    lslot[k] = s;
    slot_leaf[s] = (int32_t)k;
    double x, y;
    node_center(G, node_of_key(lkey[k]), x, y);
    cx[k] = x;
    cy[k] = y;
}

__global__ void k_scatter(int64_t NL, const int32_t *perm, const int32_t *lslot,
                          const double *__restrict__ prim, double4 *B0) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= NL) return;
    const int64_t src = perm ? perm[k] : k;
    B0[lslot[k]] = make_double4(prim[4 * src], prim[4 * src + 1], prim[4 * src + 2], prim[4 * src + 3]);
}

// ------------------------------------------------------- stencil resolve
// Tip/Tim/Tjp/Tjm and Tipp/Timm/Tjpp/Tjmm (src/XuanGua.F90:401-590):
// each of the 8 stencil entries of an interior leaf is either a same-level
// leaf (its slot) or a request: parent_value_weno on a same-level internal
// node, or child_value_weno on a coarser leaf at a target point.
struct ResolveOut {
    int32_t *slot;    // >= 0 direct slot, -1 request
    int32_t *flag;    // 1: a request
    int32_t *kind;    // 0 parent, 1 child
    int64_t *ref;     // parent: node key; child: sorted leaf index
    double *tx, *ty;  // target point
};

__device__ __forceinline__ void target_point(const Geometry &G, double cx, double cy, int lvl, int dir,
                                             int k2, double &xx, double &yy) {
    if (k2 == 1) {
        switch (dir) {
            case DIR_RIGHT: xx = cx + G.xf * G.h / ipow2d(lvl); yy = cy; break;
            case DIR_LEFT: xx = cx - G.xf * G.h / ipow2d(lvl); yy = cy; break;
            case DIR_UP: xx = cx; yy = cy + G.h / ipow2d(lvl); break;
            default: xx = cx; yy = cy - G.h / ipow2d(lvl); break;
        }
    } else {
        switch (dir) {
            case DIR_RIGHT: xx = cx + 2.0 * G.xf * G.h / ipow2d(lvl); yy = cy; break;
            case DIR_LEFT: xx = cx - 2.0 * G.xf * G.h / ipow2d(lvl); yy = cy; break;
            case DIR_UP: xx = cx; yy = cy + 2.0 * G.h / ipow2d(lvl); break;
            default: xx = cx; yy = cy - 2.0 * G.h / ipow2d(lvl); break;
        }
    }
}

// l_max: the deepest interior level
__global__ void k_resolve(Tables T, Geometry G, ResolveOut O, uint8_t *ilvl, int32_t *err, int32_t *l_max) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= T.NI) return;
    const int32_t k = T.slot_leaf[i];
    NodeRef c;
    c.n = node_of_key(T.lkey[k]);
    c.leaf = k;
    c.valid = 1;
    ilvl[i] = (uint8_t)c.n.lvl;
    if (*l_max < c.n.lvl) atomicMax(l_max, c.n.lvl);
    const double cx = T.lcx[k], cy = T.lcy[k];
    const int dirs[4] = {DIR_RIGHT, DIR_LEFT, DIR_UP, DIR_DOWN};
    for (int q = 0; q < 4; ++q) {
        const int d = dirs[q];
        const NodeRef cn = face_nb(T, G, c, d);
        if (!cn.valid) { atomicExch(err + BE_NULLNB, 1); return; }
        // T1
        int64_t e = i * 8 + q;
        if (cn.n.lvl == c.n.lvl) {
            if (cn.leaf >= 0) O.slot[e] = T.lslot[cn.leaf];
            else { O.slot[e] = -1; O.kind[e] = 0; O.ref[e] = (int64_t)node_key(cn.n); }
        } else {
            O.slot[e] = -1; O.kind[e] = 1; O.ref[e] = cn.leaf;
            target_point(G, cx, cy, c.n.lvl, d, 1, O.tx[e], O.ty[e]);
        }
        // T2
        e = i * 8 + 4 + q;
        if (cn.n.lvl == c.n.lvl) {
            const NodeRef cnn = face_nb(T, G, cn, d);
            if (!cnn.valid) { atomicExch(err + BE_NULLNB, 1); return; }
            if (cnn.n.lvl == cn.n.lvl) {
                if (cnn.leaf >= 0) O.slot[e] = T.lslot[cnn.leaf];
                else { O.slot[e] = -1; O.kind[e] = 0; O.ref[e] = (int64_t)node_key(cnn.n); }
            } else {
                O.slot[e] = -1; O.kind[e] = 1; O.ref[e] = cnn.leaf;
                target_point(G, cx, cy, c.n.lvl, d, 2, O.tx[e], O.ty[e]);
            }
        } else {
            O.slot[e] = -1; O.kind[e] = 1; O.ref[e] = cn.leaf;
            target_point(G, cx, cy, c.n.lvl, d, 2, O.tx[e], O.ty[e]);
        }
        O.flag[i * 8 + q] = O.slot[i * 8 + q] < 0;
        O.flag[e] = O.slot[e] < 0;
    }
}

struct ReqDesc {
    int32_t *kind;
    int64_t *ref;
    double *tx, *ty;
};

__global__ void k_emit(int64_t n, int64_t VS0, ResolveOut O, const int32_t *ridx, int32_t *ist, ReqDesc R) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= n) return;
    const int32_t s = O.slot[e];
    if (s >= 0) { ist[e] = s; return; }
    const int32_t r = ridx[e];
    ist[e] = (int32_t)(VS0 + r);
    R.kind[r] = O.kind[e];
    R.ref[r] = O.ref[e];
    R.tx[r] = O.tx[e];
    R.ty[r] = O.ty[e];
}

// ---------------------------------------------------------- WLS gather
// search_cell_5 (src/XuanGua.F90:152-177) on a node: its leaves in traversal
// order son1, son2, son3, son4; the first leaf of every still-unused sector
// joins the stencil.  Which leaf that is does not depend on the sectors
// already used, so the areas of a request are searched independently (one
// lane each): the first leaf of every sector of the area, as traversal rank
// (the Morton path with digits 2 and 3 exchanged) above leaf index, into
// first[8] (shared memory).
__device__ __forceinline__ void area_search(const Tables &T, const NodeRef &X, double x, double y,
                                            unsigned long long *first) {
    for (int s = 0; s < 8; ++s) first[s] = ~0ull;
    if (!X.valid) return;
    int64_t lo = X.leaf, hi = X.leaf + 1;
    if (X.leaf < 0) {
        const uint64_t p0 = node_pos(X.n);
        lo = lower_bound_pos_t(T, p0);
        hi = lower_bound_pos_t(T, p0 + span_of_level(X.n.lvl));
    }
    for (int64_t k = lo; k < hi; ++k) {
        const int s = get_direction(T.lcx[k], T.lcy[k], x, y) - 1;
        const uint64_t path = key_pos(T.lkey[k]) & ((1ull << 30) - 1ull);
        const unsigned long long v = (path ^ ((path & 0x2AAAAAAAull) >> 1)) << 32 | (unsigned long long)k;
        if (v < first[s]) first[s] = v;
    }
}

// brinv (src/XuanGua.F90:593-660): full-pivot Gauss-Jordan in place;
// returns false on the singular test (the partially reduced matrix stays).
// The matrix lives in registers: every loop is unrolled, and the row and
// column exchanges with the pivot (whose indices are data) are selects over
// the rows and columns at or after the step, so the arithmetic is the
// reference's, operation for operation.
template <int N>
__device__ __forceinline__ void brinv_swap_rows(double (&r)[N][N], int k, int p) {
#pragma unroll
    for (int q = 0; q < N; ++q)
        if (q > k) {   // q == p > k: exchange rows k and q
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const double a = r[k][j], b = r[q][j];
                const bool sw = q == p;
                r[k][j] = sw ? b : a;
                r[q][j] = sw ? a : b;
            }
        }
}
template <int N>
__device__ __forceinline__ void brinv_swap_cols(double (&r)[N][N], int k, int p) {
#pragma unroll
    for (int q = 0; q < N; ++q)
        if (q > k) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const double a = r[i][k], b = r[i][q];
                const bool sw = q == p;
                r[i][k] = sw ? b : a;
                r[i][q] = sw ? a : b;
            }
        }
}
template <int N>
__device__ __forceinline__ bool brinv_reg(double (&r)[N][N]) {
    int is[N], js[N];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        is[k] = 0; js[k] = 0;
        if (ok) {
            double d = 0.0;
            int pi = 0, pj = 0;
#pragma unroll
            for (int i = 0; i < N; ++i)
#pragma unroll
                for (int j = 0; j < N; ++j)
                    if (i >= k && j >= k && fabs(r[i][j]) > d) { d = fabs(r[i][j]); pi = i; pj = j; }
            is[k] = pi; js[k] = pj;
            if (d + 1.0 == 1.0) {
                ok = false;
            } else {
                brinv_swap_rows<N>(r, k, pi);
                brinv_swap_cols<N>(r, k, pj);
                r[k][k] = 1.0 / r[k][k];
#pragma unroll
                for (int j = 0; j < N; ++j) if (j != k) r[k][j] = r[k][j] * r[k][k];
#pragma unroll
                for (int i = 0; i < N; ++i)
                    if (i != k)
#pragma unroll
                        for (int j = 0; j < N; ++j)
                            if (j != k) r[i][j] = r[i][j] - r[i][k] * r[k][j];
#pragma unroll
                for (int i = 0; i < N; ++i) if (i != k) r[i][k] = -r[i][k] * r[k][k];
            }
        }
    }
    if (!ok) return false;
    // undo the exchanges: row k with row js[k], column k with column is[k]
#pragma unroll
    for (int k = N - 1; k >= 0; --k) {
        brinv_swap_rows<N>(r, k, js[k]);
        brinv_swap_cols<N>(r, k, is[k]);
    }
    return true;
}

struct ReqOut {
    int32_t *kind;
    int32_t *m;
    int32_t *mem;
    double *geo;
    uint64_t *node;
    unsigned long long *counts;   // [0] singular, [2] restrict
};

// Stencil gather of parent_value_weno / child_value_weno
// (src/XuanGua.F90:45-150), or the reference's fallback when fewer than 7
// points were found.  Eight lanes per request: each finds and searches one of
// the areas that the reference visits in turn, then the areas' finds are
// joined in that order.  (With one thread per request, which also formed the
// geometry below, a warp ran the longest of 32 serial searches: 613 us for 81k
// requests, 172 us for 18k; the two kernels take 223 and 59.)
constexpr int GATHER_RPB = 16;   // requests per block
__global__ void __launch_bounds__(GATHER_RPB * 8) k_gather(Tables T, Geometry G, ReqDesc D, ReqOut O, int32_t *err) {
    __shared__ unsigned long long first[GATHER_RPB][8][8];
    __shared__ int32_t list[GATHER_RPB][2][WLS_AXIS];   // axis members, diagonal members
    const int lane = threadIdx.x & 7, g = threadIdx.x >> 3, g0 = threadIdx.x & 24;
    const unsigned mask = 0xFFu << g0;
    const int64_t r = (int64_t)blockIdx.x * GATHER_RPB + g;
    if (r >= T.NR) return;   // whole groups of eight lanes
    const bool child = D.kind[r] != 0;
    NodeRef c;
    c.valid = 1;
    double x, y;
    if (!child) {   // parent_value_weno on the internal node: sons 1..4, then left, right, down, up
        c.n = node_of_key((uint64_t)D.ref[r]);
        c.leaf = -1;
        node_center(G, c.n, x, y);
    } else {        // child_value_weno on the coarse leaf
        c.leaf = (int32_t)D.ref[r];
        c.n = node_of_key(T.lkey[c.leaf]);
        x = T.lcx[c.leaf]; y = T.lcy[c.leaf];
    }
    NodeRef X;
    if (!child && lane < 4) {
        X = child_ref(T, c, lane ^ (lane >> 1));   // sons 1, 2, 3, 4 are digits 0, 1, 3, 2
    } else {
        // child: down-left, left, up-left, down, up, down-right, right, up-right
        const int dx = child ? (lane < 3 ? DIR_LEFT : DIR_RIGHT) : lane == 4 ? DIR_LEFT : DIR_RIGHT;
        const int dy = child ? (lane == 0 || lane == 3 || lane == 5 ? DIR_DOWN : DIR_UP) : lane == 6 ? DIR_DOWN : DIR_UP;
        const bool diag = child && (lane == 0 || lane == 2 || lane == 5 || lane == 7);
        if (diag) X = root_cross(G, c.n.root) >= 0 ? diagonal_nb(T, G, c, dx, dy) : null_ref();
        else X = face_nb(T, G, c, child ? (lane == 1 || lane == 6 ? dx : dy) : (lane < 6 ? dx : dy));
    }
    area_search(T, X, x, y, first[g][lane]);
    __syncwarp(mask);
    int m1 = 0, m2 = 0;
    unsigned used = 0;
    bool overflow = false;
    if (child) {
        if (lane == 0) list[g][0][0] = c.leaf;
        m1 = 1;
    }
    for (int a = 0; a < 8; ++a) {
        if (!child && a == 4 && m1 + m2 >= 8) break;
        const unsigned long long mine = first[g][a][lane];   // sector lane + 1
        for (;;) {
            unsigned long long v = (used >> lane) & 1u ? ~0ull : mine;
            unsigned long long best = v;
            for (int o = 1; o < 8; o <<= 1) best = min(best, __shfl_xor_sync(mask, best, o));
            if (best == ~0ull) break;
            const int s = __ffs((__ballot_sync(mask, v == best) >> g0) & 0xFFu) - 1;
            used |= 1u << s;
            const int32_t leaf = (int32_t)(best & 0xffffffffull);
            // an even sector (1, 3, 5, 7 of the reference) is an axis one; a
            // leaf already in the list is not taken twice
            const int which = s & 1, n = which ? m2 : m1;
            __syncwarp(mask);
            const bool dup = lane < n && list[g][which][lane] == leaf;
            if (__any_sync(mask, dup)) continue;
            if (n >= (which ? WLS_MAXM - WLS_AXIS : WLS_AXIS)) { overflow = true; continue; }
            if (lane == 0) list[g][which][n] = leaf;
            if (which) ++m2;
            else ++m1;
            __syncwarp(mask);
        }
    }
    __syncwarp(mask);
    double *geo = O.geo + rq_geo_at(r);
    int32_t *mem = O.mem + rq_mem_at(r);
    const int m = m1 + m2;
    const bool few = m < 7;
    if (lane == 0) {
        if (overflow) atomicExch(err + BE_OVERFLOW, 1);
        const uint64_t p0 = node_pos(c.n);
        O.node[r] = node_key(c.n);
        geo[G_ORIGIN * RQ_T] = child ? 1.0 : 0.0;
        geo[G_XX * RQ_T] = child ? D.tx[r] : x;
        geo[G_YY * RQ_T] = child ? D.ty[r] : y;
        O.kind[r] = !few ? RQ_WLS : child ? RQ_COPY : RQ_RESTRICT;
        O.m[2 * r] = !few ? m1 : child ? 1 : (int32_t)lower_bound_pos_t(T, p0);
        O.m[2 * r + 1] = !few ? m2 : child ? 0 : (int32_t)lower_bound_pos_t(T, p0 + span_of_level(c.n.lvl));
        if (few && child) mem[0] = T.lslot[c.leaf];
        if (few && !child) {
            geo[G_LVL * RQ_T] = (double)c.n.lvl;
            atomicAdd(O.counts + 2, 1ull);
        }
    }
    if (few) return;
    for (int i = lane; i < WLS_MAXM; i += 8) {
        const bool axis = i < WLS_AXIS, in = axis ? i < m1 : i - WLS_AXIS < m2;
        const int32_t leaf = !in ? -1 : axis ? list[g][0][i] : list[g][1][i - WLS_AXIS];
        mem[i * RQ_T] = in ? T.lslot[leaf] : -1;
        geo[(G_X + i) * RQ_T] = in ? T.lcx[leaf] : 0.0;
        geo[(G_Y + i) * RQ_T] = in ? T.lcy[leaf] : 0.0;
    }
    if (lane == 7) {
        // smoothness box of the node (compute_smoothness, src/XuanGua.F90:318-323)
        const double hx = G.xf * G.h / ipow2d(c.n.lvl + 1);
        const double hy = G.h / ipow2d(c.n.lvl + 1);
        geo[(G_BOX + 0) * RQ_T] = x - hx;
        geo[(G_BOX + 1) * RQ_T] = x + hx;
        geo[(G_BOX + 2) * RQ_T] = y - hy;
        geo[(G_BOX + 3) * RQ_T] = y + hy;
    }
}

// WLSI_US_WENO geometry of a request: the weights, P^T W P over all members
// and over the axis and the diagonal ones, and their three brinv inverses
// (src/XuanGua.F90:206-255); one thread per request, no divergence but the
// member count.
__global__ void __launch_bounds__(64) k_wls_geometry(Tables T, ReqOut O) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= T.NR || O.kind[r] != RQ_WLS) return;
    double *geo = O.geo + rq_geo_at(r);
    const int m1 = O.m[2 * r], m2 = O.m[2 * r + 1];
    const double xx = geo[G_XX * RQ_T], yy = geo[G_YY * RQ_T];
    double R[6][6], RA[3][3], RB[3][3];
#pragma unroll
    for (int a = 0; a < 6; ++a)
#pragma unroll
        for (int b = 0; b < 6; ++b) R[a][b] = 0.0;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) { RA[a][b] = 0.0; RB[a][b] = 0.0; }
#pragma unroll
    for (int i = 0; i < WLS_MAXM; ++i) {
        if (i < WLS_AXIS ? i >= m1 : i - WLS_AXIS >= m2) {
            geo[(G_W + i) * RQ_T] = 0.0;
            continue;
        }
        const double xi = geo[(G_X + i) * RQ_T], yi = geo[(G_Y + i) * RQ_T];
        const double d = sqrt((xi - xx) * (xi - xx) + (yi - yy) * (yi - yy));
        const double w = 1.0 / (d + 1.e-6);
        geo[(G_W + i) * RQ_T] = w;
        const double P[6] = {1.0, xi, yi, xi * yi, xi * xi, yi * yi};
        double pw[6];
#pragma unroll
        for (int b = 0; b < 6; ++b) pw[b] = w * P[b];
#pragma unroll
        for (int a = 0; a < 6; ++a)
#pragma unroll
            for (int b = 0; b < 6; ++b) R[a][b] = R[a][b] + P[a] * pw[b];
        if (i < WLS_AXIS) {
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) RA[a][b] = RA[a][b] + P[a] * pw[b];
        } else {
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) RB[a][b] = RB[a][b] + P[a] * pw[b];
        }
    }
    unsigned long long ns = 0;
    if (!brinv_reg<3>(RA)) ++ns;
#pragma unroll
    for (int k = 0; k < 9; ++k) geo[(G_A + k) * RQ_T] = RA[k / 3][k % 3];
    if (!brinv_reg<3>(RB)) ++ns;
#pragma unroll
    for (int k = 0; k < 9; ++k) geo[(G_B + k) * RQ_T] = RB[k / 3][k % 3];
    if (!brinv_reg<6>(R)) ++ns;
#pragma unroll
    for (int k = 0; k < 36; ++k) geo[(G_L + k) * RQ_T] = R[k / 6][k % 6];
    if (ns) atomicAdd(O.counts + 0, ns);
}

// ------------------------------------------------------------- ghosts
struct GhostOut {
    int32_t *kind, *a, *b, *flip;
    double *x, *y;
    int32_t *rlist;                   // ghosts imaged by a subtree restriction (in no particular order)
    unsigned long long *n_restrict;
};

__device__ __forceinline__ void ghost_from_ref(const Tables &T, const NodeRef &img, GhostOut &O, int64_t g) {
    if (img.leaf >= 0) {
        O.kind[g] = GH_COPY;
        O.a[g] = T.lslot[img.leaf];
        O.b[g] = 0;
    } else {
        const uint64_t p0 = node_pos(img.n);
        O.kind[g] = GH_RESTRICT;
        O.rlist[atomicAdd(O.n_restrict, 1ull)] = (int32_t)g;
        O.a[g] = (int32_t)lower_bound_pos_t(T, p0);
        O.b[g] = (int32_t)lower_bound_pos_t(T, p0 + span_of_level(img.n.lvl));
    }
}

// image node for the extension kinds: root (row1, col1) 1-based, descent along
// the ghost's path from the root with the quadrant bits transformed
// (mode 0 keep, 1 force x, 2 force y, 3 mirror y, 4 mirror x)
__device__ NodeRef ext_image(const Tables &T, const Geometry &G, const Node &gn, int row1, int col1,
                             int mode, int bit) {
    Node r0;
    r0.root = (int64_t)(row1 - 1) * G.m + (col1 - 1);
    r0.lvl = 0; r0.ix = 0; r0.iy = 0;
    NodeRef cur = resolve(T, r0);
    for (int j = 1; j <= gn.lvl; ++j) {
        if (cur.leaf >= 0) break;
        int q = (int)(((gn.ix >> (gn.lvl - j)) & 1u) | (((gn.iy >> (gn.lvl - j)) & 1u) << 1));
        if (mode == 1) q = (q & 2) | bit;
        else if (mode == 2) q = (q & 1) | (bit << 1);
        else if (mode == 3) q ^= 2;
        else if (mode == 4) q ^= 1;
        cur = child_ref(T, cur, q);
    }
    return cur;
}

__global__ void k_ghosts(Tables T, Geometry G, fdm_params P, GhostOut O) {
    const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (g >= T.NG) return;
    const int32_t k = T.slot_leaf[T.NI + g];
    const Node gn = node_of_key(T.lkey[k]);
    if (root_in_halo(G, gn.root)) {   // written by the strip's caller
        O.kind[g] = GH_NONE; O.a[g] = 0; O.b[g] = 0; O.flip[g] = 0;
        O.x[g] = T.lcx[k]; O.y[g] = T.lcy[k];
        return;
    }
    const int a = root_cross(G, gn.root);
    const int row = (int)(gn.root / G.m) + 1, col = (int)(gn.root % G.m) + 1;
    const int m = G.m, n = G.n;
    int kind;
    if (a == -4) kind = P.kind_xmbc;
    else if (a == -2) kind = P.kind_xpbc;
    else if (a == -3) kind = P.kind_ypbc;
    else kind = P.kind_ymbc;
    O.flip[g] = 0;
    O.x[g] = T.lcx[k];
    O.y[g] = T.lcy[k];
    if (kind == FDM_BC_PERIODIC) {
        // BC_cyc (src/solution.F90:116-166): image root by index arithmetic,
        // descent along the ghost's sp list taken deepest level first
        const int num1 = row, num2 = col;
        int i1;
        if (a == -4) i1 = num1 * m + num2 - 6;
        else if (a == -2) i1 = num1 * m + num2 - 2 * m + 6;
        else if (a == -3) i1 = num1 * m + num2 - (n - 5) * m;
        else i1 = num1 * m + num2 - (7 - n) * m;
        Node r0;
        r0.root = i1 - 1; r0.lvl = 0; r0.ix = 0; r0.iy = 0;
        NodeRef cur = resolve(T, r0);
        for (int j = 0; j < gn.lvl; ++j) {
            if (cur.leaf >= 0) break;
            // sp(j+1) = sp of the ancestor j levels above the ghost
            const int l = gn.lvl - j;
            const int q = (int)(((gn.ix >> (gn.lvl - l)) & 1u) | (((gn.iy >> (gn.lvl - l)) & 1u) << 1));
            cur = child_ref(T, cur, q);
        }
        ghost_from_ref(T, cur, O, g);
        return;
    }
    if (kind == FDM_BC_TRANSMISSIVE) {
        NodeRef img;
        if (a == -4) img = ext_image(T, G, gn, row, 4, 1, 0);
        else if (a == -2) img = ext_image(T, G, gn, row, m - 3, 1, 1);
        else if (a == -1) img = ext_image(T, G, gn, 4, col, 2, 0);
        else img = ext_image(T, G, gn, n - 3, col, 2, 1);
        ghost_from_ref(T, img, O, g);
        return;
    }
    if (kind == FDM_BC_WALL || kind == FDM_BC_DMR_BOTTOM) {
        if (kind == FDM_BC_DMR_BOTTOM && T.lcx[k] <= P.dmr_x0) {
            O.kind[g] = GH_STATE; O.a[g] = 4; O.b[g] = 0;
            return;
        }
        NodeRef img;
        if (a == -1) img = ext_image(T, G, gn, 7 - row, col, 3, 0);
        else if (a == -3) img = ext_image(T, G, gn, 2 * n - 5 - row, col, 3, 0);
        else if (a == -4) img = ext_image(T, G, gn, row, 7 - col, 4, 0);
        else img = ext_image(T, G, gn, row, 2 * m - 5 - col, 4, 0);
        ghost_from_ref(T, img, O, g);
        O.flip[g] = (a == -1 || a == -3) ? 2 : 1;
        return;
    }
    if (kind == FDM_BC_INFLOW) {
        O.kind[g] = GH_STATE;
        O.a[g] = a == -4 ? 0 : a == -2 ? 1 : a == -1 ? 2 : 3;
        O.b[g] = 0;
        return;
    }
    if (kind == FDM_BC_DMR_TOP) {
        O.kind[g] = GH_DMR_TOP; O.a[g] = 0; O.b[g] = 0;
        return;
    }
    O.kind[g] = GH_NONE; O.a[g] = 0; O.b[g] = 0;
}

// --------------------------------------------------------------- faces
// The right (top) face of every interior leaf is face i.  Its left (bottom)
// face is the right face of the left neighbour j when j is an interior
// same-level leaf whose 4-point face stencil is slot-for-slot the same;
// otherwise the leaf owns a separate left face.
__global__ void k_face_flags(Tables T, unsigned long long *u) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= T.NI) return;
    const int32_t *s = T.ist + i * 8;
    int shared = 0;
    const int32_t j = s[1];
    if (j >= 0 && j < T.NI) {
        const int32_t *t = T.ist + (int64_t)j * 8;
        shared = (t[1] == s[5]) && (t[0] == (int32_t)i) && (t[4] == s[0]);
    }
    int shy = 0;
    const int32_t jy = s[3];
    if (jy >= 0 && jy < T.NI) {
        const int32_t *t = T.ist + (int64_t)jy * 8;
        shy = (t[3] == s[7]) && (t[2] == (int32_t)i) && (t[6] == s[2]);
    }
    // separate x face in the low word, y face in the high one: one scan for both
    u[i] = (shared ? 0ull : 1ull) | (shy ? 0ull : 1ull << 32);
}
__global__ void k_face_assign(Tables T, const unsigned long long *__restrict__ u,
                              const unsigned long long *__restrict__ before, int32_t *ifxl, int32_t *ifyl,
                              int32_t *uxl, int32_t *uyl) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= T.NI) return;
    const int32_t *s = T.ist + i * 8;
    const unsigned long long v = u[i], p = before[i];
    const int32_t px = (int32_t)(p & 0xffffffffull), py = (int32_t)(p >> 32);
    if (v & 1ull) { ifxl[i] = (int32_t)(T.NI + px); uxl[px] = (int32_t)i; }
    else ifxl[i] = s[1];
    if (v >> 32) { ifyl[i] = (int32_t)(T.NI + py); uyl[py] = (int32_t)i; }
    else ifyl[i] = s[3];
}

// Every index a stage kernel will dereference is checked once here, so that
// no stage kernel can read or write outside its buffers.
// face_counts: the unshared left faces (nux, nuy) as the device counted them
// (words of a packed total); l_max goes to the time loop's scalars.
__global__ void k_validate(Tables T, const int32_t *__restrict__ face_counts, int32_t *err, const int32_t *l_max,
                           DevScalars *sc) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t == 0) sc->l_max = *l_max;
    T.nux = face_counts[0];
    T.nuy = face_counts[1];
    const int64_t NLEAF = T.NI + T.NG + T.NC;
    bool bad = false;
    if (t < T.NI * 8) {
        const int32_t s = T.ist[t];
        bad |= s < 0 || s >= T.NS;
    }
    if (t < T.NI) {
        bad |= T.ifxl[t] < 0 || T.ifxl[t] >= T.NI + T.nux;
        bad |= T.ifyl[t] < 0 || T.ifyl[t] >= T.NI + T.nuy;
    }
    if (t < T.nux) bad |= T.uxl[t] < 0 || T.uxl[t] >= T.NI;
    if (t < T.nuy) bad |= T.uyl[t] < 0 || T.uyl[t] >= T.NI;
    if (t < T.NR) {
        const int k = T.rq_kind[t];
        const int32_t a = T.rq_m[2 * t], b = T.rq_m[2 * t + 1];
        const int32_t *mem = T.rq_mem + rq_mem_at(t);
        if (k == RQ_WLS) {
            bad |= a < 0 || a > WLS_AXIS || b < 0 || b > WLS_MAXM - WLS_AXIS;
            if (!bad)
                for (int i = 0; i < WLS_MAXM; ++i) {
                    const bool in = i < WLS_AXIS ? i < a : i - WLS_AXIS < b;
                    bad |= in ? mem[i * RQ_T] < 0 || mem[i * RQ_T] >= NLEAF : mem[i * RQ_T] != -1;
                }
        } else if (k == RQ_RESTRICT) {
            bad |= a < 0 || b <= a || b > T.NL;
        } else if (k == RQ_COPY) {
            bad |= mem[0] < 0 || mem[0] >= NLEAF;
        } else {
            bad = true;
        }
    }
    if (t < T.NG) {
        const int k = T.gh_kind[t];
        const int32_t a = T.gh_a[t], b = T.gh_b[t];
        if (k == GH_COPY) bad |= a < 0 || a >= NLEAF;
        else if (k == GH_RESTRICT) bad |= a < 0 || b <= a || b > T.NL;
        else if (k == GH_STATE) bad |= a < 0 || a >= 6;
        else if (k != GH_DMR_TOP && k != GH_NONE) bad = true;
    }
    if (bad) atomicExch(err + BE_INDEX, 1);
}

// ------------------------------------------------------------ host side
static __global__ void k_iota_b(int64_t n, int32_t *a) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) a[i] = (int32_t)i;
}
// rf[r] = first sorted leaf of background cell r, rf[nroots] = n; cells
// without leaves (rejected later by the partition check) get the next
// cell's start; roots beyond the grid (rejected as well) are clamped
__global__ void k_root_first(int64_t n, const uint64_t *__restrict__ lkey, int64_t nroots, int32_t *rf) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i > n) return;
    auto root = [&](int64_t k) -> int64_t {
        const int64_t r = (int64_t)(lkey[k] >> 34);
        return r < nroots ? r : nroots;
    };
    const int64_t prev = i == 0 ? -1 : root(i - 1);
    const int64_t cur = i == n ? nroots : root(i);
    for (int64_t x = prev + 1; x <= cur; ++x) rf[x] = (int32_t)i;
}
// What the build counts on the device, in one block that is zeroed at the
// start and read back whole (through pinned memory) at each wait.
struct BuildWords {
    int32_t err[8];                // BuildErr flags
    int32_t l_max, nr;             // deepest interior level, requests
    unsigned long long leaves;     // interior leaves | ghosts << 32
    int32_t faces[2];              // separate left faces, bottom faces
    unsigned long long counts[8];  // [0] singular, [2] restrict requests, [4] restrict ghosts, [6] listed requests
};
static_assert(sizeof(BuildWords) <= fdm_handle::PIN_WORDS * 4, "the build's words must fit the pinned ones");
// exclusive scan; its total goes to the word `total` of dw, and (read) all
// words to the host, to be looked at after the next wait
template <class U>
static int scan_total(fdm_handle *h, const U *in, U *out, int64_t n, BuildWords *dw, U *total, bool read) {
    ScanArgs<U> a{in, out, n, total, nullptr, -1, nullptr, nullptr, nullptr, 0};
    if (read) {
        a.total2 = reinterpret_cast<U *>(reinterpret_cast<char *>(h->pin) +
                                         (reinterpret_cast<char *>(total) - reinterpret_cast<char *>(dw)));
        a.words = reinterpret_cast<const int32_t *>(dw);
        a.words_out = h->pin;
        a.nwords = sizeof(BuildWords) / 4;
    }
    FDM_CK(h, launch_scan(h, a));
    return FDM_OK;
}
static int read_back(fdm_handle *h, const BuildWords *&w) {
    FDM_CK(h, cudaMemcpyAsync(h->pin, h->tmp[7].p, sizeof(BuildWords), cudaMemcpyDeviceToHost, h->s));
    FDM_CK(h, cudaStreamSynchronize(h->s));
    w = reinterpret_cast<const BuildWords *>(h->pin);
    return FDM_OK;
}

#define FDM_RC(x)                 \
    do {                          \
        int rc_ = (x);            \
        if (rc_) return rc_;      \
    } while (0)

__global__ void k_restrict_list(int64_t NR, const int32_t *__restrict__ kind, int32_t *list,
                                unsigned long long *count) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r < NR && kind[r] == RQ_RESTRICT) list[atomicAdd(count, 1ull)] = (int32_t)r;
}

__global__ void k_descents(int64_t n, const uint64_t *__restrict__ key, int32_t *flag) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i + 1 < n && key[i] > key[i + 1]) *flag = 1;
}
int keys_sorted(fdm_handle *h, int64_t n, const uint64_t *keys_dev, bool *sorted) {
    int32_t *flag = h->flag.as<int32_t>(), f = 0;
    FDM_CK(h, cudaMemsetAsync(flag, 0, 4, h->s));
    k_descents<<<nblk(n, 256), 256, 0, h->s>>>(n, keys_dev, flag);
    FDM_CK(h, cudaMemcpyAsync(&f, flag, 4, cudaMemcpyDeviceToHost, h->s));
    FDM_CK(h, cudaStreamSynchronize(h->s));
    *sorted = f == 0;
    return FDM_OK;
}

int build_tables(fdm_handle *h, int64_t n, const uint64_t *keys_in, const double *prim_in, int key_bits) {
    Nvtx range("fdm tables");
    const int TB = 256;
    cudaStream_t s = h->s;
    if (n <= 0 || n >= (1ll << 31) - 1) return arg_fail(h, "leaf count out of range");
    h->NL = n;
    FDM_CK(h, h->tmp[7].ensure(sizeof(BuildWords)));
    FDM_CK(h, cudaMemsetAsync(h->tmp[7].p, 0, sizeof(BuildWords), s));
    FDM_CK(h, cudaMemsetAsync(h->flag.p, 0, 8 * sizeof(int32_t), s));   // a halo copy's slot error ends with its tables
    BuildWords *dw = h->tmp[7].as<BuildWords>();   // device
    const BuildWords *w = nullptr;                 // read back
    int32_t *err = dw->err;
    // 1. sort keys, carrying the input index
    FDM_CK(h, h->lkey.ensure(n * 8));
    const int32_t *perm = nullptr;
    if (key_bits <= 0) {
        if (keys_in != h->lkey.as<uint64_t>())
            FDM_CK(h, cudaMemcpyAsync(h->lkey.as<uint64_t>(), keys_in, n * 8, cudaMemcpyDeviceToDevice, s));
    } else {
        FDM_CK(h, h->tmp[0].ensure(n * 4));   // iota
        FDM_CK(h, h->tmp[1].ensure(n * 4));   // perm
        int32_t *iota = h->tmp[0].as<int32_t>();
        k_iota_b<<<nblk(n, TB), TB, 0, s>>>(n, iota);
        size_t bytes = 0;
        FDM_CK(h, cub::DeviceRadixSort::SortPairs(nullptr, bytes, keys_in, h->lkey.as<uint64_t>(), iota,
                                                  h->tmp[1].as<int32_t>(), (int)n, 0, key_bits, s));
        FDM_CK(h, h->cub_tmp.ensure(bytes));
        FDM_CK(h, cub::DeviceRadixSort::SortPairs(h->cub_tmp.p, bytes, keys_in, h->lkey.as<uint64_t>(), iota,
                                                  h->tmp[1].as<int32_t>(), (int)n, 0, key_bits, s));
        perm = h->tmp[1].as<int32_t>();
    }
    const uint64_t *lkey = h->lkey.as<uint64_t>();
    {
        const int64_t nroots = (int64_t)h->G.m * h->G.n;
        FDM_CK(h, h->rfirst.ensure((nroots + 1) * 4));
        k_root_first<<<nblk(n + 1, TB), TB, 0, s>>>(n, lkey, nroots, h->rfirst.as<int32_t>());
    }
    // 2. classify + partition check
    Carve c2;
    c2.add(n * 8); c2.add(n * 8);
    FDM_CK(h, h->tmp[2].ensure(c2.total));
    unsigned long long *lkind = c2.at<unsigned long long>(h->tmp[2], 0), *before = c2.at<unsigned long long>(h->tmp[2], 1);
    FDM_CK(h, h->lcross.ensure(n));
    k_classify<<<nblk(n, TB), TB, 0, s>>>(lkey, n, h->G, lkind, h->lcross.as<int8_t>(), err);
    FDM_RC(scan_total<unsigned long long>(h, lkind, before, n, dw, &dw->leaves, true));
    FDM_CK(h, cudaStreamSynchronize(s));
    w = reinterpret_cast<const BuildWords *>(h->pin);
    if (w->err[BE_ROOT]) return arg_fail(h, "leaf key names a background cell outside the m x n grid");
    if (w->err[BE_PARTITION]) return arg_fail(h, "leaf set does not partition the background grid (gap, overlap or duplicate)");
    if (w->err[BE_LEVEL]) return arg_fail(h, "leaf level above the supported maximum (14)");
    const int64_t NI = (int64_t)(w->leaves & 0xffffffffull), NG = (int64_t)(w->leaves >> 32), NC = n - NI - NG;
    if (NI == 0) return arg_fail(h, "no interior leaves");
    h->NI = NI; h->NG = NG; h->NC = NC;
    // 3. slots, values, centres
    FDM_CK(h, h->lslot.ensure(n * 4));
    FDM_CK(h, h->slot_leaf.ensure(n * 4));
    FDM_CK(h, h->lcx.ensure(n * 8));
    FDM_CK(h, h->lcy.ensure(n * 8));
    k_slots<<<nblk(n, TB), TB, 0, s>>>(n, NI, NG, lkey, h->G, lkind, before, h->lslot.as<int32_t>(),
                                       h->slot_leaf.as<int32_t>(), h->lcx.as<double>(), h->lcy.as<double>());
    // 4. stencil resolution
    const int64_t ne = NI * 8;
    FDM_CK(h, h->ist.ensure(ne * 4));
    FDM_CK(h, h->ilvl.ensure(NI));
    Carve c3;
    c3.add(ne * 4); c3.add(ne * 4); c3.add(ne * 8); c3.add(ne * 8); c3.add(ne * 8); c3.add(ne * 4); c3.add(ne * 4);
    FDM_CK(h, h->tmp[3].ensure(c3.total));
    ResolveOut RO;
    RO.slot = c3.at<int32_t>(h->tmp[3], 0);
    RO.kind = c3.at<int32_t>(h->tmp[3], 1);
    RO.ref = c3.at<int64_t>(h->tmp[3], 2);
    RO.tx = c3.at<double>(h->tmp[3], 3);
    RO.ty = c3.at<double>(h->tmp[3], 4);
    RO.flag = c3.at<int32_t>(h->tmp[3], 5);
    int32_t *ridx = c3.at<int32_t>(h->tmp[3], 6);
    {
        Tables T = h->tables();
        k_resolve<<<nblk(NI, 128), 128, 0, s>>>(T, h->G, RO, h->ilvl.as<uint8_t>(), err, &dw->l_max);
    }
    FDM_RC(scan_total<int32_t>(h, RO.flag, ridx, ne, dw, &dw->nr, true));
    FDM_CK(h, cudaStreamSynchronize(s));
    if (w->err[BE_NULLNB]) return arg_fail(h, "an interior leaf has a null stencil neighbour (fewer than 3 ghost layers?)");
    const int64_t NR = w->nr;
    h->NR = NR;
    h->NS = NI + NG + NC + NR;
    const int64_t VS0 = NI + NG + NC;
    const int64_t nrq = (NR > 0 ? NR + RQ_T - 1 : RQ_T) / RQ_T * RQ_T;   // whole tiles
    Carve c4;
    c4.add(nrq * 4); c4.add(nrq * 8); c4.add(nrq * 8); c4.add(nrq * 8);
    FDM_CK(h, h->tmp[4].ensure(c4.total));
    ReqDesc RD;
    RD.kind = c4.at<int32_t>(h->tmp[4], 0);
    RD.ref = c4.at<int64_t>(h->tmp[4], 1);
    RD.tx = c4.at<double>(h->tmp[4], 2);
    RD.ty = c4.at<double>(h->tmp[4], 3);
    k_emit<<<nblk(ne, TB), TB, 0, s>>>(ne, VS0, RO, ridx, h->ist.as<int32_t>(), RD);
    // 5. requests: gather + WLS geometry
    FDM_CK(h, h->rq_kind.ensure(nrq * 4));
    FDM_CK(h, h->rq_m.ensure(nrq * 8));
    FDM_CK(h, h->rq_mem.ensure(nrq * WLS_MAXM * 4));
    FDM_CK(h, h->rq_geo.ensure(nrq * RQ_GEO * 8));
    FDM_CK(h, h->rq_node.ensure(nrq * 8));
    unsigned long long *counts = dw->counts;
    if (NR > 0) {
        Tables T = h->tables();
        ReqOut O{h->rq_kind.as<int32_t>(), h->rq_m.as<int32_t>(), h->rq_mem.as<int32_t>(),
                 h->rq_geo.as<double>(), h->rq_node.as<uint64_t>(), counts};
        k_gather<<<nblk(NR, GATHER_RPB), GATHER_RPB * 8, 0, s>>>(T, h->G, RD, O, err);
        k_wls_geometry<<<nblk(NR, 64), 64, 0, s>>>(T, O);
    }
    // the interpA fallbacks among the requests, listed (in no particular
    // order: each writes only its own value), so that their warps are
    // launched for them alone
    FDM_CK(h, h->rq_rlist.ensure((NR > 0 ? NR : 1) * 4));
    if (NR > 0)
        k_restrict_list<<<nblk(NR, TB), TB, 0, s>>>(NR, h->rq_kind.as<int32_t>(), h->rq_rlist.as<int32_t>(),
                                                    counts + 6);
    // 6. ghosts
    const int64_t ngh = NG > 0 ? NG : 1;
    FDM_CK(h, h->gh_kind.ensure(ngh * 4));
    FDM_CK(h, h->gh_a.ensure(ngh * 4));
    FDM_CK(h, h->gh_b.ensure(ngh * 4));
    FDM_CK(h, h->gh_flip.ensure(ngh * 4));
    FDM_CK(h, h->gh_rlist.ensure(ngh * 4));
    FDM_CK(h, h->gh_x.ensure(ngh * 8));
    FDM_CK(h, h->gh_y.ensure(ngh * 8));
    if (NG > 0) {
        Tables T = h->tables();
        GhostOut O{h->gh_kind.as<int32_t>(), h->gh_a.as<int32_t>(), h->gh_b.as<int32_t>(),
                   h->gh_flip.as<int32_t>(), h->gh_x.as<double>(),  h->gh_y.as<double>(),
                   h->gh_rlist.as<int32_t>(), counts + 4};
        k_ghosts<<<nblk(NG, 128), 128, 0, s>>>(T, h->G, h->p, O);
    }
    // 7. faces
    Carve c6;
    c6.add(NI * 8); c6.add(NI * 8);
    FDM_CK(h, h->tmp[6].ensure(c6.total));
    unsigned long long *u = c6.at<unsigned long long>(h->tmp[6], 0), *ub = c6.at<unsigned long long>(h->tmp[6], 1);
    {
        Tables T = h->tables();
        k_face_flags<<<nblk(NI, TB), TB, 0, s>>>(T, u);
    }
    // the face counts come back with the final checks; until then the
    // buffers take their bound (at most one unshared left face per leaf)
    FDM_RC(scan_total<unsigned long long>(h, u, ub, NI, dw, reinterpret_cast<unsigned long long *>(dw->faces), false));
    const int64_t nux_max = NI, nuy_max = NI;
    FDM_CK(h, h->ifxl.ensure(NI * 4));
    FDM_CK(h, h->ifyl.ensure(NI * 4));
    FDM_CK(h, h->uxl.ensure(nux_max * 4));
    FDM_CK(h, h->uyl.ensure(nuy_max * 4));
    {
        Tables T = h->tables();
        k_face_assign<<<nblk(NI, TB), TB, 0, s>>>(T, u, ub, h->ifxl.as<int32_t>(), h->ifyl.as<int32_t>(),
                                                  h->uxl.as<int32_t>(), h->uyl.as<int32_t>());
    }
    // 8. state buffers (corner values copied into all three)
    const int64_t NS = h->NS;
    for (int b = 0; b < 3; ++b) FDM_CK(h, h->B[b].ensure(NS * 32));
    FDM_CK(h, h->Fx.ensure((NI + nux_max) * 32));
    FDM_CK(h, h->Fy.ensure((NI + nuy_max) * 32));
    FDM_CK(h, h->Ut.ensure(NI * 32));
    k_scatter<<<nblk(n, TB), TB, 0, s>>>(n, perm, h->lslot.as<int32_t>(), prim_in, h->B[0].as<double4>());
    if (NC > 0)
        for (int b = 1; b < 3; ++b)
            FDM_CK(h, cudaMemcpyAsync(h->B[b].as<double4>() + NI + NG, h->B[0].as<double4>() + NI + NG, NC * 32,
                                      cudaMemcpyDeviceToDevice, s));
    // 9. index validation of every table the stage kernels use
    {
        Tables T = h->tables();
        int64_t nv = NI * 8;
        const int64_t others[5] = {nux_max, nuy_max, NR, NG, NI};
        for (int q = 0; q < 5; ++q) nv = nv > others[q] ? nv : others[q];
        k_validate<<<nblk(nv, TB), TB, 0, s>>>(T, dw->faces, err, &dw->l_max, h->scal.as<DevScalars>());
    }
    FDM_RC(read_back(h, w));
    FDM_CK(h, cudaGetLastError());
    h->nux = w->faces[0];
    h->nuy = w->faces[1];
    if (w->counts[2] != w->counts[6]) return arg_fail(h, "internal table check failed: restrict list");
    if (w->err[BE_OVERFLOW]) return arg_fail(h, "hanging-node stencil larger than supported");
    if (w->err[BE_INDEX]) return arg_fail(h, "internal table check failed: an index is out of range");
    h->l_max = w->l_max;
    h->n_singular += (int64_t)w->counts[0];
    h->n_restrict = (int64_t)w->counts[2];
    h->n_ghost_restrict = (int64_t)w->counts[4];
    h->table_version++;
    h->gate_stage1_valid = false;
    h->lam_fresh = false;
    h->cur_buf = 0;
    h->loaded = true;
    return FDM_OK;
}

}  // namespace fdm
