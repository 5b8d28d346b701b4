// amr.cu — device regrid (src/solution.F90:408-589, src/mesh.F90:199-408).
#include <algorithm>

#include <cub/cub.cuh>

#include "handle.cuh"
#include "ordered_sum.cuh"
#include "scan.cuh"
#include "topo.cuh"

namespace fdm {

static inline int nblk(int64_t n, int t) { return (int)((n + t - 1) / t); }

void launch_requests(fdm_handle *h, const double4 *cur);

// Place of an interior leaf in the traversal of solute_div_rot (roots
// row-major, sons 1,2,3,4) given its place k in key order, where son 4
// (digit 2) comes before son 3 (digit 3): at every level it moves by the
// leaves of the other of these two sons.  Two searches in the leaf's
// background cell per digit 2 or 3, in place of a radix sort of the leaves
// (with the sums below, the indicators of 3.2k leaves take 0.043 ms instead
// of 0.247, of 100k leaves 0.158 instead of 0.311).
__device__ __forceinline__ int64_t traversal_shift(const Tables &T, uint64_t key) {
    const int lvl = (int)(key & 15u);
    const uint64_t pos = key_pos(key);
    int64_t shift = 0;
    for (int j = 1; j <= lvl; ++j) {
        const int b = 2 * (LMAX - j);
        const uint64_t q = (pos >> b) & 3u;
        if (q < 2) continue;
        const uint64_t at2 = ((pos >> (b + 2)) << (b + 2)) | (2ull << b), at3 = at2 + (1ull << b);
        const int64_t i3 = lower_bound_pos_t(T, at3);
        if (q == 2) shift += lower_bound_pos_t(T, at3 + (1ull << b)) - i3;
        else shift -= i3 - lower_bound_pos_t(T, at2);
    }
    return shift;
}

// Urot / Udiv / dux (src/solution.F90:558-589) on the stencil values
// Tip, Tim, Tjp, Tjm of every interior leaf; their squares in traversal order
// (rounded as in the sequential loop: no FMA in this build).
__global__ void k_rot_div(Tables T, LevelTab LT, const double4 *__restrict__ B, double *rot, double *div,
                          double2 *__restrict__ sq) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= T.NI) return;
    const int lvl = T.ilvl[i];
    const int32_t *s = T.ist + i * 8;
    const double4 ip = B[s[0]], im = B[s[1]], jp = B[s[2]], jm = B[s[3]];
    const double dy = LT.dy[lvl], dx = LT.dx[lvl], p15 = LT.p15[lvl];
    const double vx = (ip.z - im.z) / (2.0 * dx);
    const double uy = (jp.y - jm.y) / (2.0 * dy);
    const double r = fabs(vx - uy) * p15;
    const double ux = (ip.x - im.x) / (2.0 * dx);
    const double vy = (jp.x - jm.x) / (2.0 * dy);
    const double d = (fabs(ux) + fabs(vy)) * p15;
    rot[i] = r;
    div[i] = d;
    sq[i + traversal_shift(T, T.lkey[T.slot_leaf[i]])] = make_double2(r * r, d * d);
}

// Srot, Sdiv: left-to-right sums in traversal order, as the reference's
// recursive loop forms them (src/solution.F90:430-457), bit for bit, one
// block each (ordered_sum.cuh); launched with 2 blocks
__global__ void __launch_bounds__(OSUM_NT) k_ordered_sums(int64_t NI, const double2 *__restrict__ sq, double *out) {
    __shared__ OSumShared sh;
    const double *x = reinterpret_cast<const double *>(sq) + blockIdx.x;
    const double v = ordered_sum_block<OSUM_NT, OSUM_EPT>([&](int64_t e) { return x[2 * e]; }, NI, sh);
    if (threadIdx.x == 0) {
        out[blockIdx.x] = v;
        if (blockIdx.x == 0) out[2] = (double)NI;
    }
}

// rot/div of the current state into rot/div buffers; ordered sums to out3
static int compute_rot_div(fdm_handle *h, double *rot, double *div, double *out3) {
    Nvtx range("fdm regrid: indicators");
    const int64_t NI = h->NI;
    launch_requests(h, h->B[0].as<double4>());
    FDM_CK(h, h->tmp[0].ensure(NI * 16));
    double2 *sq = h->tmp[0].as<double2>();
    k_rot_div<<<nblk(NI, 256), 256, 0, h->s>>>(h->tables(), h->lt, h->B[0].as<double4>(), rot, div, sq);
    k_ordered_sums<<<2, OSUM_NT, 0, h->s>>>(NI, sq, out3);
    return FDM_OK;
}

// ===================================================================
// Regrid.  The tree is handled as a node set: every leaf and every internal
// node, sorted by key, each with a value.  Internal nodes carry the value
// the reference leaves in a refined cell (its U when it was refined, or the
// interpA mean when it was coarsened), because gridmodify4 can copy it back
// into new leaves (Refine_cell of a non-leaf, src/mesh.F90:389-392).
// ===================================================================

struct NodeSet {
    int64_t n = 0;
    uint64_t *key = nullptr;
    uint8_t *leaf = nullptr;
    double4 *val = nullptr;
    int32_t *rf = nullptr;         // per-cell index of key
    int64_t nroots = 0;
};

enum { D_NONE = 0, D_REFINE = 1, D_COARSEN = 2 };

__device__ __forceinline__ int64_t find_key(const uint64_t *__restrict__ keys, int64_t n, uint64_t k) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        const uint64_t v = keys[mid];
        if (v < k) lo = mid + 1;
        else hi = mid;
    }
    return (lo < n && keys[lo] == k) ? lo : -1;
}

// find_key within the nodes of k's background cell (every cell holds at
// least its root node, and its nodes are contiguous)
__device__ __forceinline__ int64_t find_key_set(const NodeSet &A, uint64_t k) {
    const int64_t r = (int64_t)(k >> 34);
    if (r >= A.nroots) return -1;
    int64_t lo = __ldg(A.rf + r), hi = __ldg(A.rf + r + 1);
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        const uint64_t v = A.key[mid];
        if (v < k) lo = mid + 1;
        else hi = mid;
    }
    return (lo < A.n && A.key[lo] == k) ? lo : -1;
}

// find_key on the leaf table, within k's background cell (T.rfirst)
__device__ __forceinline__ int64_t find_key_t(const Tables &T, uint64_t k) {
    const int64_t r = (int64_t)(k >> 34);
    if (!T.rfirst || r >= T.nroots) return find_key(T.lkey, T.NL, k);
    int64_t lo = __ldg(T.rfirst + r), hi = __ldg(T.rfirst + r + 1);
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (__ldg(T.lkey + mid) < k) lo = mid + 1;
        else hi = mid;
    }
    return (lo < T.NL && __ldg(T.lkey + lo) == k) ? lo : -1;
}

// The helpers below work on the interleaved path bits directly.  Level j's
// digit (x bit | y bit << 1) sits at key bit 4 + 2 (LMAX - j); the x bits of
// the path occupy the even path positions and the y bits the odd ones.
constexpr uint64_t KEY_PATH_X = 0x15555555ull << 4;   // x bits of the path
constexpr uint64_t KEY_PATH_Y = 0x2AAAAAAAull << 4;   // y bits of the path
constexpr uint64_t KEY_PATH = (KEY_PATH_X | KEY_PATH_Y);
FDM_HD int key_digit_shift(int lvl) { return 4 + 2 * (LMAX - lvl); }

FDM_HD uint64_t parent_key(uint64_t k) {
    const int lvl = (int)(k & 15u);
    return (k & ~(3ull << key_digit_shift(lvl))) - 1u;
}
FDM_HD uint64_t child_key(uint64_t k, int q) {
    const int lvl = (int)(k & 15u);
    return (k | ((uint64_t)q << key_digit_shift(lvl + 1))) + 1u;
}
// The ancestor of key k at level la (0 <= la <= k's level): the path digits
// below level la cleared
FDM_HD uint64_t ancestor_key(uint64_t k, int la) {
    const uint64_t below = ((1ull << (2 * (LMAX - la))) - 1ull) << 4;
    return (k & ~below & ~15ull) | (uint64_t)la;
}
// Row and column of a background cell: q = root / m from a float reciprocal
// (root < 2^24, so the estimate is off by at most one) and one correction
FDM_HD void root_row_col(uint32_t root, uint32_t m, uint32_t &row, uint32_t &col) {
    uint32_t q = (uint32_t)((float)root * (1.0f / (float)m));
    int64_t r = (int64_t)root - (int64_t)q * m;
    q = r < 0 ? q - 1u : (r >= (int64_t)m ? q + 1u : q);
    r = r < 0 ? r + m : (r >= (int64_t)m ? r - m : r);
    row = q;
    col = (uint32_t)r;
}
// same-level neighbour node key across a face; false across the grid edge.
// A step along x (y) is a dilated increment or decrement of the x (y) bits
// at the node's level; a carry out of the path (or a borrow) moves to the
// next root.  Written without branches: the lanes of a warp step in
// different directions.
FDM_HD bool shift_key(const Geometry &G, uint64_t k, int dir, uint64_t &out) {
    const int lvl = (int)(k & 15u);
    const uint64_t unit = 1ull << key_digit_shift(lvl);
    const bool alongx = dir == DIR_RIGHT || dir == DIR_LEFT;
    const bool inc = dir == DIR_RIGHT || dir == DIR_UP;
    const uint64_t mask = alongx ? KEY_PATH_X : KEY_PATH_Y;
    const uint64_t u = alongx ? unit : unit << 1;
    const uint64_t bits = k & mask;
    // carries skip the other coordinate's bits; a borrow from zero leaves all
    // ones down to the node's level, the first node of the next root back
    const uint64_t path = inc ? (((bits | ~mask) + u) & mask) : ((bits - u) & mask);
    const bool wrap = inc ? (((bits | ~mask | (u - 1)) & KEY_PATH) == KEY_PATH) : bits == 0;
    const uint32_t root = (uint32_t)(k >> 34);
    const uint32_t m = (uint32_t)G.m;
    uint32_t row, col;
    root_row_col(root, m, row, col);
    const uint32_t rc = alongx ? col : row, lim = alongx ? m : (uint32_t)G.n;
    const bool edge = inc ? rc + 1u >= lim : rc == 0u;
    const uint32_t step = alongx ? 1u : m;
    const uint32_t nroot = wrap ? (inc ? root + step : root - step) : root;
    out = ((uint64_t)nroot << 34) | (k & ~mask & ((1ull << 34) - 1ull)) | path;
    return !(wrap && edge);
}
// traversal rank of gridmodify4 / solute_div_rot (sons 1,2,3,4): Morton path
// with the digits of son3 and son4 swapped
FDM_HD uint64_t dfs_rank(uint64_t k) {
    const uint64_t path = key_pos(k) & ((1ull << 30) - 1ull);
    return ((k >> 34) << 30) | (path ^ ((path & 0x2AAAAAAAull) >> 1));
}
// Visit order of gridmodify4's traversal (sons 1,2,3,4 of every node): the
// traversal rank of the node's position, then its level, so a node comes
// before its first son, which starts at the same position.  The node's key
// is recovered from it.  Below 2^53 for up to 2^19 background cells.
FDM_HD uint64_t visit_rank(uint64_t k) { return (dfs_rank(k) << 4) | (k & 15u); }
FDM_HD uint64_t key_of_visit_rank(uint64_t r) {
    const uint64_t pr = r >> 4;
    const uint64_t path = pr & ((1ull << 30) - 1ull);
    return ((pr >> 30) << 34) | ((path ^ ((path & 0x2AAAAAAAull) >> 1)) << 4) | (r & 15u);
}
// post-order rank of gridmodify1 (a node after all of its descendants):
// 3 bits per level, sons 1,2,3,4 -> 0,1,2,3 and 4 below the node's level
FDM_HD uint64_t post_rank(uint64_t k) {
    const Node n = node_of_key(k);
    const uint64_t path = key_pos(k) & ((1ull << 30) - 1ull);
    uint64_t r = 0;
    for (int l = 1; l <= LMAX; ++l) {
        uint64_t dgt = 4;
        if (l <= n.lvl) {
            const uint64_t q = (path >> (2 * (LMAX - l))) & 3u;
            dgt = q ^ (q >> 1);
        }
        r = (r << 3) | dgt;
    }
    return ((uint64_t)n.root << 45) | r;
}

__device__ __forceinline__ double4 mean4(const double4 &c0, const double4 &c1, const double4 &c2, const double4 &c3) {
    // interpA: 0.25*(son1 + son2 + son3 + son4) with son3 = q3, son4 = q2
    double4 v;
    v.x = 0.25 * (c0.x + c1.x + c3.x + c2.x);
    v.y = 0.25 * (c0.y + c1.y + c3.y + c2.y);
    v.z = 0.25 * (c0.z + c1.z + c3.z + c2.z);
    v.w = 0.25 * (c0.w + c1.w + c3.w + c2.w);
    return v;
}

// ---------------------------------------------------- internal node values
// The internal nodes from the sorted leaves: each starts where its first
// leaf starts, so that leaf names it: leaf k names as many of its ancestors
// as its path ends in zero digits, in key order from the outermost one in.
// Nodes named by successive leaves ascend, so the list is made in key order.
__device__ __forceinline__ int named_ancestors(uint64_t k) {
    const int lvl = (int)(k & 15u);
    if (lvl == 0) return 0;
    const uint64_t path = (k & KEY_PATH) >> key_digit_shift(lvl);   // digit j at bit 2 (lvl - j)
    return path == 0 ? lvl : min(lvl, (__ffsll((long long)path) - 1) >> 1);
}
__global__ void k_anc_count(int64_t NL, const uint64_t *lkey, int32_t *cnt, int32_t *max_lvl) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int lvl = 0;
    if (k < NL) {
        const uint64_t key = lkey[k];
        cnt[k] = named_ancestors(key);
        lvl = (int)(key & 15u);
    }
    lvl = __reduce_max_sync(0xffffffffu, lvl);
    if ((threadIdx.x & 31) == 0 && lvl > 0) atomicMax(max_lvl, lvl);
}
__global__ void k_anc_emit(int64_t NL, const uint64_t *lkey, const int32_t *off, uint64_t *out) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= NL) return;
    const uint64_t key = lkey[k];
    const int l = (int)(key & 15u), c = named_ancestors(key);
    for (int j = 0; j < c; ++j) out[off[k] + j] = ancestor_key(key, l - c + j);
}
// interpA of internal nodes at one level from their children (leaves or
// deeper internal nodes, already done)
__global__ void k_internal_vals(int64_t NInt, const uint64_t *ikey, double4 *ival, int lvl, Tables T,
                                const double4 *B0) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= NInt) return;
    const uint64_t k = ikey[i];
    if ((int)(k & 15u) != lvl) return;
    double4 c[4];
    int64_t at = i;   // the sons that are internal come after this node, in key order
    for (int q = 0; q < 4; ++q) {
        const uint64_t ck = child_key(k, q);
        const int64_t li = find_key_t(T, ck);
        if (li >= 0) {
            c[q] = B0[T.lslot[li]];
        } else {
            int64_t lo = at + 1, hi = NInt;
            while (lo < hi) {
                const int64_t mid = (lo + hi) >> 1;
                if (ikey[mid] < ck) lo = mid + 1;
                else hi = mid;
            }
            at = lo;
            c[q] = lo < NInt && ikey[lo] == ck ? ival[lo] : make_double4(0, 0, 0, 0);
        }
    }
    ival[i] = mean4(c[0], c[1], c[2], c[3]);
}

// The current and the next node set; each has its three arrays (amr[0..2],
// amr[3..5]) and its per-cell index (amr[6], amr[7]), which the kernel that
// writes the set fills too: a cell's first node is its root node.
struct AmrCtx {
    fdm_handle *h;
    NodeSet A, B;
    int a = 0;   // which buffers hold A
};

// room for n nodes in the next set; the current one stays as it is
static int grow_next(fdm_handle *h, AmrCtx &X, int64_t n) {
    const int b = 1 - X.a;
    const int64_t nroots = (int64_t)h->G.m * h->G.n;
    FDM_CK(h, h->amr[3 * b + 0].ensure(n * 8));
    FDM_CK(h, h->amr[3 * b + 1].ensure(n));
    FDM_CK(h, h->amr[3 * b + 2].ensure(n * 32));
    FDM_CK(h, h->amr[6 + b].ensure((nroots + 1) * 4));
    X.B.key = h->amr[3 * b + 0].as<uint64_t>();
    X.B.leaf = h->amr[3 * b + 1].as<uint8_t>();
    X.B.val = h->amr[3 * b + 2].as<double4>();
    X.B.rf = h->amr[6 + b].as<int32_t>();
    X.B.nroots = nroots;
    X.B.n = n;
    return FDM_OK;
}
static void swap_sets(AmrCtx &X) {
    X.a = 1 - X.a;
    std::swap(X.A, X.B);
}
// the index entry of node k stored at o (and the end of the index)
__device__ __forceinline__ void index_node(const NodeSet &out, uint64_t k, int64_t o) {
    if ((k & 15u) == 0) out.rf[k >> 34] = (int32_t)o;
}
__device__ __forceinline__ void index_end(const NodeSet &out) { out.rf[out.nroots] = (int32_t)out.n; }

// Merge of two key-sorted runs (keys distinct) into the node set out: an
// entry's place is its index in its run plus the number of keys of the
// other run below it.
__global__ void k_merge_runs(const uint64_t *__restrict__ ka, const uint8_t *__restrict__ la,
                             const double4 *__restrict__ va, int64_t na, const uint64_t *__restrict__ kb,
                             const uint8_t *__restrict__ lb, const double4 *__restrict__ vb, int64_t nb, NodeSet out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= na + nb) return;
    const bool in_a = i < na;
    const int64_t j = in_a ? i : i - na;
    const uint64_t k = in_a ? ka[j] : kb[j];
    const uint64_t *other = in_a ? kb : ka;
    int64_t lo = 0, hi = in_a ? nb : na;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (other[mid] < k) lo = mid + 1;
        else hi = mid;
    }
    const int64_t o = j + lo;
    out.key[o] = k;
    out.leaf[o] = in_a ? la[j] : lb[j];
    out.val[o] = in_a ? va[j] : vb[j];
    index_node(out, k, o);
    if (i == 0) index_end(out);
}
// the runs [0, m) and [m, n) of (keys, leaf, val), each sorted, into out
static void merge_into(fdm_handle *h, const uint64_t *keys, const uint8_t *leaf, const double4 *val, int64_t m,
                       int64_t n, const NodeSet &out) {
    if (n > 0)
        k_merge_runs<<<nblk(n, 256), 256, 0, h->s>>>(keys, leaf, val, m, keys + m, leaf + m, val + m, n - m, out);
}
// exclusive scan of n counts and their total; *at_val: the prefix at index
// at (0 <= at < n); nwords device words come back in h->pin in the same round
// trip
static int scan_total32(fdm_handle *h, const int32_t *in, int32_t *out, int64_t n, int64_t &total,
                        int64_t at = -1, int64_t *at_val = nullptr, const int32_t *words = nullptr, int nwords = 0) {
    int32_t *r = h->pin_scan();
    FDM_CK(h, launch_scan(h, ScanArgs<int32_t>{in, out, n, r, nullptr, at_val ? at : -1, r + 1, words, h->pin, nwords}));
    FDM_CK(h, cudaStreamSynchronize(h->s));
    total = (int64_t)r[0];
    if (at_val) *at_val = at >= n ? total : (int64_t)r[1];
    return FDM_OK;
}

// internal nodes and their interpA values from the current leaf set
// (values as the reference's import of a leaf set would give them)
int init_internal(fdm_handle *h) {
    const int TB = 256;
    const int64_t NL = h->NL;
    Carve cv;
    cv.add(NL * 4); cv.add(NL * 4); cv.add(4);
    FDM_CK(h, h->amr[8].ensure(cv.total));
    int32_t *cnt = cv.at<int32_t>(h->amr[8], 0), *off = cv.at<int32_t>(h->amr[8], 1);
    int32_t *dl = cv.at<int32_t>(h->amr[8], 2), *deepest = h->pin;   // deepest leaf
    FDM_CK(h, cudaMemsetAsync(dl, 0, 4, h->s));
    k_anc_count<<<nblk(NL, TB), TB, 0, h->s>>>(NL, h->lkey.as<uint64_t>(), cnt, dl);
    int64_t ni = 0;
    int rc = scan_total32(h, cnt, off, NL, ni, -1, nullptr, dl, 1);   // waits
    if (rc) return rc;
    h->NInt = ni;
    if (ni == 0) return FDM_OK;
    FDM_CK(h, h->ikey.ensure(ni * 8));
    k_anc_emit<<<nblk(NL, TB), TB, 0, h->s>>>(NL, h->lkey.as<uint64_t>(), off, h->ikey.as<uint64_t>());
    FDM_CK(h, h->ival.ensure(ni * 32 + 32));
    for (int l = *deepest - 1; l >= 0; --l)
        k_internal_vals<<<nblk(ni, TB), TB, 0, h->s>>>(ni, h->ikey.as<uint64_t>(), h->ival.as<double4>(), l,
                                                      h->tables(), h->B[0].as<double4>());
    FDM_CK(h, cudaGetLastError());
    return FDM_OK;
}

// ----------------------------------------------------------- solute_ref
// refine flags of the leaves (solute_ref_sub, src/solution.F90:519-535)
__global__ void k_refine_flags(Tables T, Geometry G, fdm_params P, const double *rot_slot, const double *div_slot,
                               const double *sums, int8_t *rflag) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= T.NL) return;
    const uint64_t key = T.lkey[k];
    const int lvl = (int)(key & 15u);
    const int cr = root_cross(G, (int64_t)(key >> 34));
    const int32_t s = T.lslot[k];
    rflag[k] = 0;
    if ((cr == 0 || cr == 1) && lvl < P.lvl_amr && s < T.NI) {
        const double arot = sqrt(sums[0] / sums[2]);
        const double adiv = sqrt(sums[1] / sums[2]);
        if (rot_slot[s] > P.refine_goal_rot * arot || div_slot[s] > P.refine_goal_div * adiv) rflag[k] = 1;
    }
}
// coarsen flags of internal nodes (solute_coarse_sub, src/solution.F90:490-517):
// all four sons are leaves, none refined in this pass, means below the goals
__global__ void k_coarsen_flags(int64_t NInt, const uint64_t *ikey, Tables T, fdm_params P, const double *rot_slot,
                                const double *div_slot, const double *sums, const int8_t *rflag, int8_t *cflag) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= NInt) return;
    cflag[i] = 0;
    const uint64_t k = ikey[i];
    if ((int)(k & 15u) >= P.lvl_amr) return;
    double r[4], d[4];
    for (int q = 0; q < 4; ++q) {
        const int64_t li = find_key_t(T, child_key(k, q));
        if (li < 0 || rflag[li]) return;
        const int32_t s = T.lslot[li];
        r[q] = s < T.NI ? rot_slot[s] : 0.0;
        d[q] = s < T.NI ? div_slot[s] : 0.0;
    }
    const double arot = sqrt(sums[0] / sums[2]);
    const double adiv = sqrt(sums[1] / sums[2]);
    // son1 + son2 + son3 + son4 = q0 + q1 + q3 + q2
    if ((r[0] + r[1] + r[3] + r[2]) / 4 < P.coarse_goal_rot * arot &&
        (d[0] + d[1] + d[3] + d[2]) / 4 < P.coarse_goal_div * adiv)
        cflag[i] = 1;
}
__global__ void k_ref_count(Tables T, const int8_t *rflag, const uint64_t *ikey, int64_t NInt, const int8_t *cflag,
                            int32_t *cnt) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k < T.NL) {
        const uint64_t key = T.lkey[k];
        int c = rflag[k] ? 5 : 1;
        if ((key & 15u) > 0) {
            const int64_t pi = find_key(ikey, NInt, parent_key(key));
            if (pi >= 0 && cflag[pi]) c = 0;
        }
        cnt[k] = c;
    } else if (k < T.NL + NInt) {
        cnt[k] = 1;
    }
}
__global__ void k_ref_emit(Tables T, const double4 *B0, const int8_t *rflag, const uint64_t *ikey, const double4 *ival,
                           int64_t NInt, const int8_t *cflag, const int32_t *off, uint64_t *okey, uint8_t *oleaf,
                           double4 *oval) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k < T.NL) {
        const uint64_t key = T.lkey[k];
        if ((key & 15u) > 0) {
            const int64_t pi = find_key(ikey, NInt, parent_key(key));
            if (pi >= 0 && cflag[pi]) return;
        }
        const double4 v = B0[T.lslot[k]];
        int64_t o = off[k];
        okey[o] = key; oleaf[o] = rflag[k] ? 0 : 1; oval[o] = v;
        if (rflag[k]) {   // Refine_cell: sons copy U (src/mesh.F90:210-252)
            for (int q = 0; q < 4; ++q) {
                okey[o + 1 + q] = child_key(key, q); oleaf[o + 1 + q] = 1; oval[o + 1 + q] = v;
            }
        }
    } else if (k < T.NL + NInt) {
        const int64_t i = k - T.NL;
        const uint64_t key = ikey[i];
        const int64_t o = off[k];
        okey[o] = key;
        if (cflag[i]) {   // Coarse_cell: interpA of the four leaf sons (src/mesh.F90:397-408)
            double4 c[4];
            for (int q = 0; q < 4; ++q) c[q] = B0[T.lslot[find_key_t(T, child_key(key, q))]];
            oleaf[o] = 1;
            oval[o] = mean4(c[0], c[1], c[2], c[3]);
        } else {
            oleaf[o] = 0;
            oval[o] = ival[i];
        }
    }
}

// The largest cluster of blocks, for the kernels that iterate: the hardware's
// cluster barrier costs a fraction of a launch or a grid-wide barrier.
constexpr int CLUSTER_CTAS = 16, CLUSTER_TB = 1024;

template <class... P, class... A>
static cudaError_t launch_cluster(cudaStream_t s, void (*kernel)(P...), A... args) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CLUSTER_CTAS);
    cfg.blockDim = dim3(CLUSTER_TB);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CLUSTER_CTAS;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// ----------------------------------------------------------- gridmodify1
struct Links {
    int32_t *parent, *child, *nb;   // child[4 n], nb[4 n] (up, down, right, left)
    uint64_t *rank;                 // post-order rank key of the visit (post_rank): compared, never indexed
    uint8_t *leaf0;
    int8_t *cross;
};
__device__ __forceinline__ void gm1_link(const NodeSet &A, const Geometry &G, const Links &L, int8_t *d, int64_t i) {
    d[i] = D_NONE;
    const uint64_t k = A.key[i];
    const int lvl = (int)(k & 15u);
    L.parent[i] = lvl > 0 ? (int32_t)find_key_set(A, parent_key(k)) : -1;
    L.leaf0[i] = A.leaf[i];
    L.cross[i] = (int8_t)root_cross(G, (int64_t)(k >> 34));
    for (int q = 0; q < 4; ++q)
        L.child[4 * i + q] = A.leaf[i] ? -1 : (int32_t)find_key_set(A, child_key(k, q));
    for (int d = 0; d < 4; ++d) {
        uint64_t nk;
        L.nb[4 * i + d] = shift_key(G, k, d, nk) ? (int32_t)find_key_set(A, nk) : -1;
    }
    L.rank[i] = post_rank(k);
}
__global__ void k_gm1_links(NodeSet A, Geometry G, Links L, int8_t *d) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < A.n) gm1_link(A, G, L, d, i);
}
// "the same-level node N exists and has sons" when x is visited: decisions
// of earlier-visited nodes applied.  N is gone when a node above it was
// coarsened; then its father was (a node is coarsened only when its sons are
// leaves or coarsened, and sons come first), so the father's decision tells.
__device__ __forceinline__ bool gm1_has_son(const Links &L, const int8_t *d, int32_t N, uint64_t rx) {
    if (N < 0) return false;
    const int32_t p = L.parent[N];
    const int8_t dn = d[N];
    const bool leaf = L.leaf0[N];
    if (p >= 0 && d[p] == D_COARSEN && L.rank[p] < rx) return false;
    if (leaf) return dn == D_REFINE && L.rank[N] < rx;
    return !(dn == D_COARSEN && L.rank[N] < rx);
}
// gridmodify1 decision of one node (src/mesh.F90:305-353) given the current
// estimate of all decisions; a decision only reads decisions of nodes that
// are visited earlier, so iterating to a fixpoint gives the sequential result.
// The estimate is updated in place: a decision may read others already
// updated in the same sweep (never older than the last sweep's), which only
// shortens the chains; a sweep that changes nothing wrote nothing, so every
// decision in it read final values and the fixpoint (unique: the
// dependencies follow the visit order) is reached.  changed: one word per
// sweep; a sweep after one that changed nothing has nothing to do, so several
// are queued without a look from the host.
__device__ __forceinline__ bool gm1_decide(const Links &L, int8_t *d, int64_t x) {   // true: the decision changed
    int8_t r = D_NONE;
    if (L.cross[x] == 0) {
        const uint64_t rx = L.rank[x];
        const int4 v = *reinterpret_cast<const int4 *>(L.nb + 4 * x);
        const int32_t N[4] = {v.x, v.y, v.z, v.w};
        const bool up = gm1_has_son(L, d, N[DIR_UP], rx), down = gm1_has_son(L, d, N[DIR_DOWN], rx);
        const bool left = gm1_has_son(L, d, N[DIR_LEFT], rx), right = gm1_has_son(L, d, N[DIR_RIGHT], rx);
        if (L.leaf0[x]) {
            if ((left && right) || (up && down)) r = D_REFINE;
        } else {
            bool all_leaf = true;
            for (int q = 0; q < 4; ++q) {
                const int32_t c = L.child[4 * x + q];
                const bool lf = c >= 0 && ((L.leaf0[c] && d[c] != D_REFINE) || (!L.leaf0[c] && d[c] == D_COARSEN));
                all_leaf = all_leaf && lf;
            }
            if (all_leaf && ((!left && !right) || (!up && !down))) r = D_COARSEN;
        }
    }
    if (r == d[x]) return false;
    d[x] = r;
    return true;
}
__global__ void k_gm1_decide(int64_t n, Links L, int8_t *d, int32_t *changed, int sweep) {
    const int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (x >= n || (sweep > 0 && changed[sweep - 1] == 0)) return;
    if (gm1_decide(L, d, x)) changed[sweep] = 1;
}
// values of coarsened nodes, deepest level first (interpA of the sons as they
// are at the node's visit)
__global__ void k_gm1_vals(NodeSet A, Links L, const int8_t *d, int lvl) {
    const int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (x >= A.n || d[x] != D_COARSEN || (int)(A.key[x] & 15u) != lvl) return;
    const int32_t *c = L.child + 4 * x;
    A.val[x] = mean4(A.val[c[0]], A.val[c[1]], A.val[c[2]], A.val[c[3]]);
}
// the node goes: its father was coarsened, or one further up, and so the father too
__device__ __forceinline__ bool ancestor_coarsened(const Links &L, const int8_t *d, int32_t x) {
    const int32_t p = L.parent[x];
    return p >= 0 && d[p] == D_COARSEN;
}
// did[0]: a node is refined or coarsened; did[1]: the longest chain of
// coarsened nodes, each the father of the next; did[2]: their deepest level
__device__ __forceinline__ void gm1_count(const NodeSet &A, const Links &L, const int8_t *d, int32_t *cnt, int32_t *did,
                                          int64_t x) {
    const int8_t dx = d[x];
    cnt[x] = ancestor_coarsened(L, d, (int32_t)x) ? 0 : (dx == D_REFINE ? 5 : 1);
    if (dx == D_NONE) return;
    did[0] = 1;
    if (dx != D_COARSEN) return;
    int chain = 1;
    for (int32_t a = L.parent[x]; a >= 0 && d[a] == D_COARSEN; a = L.parent[a]) ++chain;
    const int lvl = (int)(A.key[x] & 15u);
    if (did[1] < chain) atomicMax(did + 1, chain);
    if (did[2] < lvl) atomicMax(did + 2, lvl);
}
__global__ void k_gm1_count(NodeSet A, Links L, const int8_t *d, int32_t *cnt, int32_t *did) {
    const int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (x < A.n) gm1_count(A, L, d, cnt, did, x);
}
// The pass up to the counts in one launch of a cluster, for small sets: links,
// sweeps until one changes nothing, counts.  w: [0..2] changes by sweep modulo
// 3, GM1_DID.. the did words, then the sweeps; -1 there: not settled.
enum { GM1_DID = 3, GM1_NSWEEPS = 6, GM1_W = 7 };
__global__ void __launch_bounds__(CLUSTER_TB) k_gm1_pass(NodeSet A, Geometry G, Links L, int8_t *d, int32_t *cnt,
                                                         int32_t *w) {
    const int nthr = CLUSTER_CTAS * CLUSTER_TB, me = blockIdx.x * CLUSTER_TB + threadIdx.x, n = (int)A.n;
    if (me < GM1_W) w[me] = 0;
    for (int x = me; x < n; x += nthr) gm1_link(A, G, L, d, x);
    cluster_barrier();
    int sweep = 0;
    for (;; ++sweep) {
        bool changed = false;
        for (int x = me; x < n; x += nthr) changed |= gm1_decide(L, d, x);
        if (__any_sync(0xffffffffu, changed) && (threadIdx.x & 31) == 0) __stcg(w + sweep % 3, 1);
        if (me == 0) __stcg(w + (sweep + 1) % 3, 0);   // last read before the barrier of the sweep before
        cluster_barrier();
        if (__ldcg(w + sweep % 3) == 0 || sweep > n + 2) break;
    }
    for (int x = me; x < n; x += nthr) gm1_count(A, L, d, cnt, w + GM1_DID, x);
    if (me == 0) w[GM1_NSWEEPS] = sweep > n + 2 ? -1 : sweep + 1;
}
// mean: a coarsened node's value is formed here from its sons' (no chain of
// coarsened nodes); otherwise k_gm1_vals has formed it
__global__ void k_gm1_emit(NodeSet A, Links L, const int8_t *d, const int32_t *off, NodeSet out, bool mean) {
    const int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (x == 0) index_end(out);
    if (x >= A.n || ancestor_coarsened(L, d, (int32_t)x)) return;
    const int64_t o = off[x];
    const uint64_t k = A.key[x];
    const int8_t dx = d[x];
    double4 v;
    if (mean && dx == D_COARSEN) {
        const int32_t *c = L.child + 4 * x;
        v = mean4(A.val[c[0]], A.val[c[1]], A.val[c[2]], A.val[c[3]]);
    } else {
        v = A.val[x];
    }
    out.key[o] = k;
    out.val[o] = v;
    out.leaf[o] = dx == D_REFINE ? 0 : dx == D_COARSEN ? 1 : A.leaf[x];
    index_node(out, k, o);
    if (dx == D_REFINE)
        for (int q = 0; q < 4; ++q) {
            out.key[o + 1 + q] = child_key(k, q);
            out.leaf[o + 1 + q] = 1;
            out.val[o + 1 + q] = v;
        }
}

// ----------------------------------------------------------- gridmodify4
// gridmodify4 (src/mesh.F90:355-395) visits the leaves in traversal order
// (sons 1,2,3,4), those created ahead of the traversal included.  A leaf c
// looks right, left, up, down: it refines a neighbour two or more levels
// coarser, then that neighbour's neighbour in the same direction when that
// one is.  Every Refine_cell therefore has a time of its own, (visit rank of
// c, direction, neighbour or neighbour's neighbour), and the whole pass is
// the map t: node -> time of its Refine_cell (GM4_NEVER if none), which
// obeys, for every leaf c that is still a leaf when its turn comes,
//
//     t(N) = min over the looks that find N two levels coarser of their time,
//
// where a look at time T sees the node set as it is then: a node exists at T
// when its father was refined before T.  So a look depends on earlier times
// only; t is the unique fixpoint, and iterating "all looks from the current
// estimate of t" reaches it: after k sweeps every Refine_cell whose chain of
// causes has at most k links is final, and a sweep that changes nothing
// proves the rest.  A chain has a link per level of a cascade and per leaf
// whose look an earlier refinement answers differently, 4 to 9 sweeps on the
// developed four-quadrant and double Mach meshes.
//
// The one effect outside the map is the Refine_cell of a node that has sons
// (:389-392), which drops its subtree.  Its time is known at the fixpoint
// (the earliest look that finds such a node); the node set up to and
// including it is then written out and the pass goes on from that time on
// the new set.  It happens about once in 1300 refinements.

constexpr uint64_t GM4_NEVER = ~0ull;
// time of look s (0..7: direction, then neighbour / neighbour's neighbour) of
// the leaf with visit rank r: below 2^57, above 0
FDM_HD uint64_t gm4_time(uint64_t r, int s) { return ((r << 3) | (uint64_t)s) + 1u; }
// the reference's direction order: right, left, up, down
__device__ __forceinline__ int gm4_dir(int t) { return (t + DIR_RIGHT) & 3; }

// The node of A that holds position key_pos(k): the last one that starts at
// or before it, always a leaf (an internal node's first son starts where it
// does and comes after it).
__device__ __forceinline__ int64_t holder(const NodeSet &A, uint64_t k) {
    const uint64_t pos = key_pos(k);
    const int64_t r = (int64_t)(k >> 34);
    int64_t lo = __ldg(A.rf + r), hi = (int64_t)__ldg(A.rf + r + 1) - 1;
    while (lo < hi) {
        const int64_t mid = (lo + hi + 1) >> 1;
        if (key_pos(__ldg(A.key + mid)) <= pos) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}
// Is the node with key s (or the position s stands for) inside node r?
__device__ __forceinline__ bool key_inside(uint64_t r, uint64_t s) {
    const int lr = (int)(r & 15u), ls = (int)(s & 15u);
    if (lr > ls || (r >> 34) != (s >> 34)) return false;
    const uint64_t path_mask = (1ull << 30) - 1ull;
    const uint64_t keep = lr == 0 ? 0ull : (path_mask & ~((1ull << (30 - 2 * lr)) - 1ull));
    return (((s >> 4) & path_mask) & keep) == ((r >> 4) & path_mask);
}

// Leaves that can act: a neighbour, or the neighbour's neighbour, two or
// more levels coarser in the node set at the start.  Refining a leaf only
// makes neighbours finer, so no other leaf of the set can act later.  Four
// lanes per node, one per direction; the leaves are appended to list in no
// particular order.  Only leaves whose looks come after time t0 count.
__global__ void __launch_bounds__(256) k_gm4_triggers(NodeSet A, Geometry G, uint64_t t0, int32_t *list,
                                                      int32_t *count) {
    const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t c = g >> 2;
    bool acts = false;
    if (c < A.n && A.leaf[c]) {
        const uint64_t k = A.key[c];
        const int lc = (int)(k & 15u), d = gm4_dir((int)(g & 3));
        uint64_t s;
        if (lc >= 2 && gm4_time(visit_rank(k), 7) > t0 && shift_key(G, k, d, s)) {
            const uint64_t nb = __ldg(A.key + holder(A, s));
            const int ln = min((int)(nb & 15u), lc);   // deeper: the same-level node has sons
            acts = ln <= lc - 2;
            if (!acts && shift_key(G, ln < lc ? nb : s, d, s))
                acts = (int)(__ldg(A.key + holder(A, s)) & 15u) <= lc - 2;
        }
    }
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(0xffffffffu, acts);
    const bool first = (lane & 3) == 0 && ((m >> lane) & 0xFu) != 0;   // one lane per acting leaf
    const unsigned fm = __ballot_sync(0xffffffffu, first);
    int base = 0;
    if (lane == 0 && fm) base = atomicAdd(count, __popc(fm));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (first) list[base + __popc(fm & ((1u << lane) - 1u))] = (int32_t)c;
}

// The map t and the nodes made on the way.  Nodes are named by their index
// in A (below n) or n + the order in which they were made; a node that some
// sweep refines gets four sons (first one: son), in key order, which stay
// even when a later sweep takes the refinement back (t = GM4_NEVER again).
struct Gm4 {
    uint64_t *t, *tn;      // [n + cap] current estimate, next one
    int32_t *son;          // [n + cap] first son, -1 none
    uint64_t *mkey;        // [cap] key of a made node
    int32_t *mfather;      // [cap] its father
    int32_t *refd;         // [n + cap] nodes that some sweep refined
    const int32_t *list;   // the leaves of A that can act
    int64_t cap;
    uint64_t *nl;          // [2] earliest refinement of a node with sons, by sweep parity
    int32_t *w;            // GW_* words
};
enum { GW_NLIST = 0, GW_MADE, GW_NREFD, GW_CHG0, GW_CHG1, GW_FULL, GW_STUCK, GW_SWEEPS, GW_VISITS, GW_REFINES,
       GW_NONLEAF, GW_WORDS };
struct Gm4Result {         // read back by the host
    int32_t w[GW_WORDS + 1];
    uint64_t nl_time, nl_key;
};

__device__ __forceinline__ uint64_t gm4_key(const NodeSet &A, const Gm4 &M, int32_t id) {
    return id < A.n ? __ldg(A.key + id) : __ldcg(M.mkey + (id - A.n));
}
// What a look from s towards the node at s's level finds at time T: the node
// itself (same: with its level that of s) or the leaf above it.  id is the
// node's name, or -1 for a node of A that has sons.  at holds the node of A
// at s where it is known already (-1: not), since it never changes.
struct Found {
    uint64_t key;
    int32_t id;
    bool sons;
};
__device__ __forceinline__ Found gm4_look(const NodeSet &A, const Gm4 &M, uint64_t s, uint64_t T, int32_t &at) {
    Found f;
    const int ls = (int)(s & 15u);
    if (at < 0) at = (int32_t)holder(A, s);
    int32_t id = at;
    uint64_t k = __ldg(A.key + id);
    int l = (int)(k & 15u);
    if (l > ls) {
        f.key = s; f.id = -1; f.sons = true;
        return f;
    }
    bool sons = __ldcg(M.t + id) < T;
    while (l < ls && sons) {
        ++l;
        id = __ldcg(M.son + id) + (int32_t)((s >> key_digit_shift(l)) & 3u);
        k = ancestor_key(s, l);
        sons = __ldcg(M.t + id) < T;
    }
    f.key = k; f.id = id; f.sons = sons;
    return f;
}
// look s of the leaf with key k and visit rank r: the neighbour (tn.id >= 0
// when it refines it) and the neighbour's neighbour
struct Looks {
    int32_t nb, nn;          // nodes refined, or -1
    bool nonleaf;            // the neighbour's neighbour is refined and has sons
    uint64_t nnkey;
};
// where a look's two searches ended in an earlier sweep
struct Seen {
    uint64_t s2;          // start of the second one
    int32_t at1, at2;
};
__device__ __forceinline__ Looks gm4_looks(const NodeSet &A, const Geometry &G, const Gm4 &M, uint64_t k, uint64_t r,
                                           int t, Seen &seen) {
    Looks L;
    L.nb = L.nn = -1;
    L.nonleaf = false;
    L.nnkey = 0;
    const int lc = (int)(k & 15u), d = gm4_dir(t);
    uint64_t s;
    if (!shift_key(G, k, d, s)) return L;
    const Found b = gm4_look(A, M, s, gm4_time(r, 2 * t), seen.at1);
    if ((int)(b.key & 15u) <= lc - 2) L.nb = b.id;   // no node at lc: a leaf
    if (!shift_key(G, b.key, d, s)) return L;
    if (s != seen.s2) {
        seen.s2 = s;
        seen.at2 = -1;
    }
    const Found n = gm4_look(A, M, s, gm4_time(r, 2 * t + 1), seen.at2);
    if ((int)(n.key & 15u) <= lc - 2) {
        L.nnkey = n.key;
        if (n.sons) L.nonleaf = true;
        else L.nn = n.id;
    }
    return L;
}
// is node id a leaf when its turn (rank r) comes, after time t0?
__device__ __forceinline__ bool gm4_visited(const NodeSet &A, const Gm4 &M, int32_t id, uint64_t r) {
    const uint64_t T = gm4_time(r, 0);
    if (__ldcg(M.t + id) < T) return false;
    return id < A.n || __ldcg(M.t + __ldcg(M.mfather + (id - A.n))) < T;
}
__device__ __forceinline__ void gm4_propose(const NodeSet &A, const Gm4 &M, int32_t id, uint64_t T) {
    atomicMin((unsigned long long *)(M.tn + id), (unsigned long long)T);
    if (__ldcg(M.son + id) != -1) return;
    if (atomicCAS(M.son + id, -1, -2) != -1) return;   // the first sweep that refines it makes its sons
    const int32_t j = atomicAdd(M.w + GW_MADE, 4);
    if (j + 4 > M.cap) {
        M.w[GW_FULL] = 1;
        return;
    }
    const uint64_t k = gm4_key(A, M, id);
    for (int q = 0; q < 4; ++q) {
        __stcg(M.mkey + j + q, child_key(k, q));
        __stcg(M.mfather + j + q, id);
    }
    __stcg(M.son + id, (int32_t)(A.n + j));
    M.refd[atomicAdd(M.w + GW_NREFD, 1)] = id;
}


// The fixpoint, by one cluster of blocks: a sweep is all looks (four lanes
// per leaf, one per direction), a cluster barrier, then the comparison of
// the two estimates over the nodes ever refined, and another barrier.  The
// hardware's cluster barrier costs a fraction of a grid-wide one, and a pass
// has a few thousand looks: it is bound by the latency of a look (two
// searches in a background cell's nodes, about 20 dependent L2 reads) times
// the sweeps, not by the number of SMs.  One B200, two regrids of a developed
// 128^2, 4-level four-quadrant run (82k leaves, 2029 refinements): 0.67 ms in
// 39 sweeps with 8 blocks (0.94 before a thread kept where its look's searches
// ended), 0.51 with 16, the largest cluster: the last sweeps' looks are several
// a thread; against 14.0 ms for visiting the leaves in order by one block.
// 256 x 64 double Mach at 4 levels, four regrids: 0.72 ms (0.82 with 8 blocks),
// against 10.2.
__global__ void __launch_bounds__(CLUSTER_TB) k_gm4_fixpoint(NodeSet A, Geometry G, Gm4 M, uint64_t t0, int max_sweeps, Gm4Result *out) {
    const int nthr = CLUSTER_CTAS * CLUSTER_TB;
    const int me = blockIdx.x * CLUSTER_TB + threadIdx.x;
    const int nlist = __ldcg(M.w + GW_NLIST);
    int made = 0;        // made nodes that this sweep visits
    int sweep = 0;
    bool full = false;
    Seen mine{0, -1, -1};
    if (nlist > 0) {
        for (;; ++sweep) {
            const int par = sweep & 1;
            const int64_t looks = 4 * ((int64_t)nlist + made);
            const auto look = [&](int64_t x, Seen &seen) {
                const int v = (int)(x >> 2), t = (int)(x & 3);
                const int32_t id = v < nlist ? __ldg(M.list + v) : (int32_t)(A.n + (v - nlist));
                const uint64_t k = gm4_key(A, M, id), r = visit_rank(k);
                if (gm4_time(r, 7) <= t0 || !gm4_visited(A, M, id, r)) return;
                const Looks L = gm4_looks(A, G, M, k, r, t, seen);
                const uint64_t Tb = gm4_time(r, 2 * t), Tn = gm4_time(r, 2 * t + 1);
                if (L.nb >= 0 && Tb > t0) gm4_propose(A, M, L.nb, Tb);
                if (Tn > t0) {
                    if (L.nonleaf) atomicMin((unsigned long long *)(M.nl + par), (unsigned long long)Tn);
                    else if (L.nn >= 0) gm4_propose(A, M, L.nn, Tn);
                }
            };
            // a thread's first look is the same one in every sweep
            if (me < looks) look(me, mine);
            for (int64_t x = me + nthr; x < looks; x += nthr) {
                Seen once{0, -1, -1};
                look(x, once);
            }
            cluster_barrier();
            const int nrefd = __ldcg(M.w + GW_NREFD);
            made = __ldcg(M.w + GW_MADE);
            full = made > M.cap || __ldcg(M.w + GW_FULL) != 0;
            bool changed = false;
            for (int x = me; x < nrefd; x += nthr) {
                const int32_t id = __ldcg(M.refd + x);
                const uint64_t a = __ldcg(M.t + id), b = __ldcg(M.tn + id);
                if (a != b) {
                    __stcg(M.t + id, b);
                    changed = true;
                }
                __stcg(M.tn + id, GM4_NEVER);
            }
            if (__any_sync(0xffffffffu, changed) && (threadIdx.x & 31) == 0) __stcg(M.w + GW_CHG0 + par, 1);
            if (me == 0) {   // last read before this sweep's first barrier
                __stcg(M.w + GW_CHG0 + (par ^ 1), 0);
                __stcg(M.nl + (par ^ 1), GM4_NEVER);
            }
            cluster_barrier();
            if (full || __ldcg(M.w + GW_CHG0 + par) == 0 || sweep >= max_sweeps) break;
        }
    }
    const uint64_t nl = nlist > 0 ? __ldcg(M.nl + (sweep & 1)) : GM4_NEVER;
    if (nlist > 0 && !full) {
        // counts, of what comes no later than the first refinement of a node
        // with sons
        const int nrefd = __ldcg(M.w + GW_NREFD);
        int refines = 0, visits = 0;
        for (int x = me; x < nrefd; x += nthr) refines += __ldcg(M.t + __ldcg(M.refd + x)) < nl ? 1 : 0;
        for (int v = me; v < nlist + made; v += nthr) {
            const int32_t id = v < nlist ? __ldg(M.list + v) : (int32_t)(A.n + (v - nlist));
            const uint64_t r = visit_rank(gm4_key(A, M, id)), T = gm4_time(r, 0);
            visits += T > t0 && T <= nl && gm4_visited(A, M, id, r) ? 1 : 0;
        }
        refines = __reduce_add_sync(0xffffffffu, refines);
        visits = __reduce_add_sync(0xffffffffu, visits);
        if ((threadIdx.x & 31) == 0) {
            if (refines) atomicAdd(M.w + GW_REFINES, refines);
            if (visits) atomicAdd(M.w + GW_VISITS, visits);
        }
    }
    cluster_barrier();
    if (me == 0) {
        uint64_t nlkey = 0;
        if (nl != GM4_NEVER && !full) {   // the look of that time again, for its node
            const uint64_t r = (nl - 1u) >> 3;
            Seen once{0, -1, -1};
            nlkey = gm4_looks(A, G, M, key_of_visit_rank(r), r, (int)((nl - 1u) & 7u) >> 1, once).nnkey;
        }
        for (int q = 0; q < GW_WORDS; ++q) out->w[q] = __ldcg(M.w + q);
        out->w[GW_FULL] = full;
        out->w[GW_STUCK] = nlist > 0 && !full && __ldcg(M.w + GW_CHG0 + (sweep & 1)) != 0;
        out->w[GW_SWEEPS] = nlist > 0 ? sweep + 1 : 0;
        out->w[GW_NONLEAF] = nl != GM4_NEVER;
        out->nl_time = nl;
        out->nl_key = nlkey;
    }
}

// The nodes of the set after the pass that come from node i of A, in key
// order: node i itself and, below a leaf that was refined, its made subtree.
// The node refined although it had sons (res->nl_key) keeps four new leaves
// and loses what was below it.  All of them carry node i's value
// (Refine_cell copies U, src/mesh.F90:210-252).  Returns their number;
// WRITE: stores them from place o on.
template <bool WRITE>
__device__ __forceinline__ int gm4_nodes(const NodeSet &A, const Gm4 &M, const Gm4Result *res, int64_t i, int64_t o,
                                         NodeSet out) {
    const uint64_t k0 = A.key[i], nl = res->nl_time, nlkey = res->nl_key;
    const bool hasnl = nl != GM4_NEVER;
    double4 v = make_double4(0.0, 0.0, 0.0, 0.0);
    if (WRITE) v = A.val[i];
    int n = 0;
    const auto put = [&](uint64_t k, bool leaf) {
        if (WRITE) {
            index_node(out, k, o + n);
            out.key[o + n] = k;
            out.leaf[o + n] = leaf ? 1 : 0;
            out.val[o + n] = v;
        }
        ++n;
    };
    if (hasnl && key_inside(nlkey, k0)) {
        if (k0 != nlkey) return 0;   // dropped
        put(k0, false);
        for (int q = 0; q < 4; ++q) put(child_key(k0, q), true);
        return n;
    }
    if (!A.leaf[i] || M.t[i] >= nl) {   // nl is GM4_NEVER when there is none
        put(k0, A.leaf[i] != 0);
        return n;
    }
    int32_t st[3 * LMAX + 4];
    int sp = 0;
    st[sp++] = (int32_t)i;
    while (sp > 0) {
        const int32_t id = st[--sp];
        const uint64_t k = id < A.n ? k0 : M.mkey[id - A.n];
        const bool refined = M.t[id] < nl;
        put(k, !refined);
        if (!refined) continue;
        if (hasnl && k == nlkey) {
            for (int q = 0; q < 4; ++q) put(child_key(k, q), true);
        } else {
            for (int q = 3; q >= 0; --q) st[sp++] = M.son[id] + q;
        }
    }
    return n;
}
__global__ void k_gm4_count(NodeSet A, Gm4 M, const Gm4Result *res, int32_t *cnt) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < A.n) cnt[i] = res->w[GW_FULL] ? 1 : gm4_nodes<false>(A, M, res, i, 0, A);
}
__global__ void k_gm4_emit(NodeSet A, Gm4 M, const Gm4Result *res, const int32_t *off, NodeSet out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i == 0) index_end(out);
    if (i < A.n) gm4_nodes<true>(A, M, res, i, off[i], out);
}

// ------------------------------------------------------------ extraction
__global__ void k_split_count(int64_t n, const uint8_t *leaf, int32_t *fl) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) fl[i] = leaf[i] ? 1 : 0;
}
// ol: leaves before each node; the internal nodes before it are the others
__global__ void k_split_emit(NodeSet A, const int32_t *ol, uint64_t *lk, double4 *lv, uint64_t *ik, double4 *iv) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    const int64_t l = ol[i];
    if (A.leaf[i]) { lk[l] = A.key[i]; lv[l] = A.val[i]; }
    else { ik[i - l] = A.key[i]; iv[i - l] = A.val[i]; }
}

// where the refined and coarsened leaves and internal nodes are emitted, two
// runs each in key order, before their merge into a node set
struct Emit {
    uint64_t *key;
    uint8_t *leaf;
    double4 *val;
};
static int emit_buffers(fdm_handle *h, int64_t n, Emit &E) {
    FDM_CK(h, h->amr[11].ensure(n * 8 + 16));
    FDM_CK(h, h->amr[12].ensure(n + 16));
    FDM_CK(h, h->amr[13].ensure(n * 32 + 32));
    E.key = h->amr[11].as<uint64_t>();
    E.leaf = h->amr[12].as<uint8_t>();
    E.val = h->amr[13].as<double4>();
    return FDM_OK;
}

#define AMR_RC(x)            \
    do {                     \
        int rc_ = (x);       \
        if (rc_) return rc_; \
    } while (0)

// Node sets up to this size take gridmodify1 on one cluster.  The gridmodify
// rounds of a regrid, ms, so and with a launch per sweep: 4k nodes 0.253
// (0.298), 21k 0.298 (0.309), 28k 0.280 (0.298), 31k 0.262 (0.278), 36k 0.296
// (0.292), 40k 0.294 (0.283), 53k 0.356 (0.337), 63k 0.354 (0.320): beyond,
// sixteen SMs are slower than all of them.
constexpr int64_t GM1_CLUSTER_MAX = 32768;
// One gridmodify1 pass over the node set A -> A; *did: a node was refined
// or coarsened (otherwise A is left as it is).
static int gridmodify1_pass(fdm_handle *h, AmrCtx &X, bool *did) {
    Nvtx range("fdm regrid: gridmodify1");
    const int TB = 256;
    const int64_t n = X.A.n;
    // Sweeps are queued GM1_SWEEPS at a time (2 to 6 settle a pass); the
    // counts that follow are taken as settled, and taken again when the
    // changes of the last sweep say otherwise.
    constexpr int GM1_SWEEPS = 6;
    Carve cv;
    cv.add(n * 4); cv.add(n * 16); cv.add(n * 16); cv.add(n * 8); cv.add(n); cv.add(n);
    cv.add(n); cv.add((GM1_SWEEPS + 3) * 4); cv.add(n * 4); cv.add(n * 4);
    FDM_CK(h, h->amr[14].ensure(cv.total));
    DevBuf &b = h->amr[14];
    Links L;
    L.parent = cv.at<int32_t>(b, 0); L.child = cv.at<int32_t>(b, 1); L.nb = cv.at<int32_t>(b, 2);
    L.rank = cv.at<uint64_t>(b, 3); L.leaf0 = cv.at<uint8_t>(b, 4); L.cross = cv.at<int8_t>(b, 5);
    int8_t *d = cv.at<int8_t>(b, 6);        // the decisions
    int32_t *changed = cv.at<int32_t>(b, 7), *ddid = changed + GM1_SWEEPS;
    int32_t *cnt = cv.at<int32_t>(b, 8), *off = cv.at<int32_t>(b, 9);
    const int32_t *r = h->pin, *rdid = nullptr;   // changed words, then did words
    int64_t total = 0;
    if (n <= GM1_CLUSTER_MAX) {
        FDM_CK(h, launch_cluster(h->s, k_gm1_pass, X.A, h->G, L, d, cnt, changed));
        AMR_RC(scan_total32(h, cnt, off, n, total, -1, nullptr, changed, GM1_W));   // waits
        if (r[GM1_NSWEEPS] < 0) { h->err = "gridmodify1 decisions did not settle"; return FDM_ERR_UNSUPPORTED; }
        h->gm1_iters += r[GM1_NSWEEPS];
        rdid = r + GM1_DID;
    } else {
        k_gm1_links<<<nblk(n, TB), TB, 0, h->s>>>(X.A, h->G, L, d);
        for (int64_t it = 0;; it += GM1_SWEEPS) {
            if (it > n + 2 + GM1_SWEEPS) { h->err = "gridmodify1 decisions did not settle"; return FDM_ERR_UNSUPPORTED; }
            FDM_CK(h, cudaMemsetAsync(changed, 0, (GM1_SWEEPS + 3) * 4, h->s));
            for (int k = 0; k < GM1_SWEEPS; ++k)
                k_gm1_decide<<<nblk(n, TB), TB, 0, h->s>>>(n, L, d, changed, k);
            k_gm1_count<<<nblk(n, TB), TB, 0, h->s>>>(X.A, L, d, cnt, ddid);
            AMR_RC(scan_total32(h, cnt, off, n, total, -1, nullptr, changed, GM1_SWEEPS + 3));   // waits
            for (int k = 0; k < GM1_SWEEPS; ++k) h->gm1_iters += k == 0 || r[k - 1] != 0;
            if (r[GM1_SWEEPS - 1] == 0) break;
        }
        rdid = r + GM1_SWEEPS;
    }
    *did = rdid[0] != 0;
    if (!*did) return FDM_OK;   // every decision is "nothing": A stays
    const int chain = rdid[1];
    if (chain > 1)              // sons first
        for (int l = rdid[2]; l >= 0; --l)
            k_gm1_vals<<<nblk(n, TB), TB, 0, h->s>>>(X.A, L, d, l);
    // the emit keeps key order: a refined leaf's sons follow it directly and
    // lie before every later node (they fill the leaf's own span)
    AMR_RC(grow_next(h, X, total));
    k_gm1_emit<<<nblk(n, TB), TB, 0, h->s>>>(X.A, L, d, off, X.B, chain <= 1);
    swap_sets(X);
    return FDM_OK;
}

// One gridmodify4 pass over the node set A -> A; *did: something was
// refined (otherwise A is left as it is).
static int gridmodify4_pass(fdm_handle *h, AmrCtx &X, bool *did) {
    Nvtx range("fdm regrid: gridmodify4");
    const int TB = 256;
    *did = false;
    for (cudaEvent_t &e : h->gm4_ev)
        if (!e) FDM_CK(h, cudaEventCreate(&e));
    uint64_t t0 = 0;   // everything up to this time is in A already
    int64_t pool = 0;
    bool grown = false;
    for (;;) {
        const int64_t n = X.A.n;
        pool = std::max(pool, h->gm4_first_pool > 0 ? h->gm4_first_pool : n + 4096);   // as many new nodes as the set has
        const int64_t cap = (pool + 3) / 4 * 4;
        Carve c;
        c.add((n + cap) * 8); c.add((n + cap) * 8); c.add((n + cap) * 4); c.add(2 * 8);   // set to all ones
        c.add(cap * 8); c.add(cap * 4); c.add((n + cap) * 4); c.add(n * 4);
        c.add(GW_WORDS * 4); c.add(sizeof(Gm4Result)); c.add(n * 4); c.add(n * 4);
        DevBuf &b = h->amr[15];
        if (const cudaError_t e = b.ensure(c.total); e != cudaSuccess) {
            if (!grown || e != cudaErrorMemoryAllocation) return cuda_fail(h, e, "gridmodify4 nodes");
            cudaGetLastError();   // the set is as it was: a refusal, not a loss
            h->err = "gridmodify4 cascade exceeded its node pool, and memory has no room for a larger one";
            return FDM_ERR_UNSUPPORTED;
        }
        Gm4 M;
        M.t = c.at<uint64_t>(b, 0); M.tn = c.at<uint64_t>(b, 1); M.son = c.at<int32_t>(b, 2);
        M.nl = c.at<uint64_t>(b, 3); M.mkey = c.at<uint64_t>(b, 4); M.mfather = c.at<int32_t>(b, 5);
        M.refd = c.at<int32_t>(b, 6);
        int32_t *list = c.at<int32_t>(b, 7);
        M.list = list;
        M.w = c.at<int32_t>(b, 8);
        Gm4Result *res = c.at<Gm4Result>(b, 9);
        int32_t *cnt = c.at<int32_t>(b, 10), *off = c.at<int32_t>(b, 11);
        M.cap = cap;
        FDM_CK(h, cudaMemsetAsync(M.t, 0xff, c.off[4], h->s));
        FDM_CK(h, cudaMemsetAsync(M.w, 0, GW_WORDS * 4, h->s));
        k_gm4_triggers<<<nblk(4 * n, TB), TB, 0, h->s>>>(X.A, h->G, t0, list, M.w + GW_NLIST);
        FDM_CK(h, cudaEventRecord(h->gm4_ev[0], h->s));
        FDM_CK(h, launch_cluster(h->s, k_gm4_fixpoint, X.A, h->G, M, t0, 1 << 16, res));
        FDM_CK(h, cudaEventRecord(h->gm4_ev[1], h->s));
        k_gm4_count<<<nblk(n, TB), TB, 0, h->s>>>(X.A, M, res, cnt);
        Gm4Result &hr = *reinterpret_cast<Gm4Result *>(h->pin);
        static_assert(sizeof(Gm4Result) <= fdm_handle::PIN_WORDS * 4, "the result must fit the pinned words");
        int64_t total = 0;
        AMR_RC(scan_total32(h, cnt, off, n, total, -1, nullptr, reinterpret_cast<const int32_t *>(res),
                            sizeof hr / 4));   // waits
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, h->gm4_ev[0], h->gm4_ev[1]) == cudaSuccess) h->gm4_ms += ms;
        if (hr.w[GW_FULL]) {
            // A is untouched: the pass again with twice the room.  A node that
            // one sweep refines and a later one does not keeps its sons, so a
            // rough set can need more room than it ends with.
            if (n + 2 * cap >= (1ll << 31) - 1) {
                h->err = "gridmodify4 cascade exceeded its node pool";
                return FDM_ERR_UNSUPPORTED;
            }
            pool = 2 * cap;
            grown = true;
            continue;
        }
        if (hr.w[GW_STUCK]) { h->err = "gridmodify4 times did not settle"; return FDM_ERR_UNSUPPORTED; }
        h->gm4_visits += hr.w[GW_VISITS];
        h->gm4_nonleaf += hr.w[GW_NONLEAF];
        h->gm4_refines += hr.w[GW_REFINES] + hr.w[GW_NONLEAF];
        h->gm4_steps += hr.w[GW_SWEEPS];
        if (t0 == 0) h->gm4_triggers += hr.w[GW_NLIST];
        if (hr.w[GW_REFINES] == 0 && !hr.w[GW_NONLEAF]) return FDM_OK;
        *did = true;
        AMR_RC(grow_next(h, X, total));
        k_gm4_emit<<<nblk(n, TB), TB, 0, h->s>>>(X.A, M, res, off, X.B);
        swap_sets(X);
        if (!hr.w[GW_NONLEAF]) return FDM_OK;
        t0 = hr.nl_time;
    }
}

// AMR (src/solution.F90:408-421) after the trigger test: indicators,
// refine/coarsen, lvlAMR rounds of gridmodify1 + gridmodify4, new tables.
static int run_amr_impl(fdm_handle *h, fdm_handle *lead);

// A regrid that fails part way (an allocation, a CUDA call) leaves the node
// set and the tables out of step: the handle then counts as not loaded, so
// every stage call returns FDM_ERR_STATE until the next upload.  With a
// leader (lead != nullptr), the refine/coarsen decisions come from the
// leader's indicators on the leader's state; both must hold the same leaf
// set, which is checked on the device.
int run_amr(fdm_handle *h, fdm_handle *lead) {
    const int rc = run_amr_impl(h, lead);
    if (rc && rc != FDM_ERR_UNSUPPORTED && rc != FDM_ERR_ARG) h->loaded = false;
    return rc;
}

__global__ void k_keys_differ(int64_t n, const uint64_t *__restrict__ a, const uint64_t *__restrict__ b,
                              int32_t *flag) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n && a[i] != b[i]) *flag = 1;
}

// the same leaf set (keys in the same order) in both handles
static int same_leaves(fdm_handle *h, fdm_handle *lead, bool *same) {
    *same = false;
    if (h->NL != lead->NL || h->NI != lead->NI || h->NInt != lead->NInt) return FDM_OK;
    FDM_CK(h, cudaStreamSynchronize(lead->s));
    int32_t *flag = h->flag.as<int32_t>() + 7;
    FDM_CK(h, cudaMemsetAsync(flag, 0, 4, h->s));
    k_keys_differ<<<nblk(h->NL, 256), 256, 0, h->s>>>(h->NL, h->lkey.as<uint64_t>(), lead->lkey.as<uint64_t>(), flag);
    int32_t f = 1;
    FDM_CK(h, cudaMemcpyAsync(&f, flag, 4, cudaMemcpyDeviceToHost, h->s));
    FDM_CK(h, cudaStreamSynchronize(h->s));
    *same = f == 0;
    return FDM_OK;
}

static int run_amr_impl(fdm_handle *h, fdm_handle *lead) {
    Nvtx range("fdm regrid");
    const int TB = 256;
    const int64_t NL = h->NL, NI = h->NI, NInt = h->NInt;
    if (h->p.window_rows != 0) {
        h->err = "a strip of a mesh takes no regrid: regrid the whole mesh";
        return FDM_ERR_UNSUPPORTED;
    }
    if ((int64_t)h->p.m * h->p.n >= (1ll << 19)) {
        h->err = "device regrid supports up to 2^19 background cells";
        return FDM_ERR_UNSUPPORTED;
    }
    for (int k = 0; k <= fdm_handle::AMR_PHASES; ++k)
        if (!h->amr_ev[k]) FDM_CK(h, cudaEventCreate(&h->amr_ev[k]));
    FDM_CK(h, cudaEventRecord(h->amr_ev[0], h->s));
    // 1. indicators and their ordered sums
    Carve ci;
    ci.add(NI * 8); ci.add(NI * 8); ci.add(32); ci.add(NL); ci.add((NInt > 0 ? NInt : 1));
    FDM_CK(h, h->amr[18].ensure(ci.total));
    double *rot = ci.at<double>(h->amr[18], 0), *div = ci.at<double>(h->amr[18], 1), *sums = ci.at<double>(h->amr[18], 2);
    int8_t *rflag = ci.at<int8_t>(h->amr[18], 3), *cflag = ci.at<int8_t>(h->amr[18], 4);
    if (lead) {
        bool same = false;
        AMR_RC(same_leaves(h, lead, &same));
        if (!same) {
            h->err = "the leader's leaf set differs from this handle's";
            return FDM_ERR_ARG;
        }
        const int rc = compute_rot_div(lead, rot, div, sums);
        if (rc) { h->err = "leader's indicators: " + lead->err; return rc; }
        FDM_CK(h, cudaStreamSynchronize(lead->s));
    } else {
        AMR_RC(compute_rot_div(h, rot, div, sums));
    }
    FDM_CK(h, cudaEventRecord(h->amr_ev[1], h->s));
    // 2. solute_ref: refine and coarsen flags, applied at once
    const Tables T = h->tables();
    k_refine_flags<<<nblk(NL, TB), TB, 0, h->s>>>(T, h->G, h->p, rot, div, sums, rflag);
    if (NInt > 0)
        k_coarsen_flags<<<nblk(NInt, TB), TB, 0, h->s>>>(NInt, h->ikey.as<uint64_t>(), T, h->p, rot, div, sums, rflag,
                                                        cflag);
    const int64_t nn = NL + NInt;
    FDM_CK(h, h->amr[19].ensure(nn * 8 + 16));
    int32_t *cnt = h->amr[19].as<int32_t>(), *off = cnt + nn;
    k_ref_count<<<nblk(nn, TB), TB, 0, h->s>>>(T, rflag, h->ikey.as<uint64_t>(), NInt, cflag, cnt);
    int64_t total = 0, split = 0;   // the leaves' entries (sorted) come first, then the internal nodes' (sorted)
    AMR_RC(scan_total32(h, cnt, off, nn, total, NL, &split));
    Emit E;
    AMR_RC(emit_buffers(h, total, E));
    k_ref_emit<<<nblk(nn, TB), TB, 0, h->s>>>(T, h->B[0].as<double4>(), rflag, h->ikey.as<uint64_t>(),
                                              h->ival.as<double4>(), NInt, cflag, off, E.key, E.leaf, E.val);
    AmrCtx X;
    X.h = h;
    AMR_RC(grow_next(h, X, total));
    merge_into(h, E.key, E.leaf, E.val, split, total, X.B);
    swap_sets(X);
    FDM_CK(h, cudaEventRecord(h->amr_ev[2], h->s));
    // 3. solute_gridmodify: lvlAMR rounds (src/solution.F90:537-556)
    // A round that changes nothing leaves the node set as it found it, so
    // the rounds after it would change nothing either.
    for (int k = 1; k <= h->p.lvl_amr; ++k) {
        bool did1 = false, did4 = false;
        AMR_RC(gridmodify1_pass(h, X, &did1));
        AMR_RC(gridmodify4_pass(h, X, &did4));
        if (!did1 && !did4) break;
    }
    FDM_CK(h, cudaEventRecord(h->amr_ev[3], h->s));
    // 4. split leaves / internal nodes, rebuild the tables (idneighbor + IDgrid)
    const int64_t n = X.A.n;
    Carve cs;
    cs.add(n * 4); cs.add(n * 4);
    FDM_CK(h, h->amr[8].ensure(cs.total));
    int32_t *fl = cs.at<int32_t>(h->amr[8], 0), *ol = cs.at<int32_t>(h->amr[8], 1);
    k_split_count<<<nblk(n, TB), TB, 0, h->s>>>(n, X.A.leaf, fl);
    int64_t nleaf = 0;
    AMR_RC(scan_total32(h, fl, ol, n, nleaf));
    const int64_t nint = n - nleaf;   // every node is one or the other
    DevBuf &lv = h->amr[21];   // kept between regrids
    FDM_CK(h, h->lkey.ensure(nleaf * 8));   // the new leaves' keys, where the tables have them
    FDM_CK(h, lv.ensure(nleaf * 32 + 32));
    FDM_CK(h, h->ikey.ensure(nint * 8 + 8));
    FDM_CK(h, h->ival.ensure(nint * 32 + 32));
    k_split_emit<<<nblk(n, TB), TB, 0, h->s>>>(X.A, ol, h->lkey.as<uint64_t>(), lv.as<double4>(),
                                               h->ikey.as<uint64_t>(), h->ival.as<double4>());
    FDM_CK(h, cudaEventRecord(h->amr_ev[4], h->s));
    h->NInt = nint;   // the rebuild is ordered after the split on the stream
    const int rc = build_tables(h, nleaf, h->lkey.as<uint64_t>(), lv.as<double>(), 0);   // split keeps key order
    if (rc) return rc;
    FDM_CK(h, cudaEventRecord(h->amr_ev[5], h->s));
    FDM_CK(h, cudaEventSynchronize(h->amr_ev[5]));
    for (int k = 0; k < fdm_handle::AMR_PHASES; ++k) {
        float t = 0.f;
        cudaEventElapsedTime(&t, h->amr_ev[k], h->amr_ev[k + 1]);
        h->amr_phase_ms[k] = t;
        h->amr_phase_total_ms[k] += t;
    }
    h->n_regrids++;
    return FDM_OK;
}

}  // namespace fdm

// Device-timeline milliseconds of the regrid phases: indicators and
// ordered sums, refine/coarsen flags and the first node sort, the lvlAMR
// gridmodify rounds, the leaf/internal split, the table rebuild; ms[0..4]
// for the last regrid, ms[5..9] summed over all regrids of the handle.
extern "C" int fdm_amr_phase_ms(const fdm_handle *h, double *ms) {
    if (!h || !ms) return FDM_ERR_ARG;
    for (int k = 0; k < fdm_handle::AMR_PHASES; ++k) {
        ms[k] = h->amr_phase_ms[k];
        ms[fdm_handle::AMR_PHASES + k] = h->amr_phase_total_ms[k];
    }
    return FDM_OK;
}

extern "C" int fdm_debug_rot_div(fdm_handle *h, int64_t cap, double *rot, double *div, double *sums) {
    using namespace fdm;
    if (!h) return FDM_ERR_ARG;
    if (!h->loaded) return FDM_ERR_STATE;
    if (cap < h->NI) return arg_fail(h, "capacity below the interior leaf count");
    DevBuf d;
    Carve cv;
    cv.add(h->NI * 8); cv.add(h->NI * 8); cv.add(3 * 8);
    FDM_CK(h, d.ensure(cv.total));
    double *dr = cv.at<double>(d, 0), *dd = cv.at<double>(d, 1), *ds = cv.at<double>(d, 2);
    int rc = compute_rot_div(h, dr, dd, ds);
    if (rc) return rc;
    if (rot) FDM_CK(h, cudaMemcpyAsync(rot, dr, h->NI * 8, cudaMemcpyDeviceToHost, h->s));
    if (div) FDM_CK(h, cudaMemcpyAsync(div, dd, h->NI * 8, cudaMemcpyDeviceToHost, h->s));
    if (sums) FDM_CK(h, cudaMemcpyAsync(sums, ds, 24, cudaMemcpyDeviceToHost, h->s));
    FDM_CK(h, cudaStreamSynchronize(h->s));
    d.release();
    return FDM_OK;
}

namespace fdm {
__global__ void k_interleave2(int64_t n, const double *__restrict__ a, const double *__restrict__ b, double2 *out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = make_double2(a[i], b[i]);
}
}  // namespace fdm

extern "C" int fdm_debug_ordered_sum(const double *a, const double *b, int64_t n, double *sums) {
    using namespace fdm;
    if (!a || !b || !sums || n < 0 || n >= (1ll << 31)) return FDM_ERR_ARG;
    double *da = nullptr, *db = nullptr, *dout = nullptr;
    double2 *dq = nullptr;
    const size_t bytes = (size_t)(n > 0 ? n : 1) * 8;
    cudaError_t e = cudaMalloc(&da, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&db, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&dq, 2 * bytes);
    if (e == cudaSuccess) e = cudaMalloc(&dout, 32);
    if (e == cudaSuccess && n > 0) e = cudaMemcpy(da, a, n * 8, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && n > 0) e = cudaMemcpy(db, b, n * 8, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        if (n > 0) k_interleave2<<<nblk(n, 256), 256>>>(n, da, db, dq);
        k_ordered_sums<<<2, OSUM_NT>>>(n, dq, dout);
        e = cudaGetLastError();
    }
    double out[3] = {0.0, 0.0, 0.0};
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, 24, cudaMemcpyDeviceToHost);
    cudaFree(da); cudaFree(db); cudaFree(dq); cudaFree(dout);
    if (e != cudaSuccess) return FDM_ERR_CUDA;
    sums[0] = out[0];
    sums[1] = out[1];
    return FDM_OK;
}
