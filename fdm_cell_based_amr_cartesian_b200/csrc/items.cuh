// items.cuh — the per-item work of one SSP-RK3 stage, shared by the
// single-mesh kernels (stage.cu, gate.cu) and the batched persistent kernel
// (batch.cu), so both paths run the same arithmetic:
//
//   request_item / request_restrict_warp   hanging-node values
//                                          (src/XuanGua.F90:45-398)
//   face_item                              WCNS flux of one face
//                                          (src/nnd_center_RK.F90:66-353)
//   cell_item + cells_block_reduce         residual, forward-Euler candidate,
//                                          RK3 blend, residual norms, lambda
//                                          (src/nnd_center_RK.F90:15-64,
//                                           src/solution.F90:279-286,386-404)
//   ghost_warp                             boundary images
//                                          (src/solution.F90:288-293,109-168)
//   step_control_item / step_end_item /    solute bookkeeping
//   res_finalize_block                     (src/solution.F90:185-215)
#pragma once

#include "handle.cuh"
#include "numerics.cuh"
#include "numerics_nr.cuh"

namespace fdm {

// interpA over a subtree whose leaves are [lo, hi) of the sorted array
// (src/XuanGua.F90:359-398): children combined as
// 0.25*(son1 + son2 + son3 + son4) = 0.25*(((q0 + q1) + q3) + q2).
// One warp: the lanes stage the subtree's leaves in shared memory.  A
// subtree of up to RW_CAP leaves is folded level by level by all lanes; a
// larger one is folded by lane 0 in key order with a stack of pending
// sibling groups.  Every father is formed from the same four values in the
// same order either way.
constexpr int RW_CAP = 256;     // leaves staged per pass
constexpr int RW_STACK = 48;    // >= 3 pending siblings x 15 levels + 1
struct RestrictSmem {
    double4 v[RW_CAP];
    int8_t l[RW_CAP];
    union {
        struct {
            double4 st[RW_STACK];
            int8_t sl[RW_STACK];
        } s;                   // the stack of the lane-0 fold
        uint32_t p[RW_CAP];    // path bits of the staged entries (level fold)
    } u;
};

// the fold of n <= RW_CAP leaves from lo: at the deepest level present,
// every group of four siblings (consecutive in key order, the first with
// digit 0) becomes its father; the list is compacted and the next level up
// follows
__device__ __forceinline__ double4 restrict_warp_levels(const Tables &T, const double4 *__restrict__ buf,
                                                        int64_t lo, int n, RestrictSmem &sm) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int lmax = 0;
    for (int k = lane; k < n; k += 32) {
        const uint64_t key = __ldg(T.lkey + lo + k);
        sm.v[k] = buf[__ldg(T.lslot + lo + k)];
        sm.l[k] = (int8_t)(key & 15u);
        sm.u.p[k] = (uint32_t)((key >> 4) & ((1ull << 30) - 1ull));
        lmax = max(lmax, (int)(key & 15u));
    }
    lmax = __reduce_max_sync(FULL, lmax);
    __syncwarp();
    while (n > 1 && lmax > 0) {
        const int sh = 2 * (LMAX - lmax);
        int off = 0;
        for (int base = 0; base < n; base += 32) {
            const int i = base + lane;
            double4 vi = make_double4(0.0, 0.0, 0.0, 0.0);
            int8_t li = 0;
            uint32_t pi = 0;
            bool keep = false;
            if (i < n) {
                vi = sm.v[i];
                li = sm.l[i];
                pi = sm.u.p[i];
                const bool deep = li == lmax;
                const bool first = deep && ((pi >> sh) & 3u) == 0u && i + 3 < n;
                keep = !deep || first;
                if (first) {   // the father (its path: the first son's, digit 0)
                    const double4 e0 = vi, e1 = sm.v[i + 1], e2 = sm.v[i + 2], e3 = sm.v[i + 3];
                    vi.x = 0.25 * (e0.x + e1.x + e3.x + e2.x);
                    vi.y = 0.25 * (e0.y + e1.y + e3.y + e2.y);
                    vi.z = 0.25 * (e0.z + e1.z + e3.z + e2.z);
                    vi.w = 0.25 * (e0.w + e1.w + e3.w + e2.w);
                    li = (int8_t)(lmax - 1);
                }
            }
            const unsigned km = __ballot_sync(FULL, keep);
            const int pos = off + __popc(km & ((1u << lane) - 1u));
            off += __popc(km);
            __syncwarp();
            if (keep) {   // positions only move down, below what later chunks read
                sm.v[pos] = vi;
                sm.l[pos] = li;
                sm.u.p[pos] = pi;
            }
            __syncwarp();
        }
        n = off;
        --lmax;
    }
    const double4 r = sm.v[0];
    __syncwarp();
    return r;
}

__device__ __forceinline__ double4 restrict_warp(const Tables &T, const double4 *__restrict__ buf, int64_t lo,
                                                 int64_t hi, RestrictSmem &sm) {
    if (hi - lo <= RW_CAP) return restrict_warp_levels(T, buf, lo, (int)(hi - lo), sm);
    const int lane = threadIdx.x & 31;
    int top = 0;
    for (int64_t base = lo; base < hi; base += RW_CAP) {
        const int n = (int)min((int64_t)RW_CAP, hi - base);
        for (int k = lane; k < n; k += 32) {
            sm.v[k] = buf[__ldg(T.lslot + base + k)];
            sm.l[k] = (int8_t)(__ldg(T.lkey + base + k) & 15u);
        }
        __syncwarp();
        if (lane == 0) {
            for (int k = 0; k < n; ++k) {
                if (top >= RW_STACK) break;  // cannot happen for a valid subtree
                sm.u.s.st[top] = sm.v[k];
                sm.u.s.sl[top] = sm.l[k];
                ++top;
                while (top >= 4 && sm.u.s.sl[top - 1] == sm.u.s.sl[top - 2] && sm.u.s.sl[top - 1] == sm.u.s.sl[top - 3] &&
                       sm.u.s.sl[top - 1] == sm.u.s.sl[top - 4]) {
                    const double4 e0 = sm.u.s.st[top - 4], e1 = sm.u.s.st[top - 3], e2 = sm.u.s.st[top - 2], e3 = sm.u.s.st[top - 1];
                    double4 v;
                    v.x = 0.25 * (e0.x + e1.x + e3.x + e2.x);
                    v.y = 0.25 * (e0.y + e1.y + e3.y + e2.y);
                    v.z = 0.25 * (e0.z + e1.z + e3.z + e2.z);
                    v.w = 0.25 * (e0.w + e1.w + e3.w + e2.w);
                    const int8_t l = (int8_t)(sm.u.s.sl[top - 1] - 1);
                    top -= 4;
                    sm.u.s.st[top] = v;
                    sm.u.s.sl[top] = l;
                    ++top;
                }
            }
        }
        __syncwarp();
    }
    double4 r = sm.u.s.st[0];
    __syncwarp();
    return r;
}

// components v..v+NV-1 of hanging-node request r of kind WLS or COPY (v a
// multiple of NV): the four components of a value are independent, so 4 / NV
// threads share a request.  geo: element 0 of the request's geometry block
// (global memory, or a copy of its tile in shared memory).
template <int NV>
__device__ __forceinline__ void load_components(const double *rec, double (&c)[NV]) {
    if constexpr (NV == 2) {
        const double2 q = *reinterpret_cast<const double2 *>(rec);
        c[0] = q.x; c[1] = q.y;
    } else {
        c[0] = *rec;
    }
}
template <int NV>
__device__ __forceinline__ void request_item(const Tables &T, double4 *cur, int64_t r, int v, const double *geo) {
    static_assert(NV == 1 || NV == 2, "components per thread");
    const int kind = T.rq_kind[r];
    if (kind == RQ_RESTRICT) return;
    const int32_t *mem = T.rq_mem + rq_mem_at(r);
    double out[NV];
    if (kind == RQ_COPY) {
        load_components<NV>(reinterpret_cast<const double *>(cur + mem[0]) + v, out);
    } else {
        int32_t slot[WLS_MAXM];
#pragma unroll
        for (int i = 0; i < WLS_MAXM; ++i) slot[i] = mem[i * RQ_T];
        double phi[NV][WLS_MAXM];
#pragma unroll
        for (int i = 0; i < WLS_MAXM; ++i) {
            double c[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) c[q] = 0.0;
            if (slot[i] >= 0) load_components<NV>(reinterpret_cast<const double *>(cur + slot[i]) + v, c);
#pragma unroll
            for (int q = 0; q < NV; ++q) phi[q][i] = c[q];
        }
        wls_eval<NV>(geo, phi, out);
    }
    double *o = reinterpret_cast<double *>(cur + T.NI + T.NG + T.NC + r) + v;
    if constexpr (NV == 2) *reinterpret_cast<double2 *>(o) = make_double2(out[0], out[1]);
    else *o = out[0];
}

// The geometry blocks of the RQ_TILE requests from r0 on (contiguous in
// rq_geo) into shared memory, 16 bytes per cp.async; all BT threads of the
// block call it, and it returns after the copy has landed and the block has
// synchronised.
constexpr int RQ_TILE = 64;
__device__ __forceinline__ void stage_request_geometry(const Tables &T, int64_t r0, double *smem_geo, int nthreads) {
    int64_t nreq = T.NR - r0;
    if (nreq > RQ_TILE) nreq = RQ_TILE;
    nreq = (nreq + RQ_T - 1) / RQ_T * RQ_T;   // whole tiles
    const int nch = nreq > 0 ? (int)(nreq * RQ_GEO / 2) : 0;   // 16-byte chunks
    const double *src = T.rq_geo + r0 * RQ_GEO;
    for (int k = threadIdx.x; k < nch; k += nthreads) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(smem_geo + 2 * k);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src + 2 * k) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
}

// interpA fallback of parent_value_weno for request r (whole warp)
__device__ __forceinline__ void request_restrict_warp(const Tables &T, double4 *cur, int64_t r, RestrictSmem &sm) {
    if (T.rq_kind[r] != RQ_RESTRICT) return;
    const double4 v = restrict_warp(T, cur, T.rq_m[2 * r], T.rq_m[2 * r + 1], sm);
    if ((threadIdx.x & 31) == 0) cur[T.NI + T.NG + T.NC + r] = v;
}

// The four stencil slots of face f.  Faces [0, NI) are the right (top) faces
// of the interior leaves; faces [NI, NI+nu) are left (bottom) faces that are
// not shared with a same-level neighbour.
template <int DIR>
__device__ __forceinline__ void face_slots(const Tables &T, int64_t f, int32_t &a, int32_t &b, int32_t &c,
                                           int32_t &d) {
    if (f < T.NI) {
        const int32_t *s = T.ist + f * 8;
        if (DIR == 0) { a = s[1]; b = (int32_t)f; c = s[0]; d = s[4]; }
        else { a = s[3]; b = (int32_t)f; c = s[2]; d = s[6]; }
    } else {
        const int32_t i = DIR == 0 ? T.uxl[f - T.NI] : T.uyl[f - T.NI];
        const int32_t *s = T.ist + (int64_t)i * 8;
        if (DIR == 0) { a = s[5]; b = s[1]; c = i; d = s[0]; }
        else { a = s[7]; b = s[3]; c = i; d = s[2]; }
    }
}

template <int DIR>
__device__ __forceinline__ void face_item(const Tables &T, const double4 *__restrict__ cur, double4 *F, double lam,
                                          double g, const FluxDen &den, int64_t f) {
    int32_t a, b, c, d;
    face_slots<DIR>(T, f, a, b, c, d);
    store_record(F + f, face_flux_of<DIR>(cur, a, b, c, d, g, den, lam));
}

// the same by two neighbouring lanes, face f of n (lanes past the last face
// compute it again and store nothing)
template <int DIR>
__device__ __forceinline__ void face_item_pair(const Tables &T, const double4 *__restrict__ cur, double4 *F, double lam,
                                               double g, const FluxDen &den, int64_t f, int64_t n) {
    int32_t a, b, c, d;
    face_slots<DIR>(T, f < n ? f : n - 1, a, b, c, d);
    const double2 v = face_flux_pair<DIR>(cur, a, b, c, d, g, den, lam);
    if (f < n) reinterpret_cast<double2 *>(F + f)[threadIdx.x & 1] = v;
}

// Residual + forward-Euler candidate (LXL) fused with updateRK for leaf i.
// mode 0: the blended stage value; mode 1: the primitive candidate Ut (no
// blend) for the split API.  rm / rs / lx / ly are the leaf's residual norms
// and (stage 3) wave speeds.  Divisions through D: the branch-free ones
// (DivNR, ok false when an operand is outside their range) or the compiler's.
struct CellValue {
    double4 o;
    double rm[4], rs[4], lx, ly;
    bool ok;
};
// the value from the records: q the cell, qp/qm/rp/rm_ its x and y neighbours,
// fr/fl/hr/hl its face fluxes; k the level's coefficients
struct CellCoef {
    double cxa, cxb, cya, cyb, dx, dy;
};
template <class D>
__device__ __forceinline__ CellValue cell_update(const Prim &q, const Prim &qp, const Prim &qm, const Prim &rp,
                                                 const Prim &rmn, const double4 &fr, const double4 &fl,
                                                 const double4 &hr, const double4 &hl, const CellCoef &k,
                                                 const double4 *un, double tstep, int krk, int mode, double g,
                                                 const FluxDen &den) {
    D dv(den);
    dv.test_numerator(q.p);
    dv.test_numerator(qp.p);
    dv.test_numerator(qm.p);
    dv.test_numerator(rp.p);
    dv.test_numerator(rmn.p);
    double Ep[4], Em[4], Gp[4], Gm[4];
    phys_flux_nr<0>(qp, dv, Ep);
    phys_flux_nr<0>(qm, dv, Em);
    phys_flux_nr<1>(rp, dv, Gp);
    phys_flux_nr<1>(rmn, dv, Gm);
    const double FR[4] = {fr.x, fr.y, fr.z, fr.w}, FL[4] = {fl.x, fl.y, fl.z, fl.w};
    const double HR[4] = {hr.x, hr.y, hr.z, hr.w}, HL[4] = {hl.x, hl.y, hl.z, hl.w};
    double U[4];
    U[0] = q.r;
    U[1] = q.r * q.u;
    U[2] = q.r * q.v;
    U[3] = D::q(q.p, dv.gm1) + 0.5 * q.r * (q.u * q.u + q.v * q.v);
    CellValue c;
    double Ut[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        const double dE = k.cxa * (FR[n] - FL[n]) - k.cxb * (Ep[n] - Em[n]);
        const double dF = k.cya * (HR[n] - HL[n]) - k.cyb * (Gp[n] - Gm[n]);
        const double fu = -dE - dF;
        Ut[n] = U[n] + fu * tstep;
        const double f = fu * k.dx * k.dy;
        c.rm[n] = fabs(f);
        c.rs[n] = f * f;
    }
    const double r0 = Ut[0];
    dv.test_bits(r0);
    dv.template test_range<-100, 100>(r0);
    dv.test_numerator(Ut[1]);
    dv.test_numerator(Ut[2]);
    dv.test_numerator(Ut[3]);
    const Den dr = D::den(r0);
    const double u0 = D::q(Ut[1], dr);
    const double v0 = D::q(Ut[2], dr);
    const double p0 = (g - 1.0) * r0 * (D::q(Ut[3], dr) - 0.5 * (u0 * u0 + v0 * v0));
    c.lx = c.ly = 0.0;
    if (mode == 1) {
        c.o = make_double4(r0, u0, v0, p0);
    } else {
        const double4 n0 = load_record(un);
        const double ra = krk == 1 ? 0.0 : krk == 2 ? 3.0 / 4.0 : 1.0 / 3.0;
        const double rb = krk == 1 ? 1.0 : krk == 2 ? 1.0 / 4.0 : 2.0 / 3.0;
        c.o.x = ra * n0.x + rb * r0;
        c.o.y = ra * n0.y + rb * u0;
        c.o.z = ra * n0.z + rb * v0;
        c.o.w = ra * n0.w + rb * p0;
        if (krk == 3) {
            const double a = sqrt(g * c.o.w / c.o.x);
            c.lx = fabs(c.o.y) + a;
            c.ly = fabs(c.o.z) + a;
        }
    }
    c.ok = dv.ok;
    return c;
}
template <class D>
__device__ __forceinline__ CellValue cell_value(const Tables &T, const LevelTab &LT, const double4 *__restrict__ cur,
                                                const double4 *un, const double4 *__restrict__ Fx,
                                                const double4 *__restrict__ Fy, double tstep, int krk, int mode,
                                                double g, const FluxDen &den, int64_t i) {
    const int lvl = T.ilvl[i];
    const int4 s = *reinterpret_cast<const int4 *>(T.ist + i * 8);
    const CellCoef k{LT.cxa[lvl], LT.cxb[lvl], LT.cya[lvl], LT.cyb[lvl], LT.dx[lvl], LT.dy[lvl]};
    return cell_update<D>(load_prim(cur, i), load_prim(cur, s.x), load_prim(cur, s.y), load_prim(cur, s.z),
                          load_prim(cur, s.w), load_record(Fx + i), load_record(Fx + T.ifxl[i]), load_record(Fy + i),
                          load_record(Fy + T.ifyl[i]), k, un + i, tstep, krk, mode, g, den);
}
// a leaf that DivNR refuses, out of line
__device__ __noinline__ inline CellValue cell_value_again(const Tables &T, const LevelTab &LT, const double4 *cur,
                                                          const double4 *un, const double4 *Fx, const double4 *Fy,
                                                          double tstep, int krk, int mode, double g,
                                                          const FluxDen &den, int64_t i) {
    return cell_value<DivIEEE>(T, LT, cur, un, Fx, Fy, tstep, krk, mode, g, den, i);
}
__device__ __forceinline__ void cell_item(const Tables &T, const LevelTab &LT, const double4 *__restrict__ cur,
                                          const double4 *un, double4 *next, const double4 *__restrict__ Fx,
                                          const double4 *__restrict__ Fy, double tstep, int krk, int mode, double g,
                                          const FluxDen &den, int64_t i, double rm[4], double rs[4], double &lx,
                                          double &ly) {
    CellValue c = cell_value<DivNR>(T, LT, cur, un, Fx, Fy, tstep, krk, mode, g, den, i);
    if (!c.ok) c = cell_value_again(T, LT, cur, un, Fx, Fy, tstep, krk, mode, g, den, i);
#pragma unroll
    for (int n = 0; n < 4; ++n) { rm[n] = c.rm[n]; rs[n] = c.rs[n]; }
    lx = c.lx;
    ly = c.ly;
    store_record(next + i, c.o);
}

// Block reduction of one 256-leaf tile: residual max / sum of squares into
// res_slot[0..7], lambda maxima into the scalars at stage 3.  Called by all
// threads of a 256-thread block; sh / shl are the block's shared scratch.
struct CellsSmem {
    double sh[8][8];
    double shl[8][2];
};
__device__ __forceinline__ void cells_block_reduce(double rm[4], double rs[4], double lx, double ly,
                                                   double *res_slot, DevScalars *sc, bool lam, CellsSmem &S) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        for (int o = 16; o; o >>= 1) {
            rm[n] = fmax(rm[n], __shfl_xor_sync(0xffffffffu, rm[n], o));
            rs[n] += __shfl_xor_sync(0xffffffffu, rs[n], o);
        }
    }
    for (int o = 16; o; o >>= 1) {
        lx = fmax(lx, __shfl_xor_sync(0xffffffffu, lx, o));
        ly = fmax(ly, __shfl_xor_sync(0xffffffffu, ly, o));
    }
    if (lane == 0) {
        for (int n = 0; n < 4; ++n) { S.sh[wid][n] = rm[n]; S.sh[wid][4 + n] = rs[n]; }
        S.shl[wid][0] = lx;
        S.shl[wid][1] = ly;
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        const int n = threadIdx.x;
        double v = S.sh[0][n];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) v = n < 4 ? fmax(v, S.sh[w][n]) : v + S.sh[w][n];
        res_slot[n] = v;
    }
    if (lam && threadIdx.x == 0) {
        double a = S.shl[0][0], b = S.shl[0][1];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) { a = fmax(a, S.shl[w][0]); b = fmax(b, S.shl[w][1]); }
        atomicMax((unsigned long long *)&sc->lam_next_x, (unsigned long long)__double_as_longlong(a));
        atomicMax((unsigned long long *)&sc->lam_next_y, (unsigned long long)__double_as_longlong(b));
    }
    __syncthreads();
}

struct GhostStates {
    double s[6][4];   // bc_state[0..3], dmr_post, dmr_pre
    double x0, cot, speed;
};

// value of a ghost leaf of kind COPY or a boundary state
__device__ __forceinline__ double4 ghost_simple_value(const Tables &T, const double4 *buf, const GhostStates &GS,
                                                      const DevScalars *__restrict__ sc, int j, int64_t gi,
                                                      int kind) {
    if (kind == GH_COPY) return buf[T.gh_a[gi]];
    // boundary time of body_boundary_RK (src/solution.F90:320-326)
    double t = sc->tt;
    if (j == 2) t = sc->tt + sc->tstep;
    else if (j == 3) t = sc->tt + 0.5 * sc->tstep;
    int st = T.gh_a[gi];
    if (kind == GH_DMR_TOP) {
        const double xs = GS.x0 + T.gh_y[gi] * GS.cot + GS.speed * t;
        st = T.gh_x[gi] < xs ? 4 : 5;
    }
    return make_double4(GS.s[st][0], GS.s[st][1], GS.s[st][2], GS.s[st][3]);
}
// mirror (wall) flip and store of a ghost value
__device__ __forceinline__ void ghost_store(const Tables &T, double4 *buf, int64_t gi, double4 v) {
    const int fl = T.gh_flip[gi];
    if (fl == 1) v.y = -v.y;
    else if (fl == 2) v.z = -v.z;
    buf[T.NI + gi] = v;
}

// ghost leaf gi (whole warp: interpA images can span hundreds of leaves)
__device__ __forceinline__ void ghost_warp(const Tables &T, double4 *buf, const GhostStates &GS,
                                           const DevScalars *__restrict__ sc, int j, int64_t gi, RestrictSmem &sm) {
    const int lane = threadIdx.x & 31;
    const int kind = T.gh_kind[gi];
    if (kind == GH_NONE) return;
    double4 v;
    if (kind == GH_RESTRICT) v = restrict_warp(T, buf, T.gh_a[gi], T.gh_b[gi], sm);
    else v = ghost_simple_value(T, buf, GS, sc, j, gi, kind);
    if (lane != 0) return;
    ghost_store(T, buf, gi, v);
}

__host__ inline GhostStates ghost_states(const fdm_params &p) {
    GhostStates GS;
    for (int s = 0; s < 4; ++s)
        for (int k = 0; k < 4; ++k) GS.s[s][k] = p.bc_state[s][k];
    for (int k = 0; k < 4; ++k) { GS.s[4][k] = p.dmr_post[k]; GS.s[5][k] = p.dmr_pre[k]; }
    GS.x0 = p.dmr_x0;
    GS.cot = p.dmr_angle_cot;
    GS.speed = p.dmr_shock_speed;
    return GS;
}

// lambda/time-step control (src/solution.F90:185-201); one thread
__device__ __forceinline__ void step_control_item(DevScalars *sc, const fdm_params &P, int use_dt) {
    if (sc->done) return;   // (the caller resets lam_next for a step that goes on all the same)
    sc->lambda_x = fmax(sc->lambda_x, sc->lam_next_x);
    sc->lambda_y = fmax(sc->lambda_y, sc->lam_next_y);
    sc->lam_next_x = 0.0;
    sc->lam_next_y = 0.0;
    if (use_dt && P.iflag_localdt) {
        const double div = (double)(1ll << sc->l_max);
        sc->tstep = P.cfl / (sc->lambda_x / (P.x_factor * P.h / div) + sc->lambda_y / (P.h / div));
    }
    if (sc->tt + sc->tstep > P.t_end) sc->tstep = P.t_end - sc->tt;
}

// residual partials -> Res_max / Res_rms sums over a fixed reduction tree
// (256 strided sums of each component, then pairwise), so the result is
// identical run to run and for every NT (256 or 1024 threads, the components
// of a strided sum shared by NT / 256 of them); all threads of the block
template <int NT>
__device__ __forceinline__ void res_finalize_block(const double *__restrict__ res_part, int nb, DevScalars *sc,
                                                   double (*sh)[8]) {
    constexpr int NC = 8 * 256 / NT;   // components per thread
    const int t = threadIdx.x & 255, c0 = (threadIdx.x >> 8) * NC;
    double v[NC];
#pragma unroll
    for (int n = 0; n < NC; ++n) v[n] = 0.0;
#pragma unroll 4
    for (int b = t; b < nb; b += 256)
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            const double x = res_part[b * 8 + c0 + n];
            v[n] = c0 + n < 4 ? fmax(v[n], x) : v[n] + x;
        }
#pragma unroll
    for (int n = 0; n < NC; ++n) sh[t][c0 + n] = v[n];
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (t < w)
#pragma unroll
            for (int n = 0; n < NC; ++n)
                sh[t][c0 + n] = c0 + n < 4 ? fmax(sh[t][c0 + n], sh[t + w][c0 + n]) : sh[t][c0 + n] + sh[t + w][c0 + n];
        __syncthreads();
    }
    if (threadIdx.x < 8) {
        const int n = threadIdx.x;
        if (n < 4) sc->res_max[n] = sh[0][n];
        else sc->res_rms[n - 4] = sh[0][n];
    }
    __syncthreads();
}

// end of one solute iteration: tt, rms, NaN stop, t_end
// (src/solution.F90:205-215); one thread
__device__ __forceinline__ void step_end_item(DevScalars *sc, int64_t NI) {
    if (sc->done) return;
    sc->tt = sc->tt + sc->tstep;
    sc->it = sc->it + 1;
    for (int n = 0; n < 4; ++n) {
        sc->res_rms[n] = sqrt(sc->res_rms[n] / (1.0 * (double)NI));
        if (isnan(sc->res_rms[n])) sc->status = FDM_ERR_NAN;
    }
    // the reference stops at t_end and at a NaN residual: later iterations
    // are no-ops
    if (!(sc->tt < sc->t_end) || sc->status == FDM_ERR_NAN) sc->done = 1;
}

}  // namespace fdm
