// stage.cu — one SSP-RK3 stage on the device.
//
//   k_requests  hanging-node values (WLS-WENO / interpA / copy) into the
//               virtual slots                 (src/XuanGua.F90:45-398)
//   k_faces     WCNS flux of every distinct face, x and y
//                                             (src/nnd_center_RK.F90:66-353)
//   k_cells     residual, forward-Euler candidate, RK3 blend, residual
//               norms and the next lambda     (src/nnd_center_RK.F90:15-64,
//                                              src/solution.F90:279-286,386-404)
//   k_ghost     boundary images               (src/solution.F90:288-293,109-168)
//
// State lives in three slot arrays of 32-byte (rho,u,v,p) records: interior
// leaves (key order), ghost leaves, corner leaves, then the virtual slots.
#include <algorithm>

#include "handle.cuh"
#include "items.cuh"
#include "numerics.cuh"

namespace fdm {

static inline int nblk(int64_t n, int t) { return (int)((n + t - 1) / t); }

// 4 / NV threads per request, NV components each; eight neighbouring lanes
// read one tile of the geometry, so a load of an element is 64 contiguous
// bytes for each group of them.  The 712 bytes of geometry per value bound it
// (58 MB for 81k values, from L2 while the mesh stays); the fixed slots let
// the loads run ahead of the sums.  81k values 24 us cold, 57k 13 us (41 and
// 23 with one block of geometry per request, member counts as predicates and
// a thread per component).
constexpr int RQ_NV = 2;
__device__ __forceinline__ void requests_block(const Tables &T, double4 *cur) {
    constexpr int PER = 32 * RQ_NV / 4;   // requests per warp
    const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t r = (g >> 5) * PER + (g & (PER - 1));
    if (r >= T.NR) return;
    request_item<RQ_NV>(T, cur, r, ((int)g & 31) / PER * RQ_NV, T.rq_geo + rq_geo_at(r));
}
__global__ void __launch_bounds__(128) k_requests(Tables T, double4 *cur) {
    dep_begin();
    requests_block(T, cur);
}

// lambda/time-step control (src/solution.F90:185-201)
__device__ __forceinline__ void step_control(DevScalars *sc, const fdm_params &P, int use_dt, bool step_follows) {
    step_control_item(sc, P, use_dt);
    // the step's stage 3 collects the next lambda from zero
    if (step_follows) { sc->lam_next_x = 0.0; sc->lam_next_y = 0.0; }
}
__global__ void k_step_control(DevScalars *sc, fdm_params P, int use_dt, bool step_follows) {
    dep_begin();
    if (threadIdx.x || blockIdx.x) return;
    step_control(sc, P, use_dt, step_follows);
}
// a step's first kernel: its control, which the values do not depend on, by
// the last block, beside stage 1's values by the others
__global__ void __launch_bounds__(128) k_step_begin(Tables T, double4 *cur, DevScalars *sc, fdm_params P) {
    dep_begin();
    if (blockIdx.x + 1 < gridDim.x) requests_block(T, cur);
    else if (threadIdx.x == 0) step_control(sc, P, 1, true);
}

// interpA fallbacks of parent_value_weno: one warp per listed request
__global__ void __launch_bounds__(128) k_requests_restrict(Tables T, double4 *cur) {
    __shared__ RestrictSmem sm[4];
    const int64_t w = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (w >= T.NRR) return;
    request_restrict_warp(T, cur, T.rq_rlist[w], sm[threadIdx.x >> 5]);
}

// One thread per face; TB threads per block, at least MINB blocks per SM
// (the register budget follows from both).  One launch covers the x faces
// and then the y faces (nbx blocks of x), so both share the last wave.
//
// Bound by the FP64 pipe: about 2000 FP64 instructions per face, two cycles
// each on a quarter of an SM.  What it took to keep the pipe busy was
// straight-line code (numerics_nr.cuh), not occupancy: 16 warps at 128
// registers or 12 at 168 or 20 at 96 are within 2 %.  One B200, x+y pair, ms,
// beside the compiler's division in one launch per direction (its best
// shape): 1.03M leaves 0.213 (0.432), 260k 0.060 (0.113), 148k 0.037 (0.077),
// 17k 0.0104 (0.0309), 3k 0.0067 (0.0247).
template <int TB, int MINB>
__global__ void __launch_bounds__(TB, MINB) k_faces(Tables T, const double4 *__restrict__ cur, double4 *Fx,
                                                    double4 *Fy, const DevScalars *__restrict__ sc, double g,
                                                    FluxDen den, int nbx) {
    dep_begin();
    const int64_t b = blockIdx.x;
    if (b < nbx) {
        const int64_t f = b * TB + threadIdx.x;
        if (f < T.NI + T.nux) face_item<0>(T, cur, Fx, sc->lambda_x, g, den, f);
    } else {
        const int64_t f = (b - nbx) * TB + threadIdx.x;
        if (f < T.NI + T.nuy) face_item<1>(T, cur, Fy, sc->lambda_y, g, den, f);
    }
}

// Two lanes per face, for meshes whose faces do not fill the GPU once with one
// thread each: there a face's chain of dependent operations is the time, and
// half of the work per lane nearly halves it, for 12 % more operations.  The
// 168 registers of three blocks per SM beat 128 by 5 %.  x+y pair, ms, beside
// one thread per face: 3k leaves 0.0040 (0.0053), 11k 0.0052 (0.0063), 20k
// 0.0070 (0.0080), 36k 0.0111 (0.0122), 45k 0.0142 (0.0141).  Four lanes (left
// and right apart too) give 0.0035 at 3k, 0.0057 at 11k and are slower above.
template <int TB, int MINB>
__global__ void __launch_bounds__(TB, MINB) k_faces_pair(Tables T, const double4 *__restrict__ cur, double4 *Fx,
                                                         double4 *Fy, const DevScalars *__restrict__ sc, double g,
                                                         FluxDen den, int nbx) {
    dep_begin();
    const int64_t b = blockIdx.x;
    if (b < nbx) face_item_pair<0>(T, cur, Fx, sc->lambda_x, g, den, (b * TB + threadIdx.x) >> 1, T.NI + T.nux);
    else face_item_pair<1>(T, cur, Fy, sc->lambda_y, g, den, ((b - nbx) * TB + threadIdx.x) >> 1, T.NI + T.nuy);
}

// Diagnostics: the faces whose branch-free division meets an operand
// outside its range (and so are computed again with the compiler's
// division), counted over the current state; nothing is written to F.
template <int DIR>
__global__ void __launch_bounds__(128) k_faces_nr_count(Tables T, const double4 *__restrict__ cur,
                                                        const DevScalars *__restrict__ sc, double g,
                                                        FluxDen den, unsigned long long *count) {
    const int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nu = DIR == 0 ? T.nux : T.nuy;
    bool fell = false;
    if (f < T.NI + nu) {
        int32_t a, b, c, d;
        face_slots<DIR>(T, f, a, b, c, d);
        double out[4];
        DivNR dv(den);
        face_flux_nr<DIR>(cur, a, b, c, d, g, dv, DIR == 0 ? sc->lambda_x : sc->lambda_y, out);
        fell = !dv.ok;
    }
    const unsigned m = __ballot_sync(0xffffffffu, fell);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(count, (unsigned long long)__popc(m));
}
int count_nr_fallbacks(fdm_handle *h, int64_t out[2]) {
    const Tables T = h->tables();
    const DevScalars *sc = h->scal.as<DevScalars>();
    const double g = h->G.gama;
    const FluxDen den = flux_den(g);
    FDM_CK(h, h->tmp[7].ensure(2 * sizeof(unsigned long long)));
    unsigned long long *cnt = h->tmp[7].as<unsigned long long>();
    FDM_CK(h, cudaMemsetAsync(cnt, 0, 2 * sizeof(unsigned long long), h->s));
    launch_requests(h, h->B[0].as<double4>());
    k_faces_nr_count<0><<<nblk(h->NI + h->nux, 128), 128, 0, h->s>>>(T, h->B[0].as<double4>(), sc, g, den, cnt);
    k_faces_nr_count<1><<<nblk(h->NI + h->nuy, 128), 128, 0, h->s>>>(T, h->B[0].as<double4>(), sc, g, den,
                                                                       cnt + 1);
    unsigned long long hc[2];
    FDM_CK(h, cudaMemcpyAsync(hc, cnt, sizeof hc, cudaMemcpyDeviceToHost, h->s));
    FDM_CK(h, cudaStreamSynchronize(h->s));
    out[0] = (int64_t)hc[0];
    out[1] = (int64_t)hc[1];
    return FDM_OK;
}

// Residual + forward-Euler candidate fused with updateRK, 256 leaves per
// block (the residual partials are per block of 256).  Bound by L1: ten
// records a leaf, of which neighbours share most.  At 1.03 M leaves 64 us with
// 128-bit accesses and the compiler's divisions (128 registers), 55 us with
// 256-bit ones and branch-free quotients, 45 us at 80 registers (MINB 3), 33 us
// in stages 1 and 2, which reduce no residual.
template <int MINB>
__global__ void __launch_bounds__(256, MINB) k_cells(const __grid_constant__ Tables T,
                                                const __grid_constant__ LevelTab LT,
                                                const double4 *__restrict__ cur,
                                                const double4 *un, double4 *next,
                                                const double4 *__restrict__ Fx, const double4 *__restrict__ Fy,
                                                DevScalars *sc, double *res_part, int krk, int mode, double g,
                                                const __grid_constant__ FluxDen den) {
    __shared__ CellsSmem S;
    dep_begin();
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    double rm[4] = {0.0, 0.0, 0.0, 0.0}, rs[4] = {0.0, 0.0, 0.0, 0.0};
    double lx = 0.0, ly = 0.0;
    // an iteration after t_end (or after a NaN residual) leaves the state as it is
    if (i < T.NI && !(mode == 0 && sc->done))
        cell_item(T, LT, cur, un, next, Fx, Fy, sc->tstep, krk, mode, g, den, i, rm, rs, lx, ly);
    // the norms and wave speeds of a step are those of its last stage
    if (mode == 0 && krk != 3) return;
    cells_block_reduce(rm, rs, lx, ly, res_part + blockIdx.x * 8, sc, krk == 3 && mode == 0, S);
}

__global__ void k_blend(int64_t NI, const double4 *__restrict__ un, const double4 *__restrict__ ut, double4 *cur,
                        int krk) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= NI) return;
    const double ra = krk == 1 ? 0.0 : krk == 2 ? 3.0 / 4.0 : 1.0 / 3.0;
    const double rb = krk == 1 ? 1.0 : krk == 2 ? 1.0 / 4.0 : 2.0 / 3.0;
    const double4 a = un[i], b = ut[i];
    cur[i] = make_double4(ra * a.x + rb * b.x, ra * a.y + rb * b.y, ra * a.z + rb * b.z, ra * a.w + rb * b.w);
}

// ghost leaves: the first nbs blocks take a thread for each that is imaged by
// a copy or a boundary state, the others a warp for each that is imaged by a
// subtree restriction (interpA images can span hundreds of leaves)
__global__ void __launch_bounds__(128) k_ghost(Tables T, double4 *buf, GhostStates GS,
                                               const DevScalars *__restrict__ sc, int j, int nbs) {
    __shared__ RestrictSmem sm[4];
    dep_begin();
    const int64_t b = blockIdx.x;
    if (b < nbs) {
        const int64_t gi = b * 128 + threadIdx.x;
        if (gi >= T.NG) return;
        const int kind = T.gh_kind[gi];
        if (kind == GH_NONE || kind == GH_RESTRICT) return;
        ghost_store(T, buf, gi, ghost_simple_value(T, buf, GS, sc, j, gi, kind));
    } else {
        const int64_t w = (b - nbs) * 4 + (threadIdx.x >> 5);
        if (w < T.NGR) ghost_warp(T, buf, GS, sc, j, T.gh_rlist[w], sm[threadIdx.x >> 5]);
    }
}

// Largest wave speeds.  One atomic per block, and only where it raises the
// maximum: one per warp (32k of them on one word at 1.03 M leaves) took 46 us.
__global__ void __launch_bounds__(256) k_lambda(int64_t NI, const double4 *__restrict__ cur, DevScalars *sc, double g) {
    __shared__ double sx[8], sy[8];
    double lx = 0.0, ly = 0.0;
    for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < NI; i += gridDim.x * 256ll) {
        const double4 o = load_record(cur + i);
        const double c = sqrt(g * o.w / o.x);
        lx = fmax(lx, fabs(o.y) + c);
        ly = fmax(ly, fabs(o.z) + c);
    }
    for (int o = 16; o; o >>= 1) {
        lx = fmax(lx, __shfl_xor_sync(0xffffffffu, lx, o));
        ly = fmax(ly, __shfl_xor_sync(0xffffffffu, ly, o));
    }
    if ((threadIdx.x & 31) == 0) { sx[threadIdx.x >> 5] = lx; sy[threadIdx.x >> 5] = ly; }
    __syncthreads();
    if (threadIdx.x) return;
    for (int k = 1; k < 8; ++k) { lx = fmax(lx, sx[k]); ly = fmax(ly, sy[k]); }
    if (lx > __ldcg(&sc->lam_next_x))
        atomicMax((unsigned long long *)&sc->lam_next_x, (unsigned long long)__double_as_longlong(lx));
    if (ly > __ldcg(&sc->lam_next_y))
        atomicMax((unsigned long long *)&sc->lam_next_y, (unsigned long long)__double_as_longlong(ly));
}

// residual partials -> Res_max / Res_rms sums, and (end) the end of one
// solute iteration: tt, rms, NaN stop, t_end (src/solution.F90:205-215)
__global__ void __launch_bounds__(1024) k_res_finalize(const double *__restrict__ res_part, int nb, DevScalars *sc,
                                                       int keep_when_done, bool end, int64_t NI) {
    __shared__ double sh[256][8];
    dep_begin();
    if (keep_when_done && sc->done) return;   // a no-op iteration keeps the last residual
    res_finalize_block<1024>(res_part, nb, sc, sh);
    if (end && threadIdx.x == 0) step_end_item(sc, NI);
}

__global__ void k_set_tstep(DevScalars *sc, double tstep) {
    if (threadIdx.x || blockIdx.x) return;
    sc->tstep = tstep;
}

// ------------------------------------------------------------ launchers
static void launch_requests_restrict(fdm_handle *h, const double4 *cur) {
    if (h->n_restrict > 0)
        k_requests_restrict<<<nblk(h->n_restrict, 4), 128, 0, h->s>>>(h->tables(), (double4 *)cur);
}
void launch_requests(fdm_handle *h, const double4 *cur) {
    if (h->NR == 0) return;
    launch_after(h->s, nblk(h->NR, 128 * RQ_NV / 4), 128, k_requests, h->tables(), (double4 *)cur);
    launch_requests_restrict(h, cur);
}
// Launch shapes of the face kernel that the autotuner chooses from; shape 0
// is what a handle starts with.  The variant numbers run on past the shapes
// and repeat them.
template <int TB, int MINB>
static void faces(fdm_handle *h, const double4 *cur) {
    const double g = h->G.gama;
    const int nbx = nblk(h->NI + h->nux, TB), nby = nblk(h->NI + h->nuy, TB);
    launch_after(h->s, nbx + nby, TB, k_faces<TB, MINB>, h->tables(), cur, h->Fx.as<double4>(), h->Fy.as<double4>(),
                 h->scal.as<DevScalars>(), g, flux_den(g), nbx);
}
template <int TB, int MINB>
static void faces_pair(fdm_handle *h, const double4 *cur) {
    const double g = h->G.gama;
    const int nbx = nblk(h->NI + h->nux, TB / 2), nby = nblk(h->NI + h->nuy, TB / 2);
    launch_after(h->s, nbx + nby, TB, k_faces_pair<TB, MINB>, h->tables(), cur, h->Fx.as<double4>(),
                 h->Fy.as<double4>(), h->scal.as<DevScalars>(), g, flux_den(g), nbx);
}
void launch_faces(fdm_handle *h, const double4 *cur, int krk) {
    if (h->gate_on) {
        launch_gated_faces(h, cur, krk);
        return;
    }
    if (h->p.flux_variant == 1) {
        launch_faces_fast(h, cur);
        return;
    }
    switch (h->face_variant % N_FACE_SHAPES) {
        case 1: faces<128, 3>(h, cur); break;
        case 2: faces<64, 8>(h, cur); break;
        case 3: faces<256, 2>(h, cur); break;
        case 4: faces<128, 5>(h, cur); break;
        case 5: faces<128, 6>(h, cur); break;
        default:
            // two lanes per face up to three waves of theirs (64 faces a block,
            // three blocks on each of the 148 SMs), about 41k leaves: 36k
            // leaves 0.0111 ms against 0.0122, 45k 0.0142 against 0.0141
            if (2 * h->NI + h->nux + h->nuy <= 3 * 3 * 148 * 64) faces_pair<128, 3>(h, cur);
            else faces<128, 4>(h, cur);
            break;
    }
}

static void launch_res_finalize(fdm_handle *h, bool keep_when_done, bool end) {
    launch_after(h->s, 1, 1024, k_res_finalize, h->res_part.as<double>(), nblk(h->NI, 256), h->scal.as<DevScalars>(),
                 keep_when_done, end, h->NI);
}
void launch_cells(fdm_handle *h, const double4 *cur, const double4 *un, double4 *next, int krk, int mode,
                  bool finalize) {
    // three blocks per SM above four blocks on each of the 148 SMs.  A step with
    // three and with two, ms: 194k leaves 0.1924 (0.1935), 260k 0.244 (0.247),
    // 328k 0.2915 (0.303), 402k 0.354 (0.365), 628k 0.543 (0.560), 1.03M 0.834
    // (0.859); below the line, at 148k (two full waves of two), 0.1510 (0.1495).
    const unsigned nb = nblk(h->NI, 256);
    launch_after(h->s, nb, 256, nb > 4u * 148u ? k_cells<3> : k_cells<2>, h->tables(), h->lt, cur, un, next,
                 h->Fx.as<double4>(), h->Fy.as<double4>(), h->scal.as<DevScalars>(), h->res_part.as<double>(), krk, mode,
                 h->G.gama, flux_den(h->G.gama));
    // Res_max / Res_rms are reset every stage and read after the last one
    // (src/solution.F90:276-277, 209-210): reduce them once, after stage 3
    if (finalize && (krk == 3 || mode == 1)) launch_res_finalize(h, mode == 0, false);
}
void launch_ghosts(fdm_handle *h, double4 *next, int j) {
    if (h->NG == 0) return;
    const int nbs = nblk(h->NG, 128);
    launch_after(h->s, nbs + nblk(h->n_ghost_restrict, 4), 128, k_ghost, h->tables(), next, ghost_states(h->p),
                 h->scal.as<DevScalars>(), j, nbs);
}
void launch_blend(fdm_handle *h, const double4 *un, double4 *cur, int krk) {
    k_blend<<<nblk(h->NI, 256), 256, 0, h->s>>>(h->NI, un, h->Ut.as<double4>(), cur, krk);
}
void launch_lambda(fdm_handle *h, const double4 *cur) {
    k_lambda<<<std::min(nblk(h->NI, 256), 8 * 148), 256, 0, h->s>>>(h->NI, cur, h->scal.as<DevScalars>(), h->G.gama);
}
void launch_step_control(fdm_handle *h) {
    k_step_control<<<1, 32, 0, h->s>>>(h->scal.as<DevScalars>(), h->p, 1, false);
}
void launch_set_tstep(fdm_handle *h, double tstep) {
    k_set_tstep<<<1, 32, 0, h->s>>>(h->scal.as<DevScalars>(), tstep);
}

// One RK stage on the three state buffers: B0 holds the step-start state
// (Un); stage 1: B0 -> B1, stage 2: B1 -> B2, stage 3: B2 -> B0.
static void stage_faces_cells(fdm_handle *h, int krk, bool finalize) {
    double4 *b[3] = {h->B[0].as<double4>(), h->B[1].as<double4>(), h->B[2].as<double4>()};
    const double4 *cur = b[krk - 1];
    launch_faces(h, cur, krk);
    launch_cells(h, cur, b[0], b[krk % 3], krk, 0, finalize);
}
int launch_stage(fdm_handle *h, int krk) {
    launch_requests(h, h->B[krk - 1].as<double4>());
    stage_faces_cells(h, krk, true);
    launch_ghosts(h, h->B[krk % 3].as<double4>(), 3);
    return FDM_OK;
}
// One solute iteration without AMR: step control, RK3, tt/residual/NaN;
// refresh: followed by the j = 1 ghost refresh that solute does after an
// iteration without regrid.  That refresh writes every ghost that the stage-3
// fill (j = 3) writes, and nothing reads them in between, so it stands for it.
//
// A step of a small mesh is a chain of short kernels: the control rides with
// the first one (3.8k leaves 41.1 -> 39.1 us, 15k 62.4 -> 60.6).  The step's
// end by the last block of the last cell update took as long as its kernel.
void launch_step(fdm_handle *h, bool refresh) {
    double4 *B0 = h->B[0].as<double4>();
    if (h->NR > 0) {
        launch_after(h->s, nblk(h->NR, 128 * RQ_NV / 4) + 1, 128, k_step_begin, h->tables(), B0,
                     h->scal.as<DevScalars>(), h->p);
        launch_requests_restrict(h, B0);
    } else {
        launch_after(h->s, 1, 32, k_step_control, h->scal.as<DevScalars>(), h->p, 1, true);
    }
    stage_faces_cells(h, 1, false);
    launch_ghosts(h, h->B[1].as<double4>(), 3);
    launch_stage(h, 2);
    launch_requests(h, h->B[2].as<double4>());
    stage_faces_cells(h, 3, false);
    if (!refresh) launch_ghosts(h, B0, 3);   // before tt moves on
    launch_res_finalize(h, true, true);
    if (refresh) launch_ghosts(h, B0, 1);
}

}  // namespace fdm
