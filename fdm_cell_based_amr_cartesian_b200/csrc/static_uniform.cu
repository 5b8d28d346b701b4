// static_uniform.cu — one SSP-RK3 step of the WCNS scheme on a uniform
// periodic grid without any device allocation.
//
// Some callers cannot allocate device memory: a Fortran or C host whose GPU
// memory is handed out by its own pool (an OpenACC or CUDA Fortran runtime
// that owns the heap), code that must run under a fixed memory budget set
// at start-up, or a process that forbids cudaMalloc after initialisation.
// For them this entry point keeps its working memory (the two intermediate
// stage states and the x/y face fluxes) in one file-scope static __device__
// array of fixed size (8.5 MiB), which every GPU that loads libfdm holds
// until the process exits.  The caller passes the input and output states.
//
// The arithmetic is the exact build's (same face_flux and update as the
// handle path, same operation order), so the result equals fdm_time_advance_rk
// on the same uniform periodic leaf set.
#include <algorithm>
#include <cstdint>

#include "handle.cuh"
#include "items.cuh"

namespace fdm {
namespace uniform_static {

// worst cases over 3 <= nx, ny <= FDM_STATIC_MAX_SIDE, nx*ny <= FDM_STATIC_MAX_CELLS
constexpr int64_t GRID_CAP = 72100;   // (nx+6)*(ny+6) records
constexpr int64_t FACE_CAP = 66560;   // max((nx+1)*ny, nx*(ny+1)) records
constexpr int64_t SCRATCH_RECORDS = 2 * GRID_CAP + 2 * FACE_CAP;

// The scratch.  In host code this name is only a stand-in for the device
// symbol; its device address comes from cudaGetSymbolAddress below.
static __device__ __align__(256) double4 scratch[SCRATCH_RECORDS];

// Device address of the scratch on the current device.  It is looked up on
// every call, with the caller's device current: a cached address would go
// stale when the context that loaded the module is torn down and created
// again (cudaDeviceReset), and the lookup is a cheap runtime call.  The
// first call on a device also loads the module there (lazy loading).
static cudaError_t scratch_address(double4 **out) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, scratch);
    if (e != cudaSuccess) return e;
    *out = (double4 *)p;
    return cudaSuccess;
}

struct Grid2 {
    int nx, ny, W;   // W = nx + 6 records per row
    __device__ __forceinline__ int64_t at(int r, int c) const { return (int64_t)r * W + c; }
};

// face i of row r in x lies between interior columns 3+i-1 and 3+i; the x
// faces' blocks (nbx), then the y faces'.  Two lanes per face (as in
// k_faces_pair): the faces fill the GPU a few times at most.
template <int DIR>
__device__ __forceinline__ void uface(const Grid2 &G, const double4 *__restrict__ cur, double4 *F, double g,
                                      const FluxDen &den, double lam, int t) {
    const int nfr = DIR == 0 ? G.nx + 1 : G.nx;          // faces per row
    const int nrow = DIR == 0 ? G.ny : G.ny + 1;
    const int f = min(t >> 1, nfr * nrow - 1);
    const int r = f / nfr, i = f - r * nfr;
    const int step = DIR == 0 ? 1 : G.W, c = (int)G.at(3 + r, 3 + i);
    const double2 v = face_flux_pair<DIR>(cur, c - 2 * step, c - step, c, c + step, g, den, lam);
    if (f == t >> 1) reinterpret_cast<double2 *>(F + f)[t & 1] = v;
}
// One step (six launches), us: 45 x 38 19.4, 128 x 128 24.7, 256 x 256 57.6;
// with one thread per face 21.6, 27.2, 58.5, and with launches that wait for
// the end of the kernel before 30.9, 37.1, 67.8 (and the cells' divisions the
// compiler's).
__global__ void __launch_bounds__(64, 6) k_ufaces(Grid2 G, const double4 *__restrict__ cur, double4 *Fx, double4 *Fy,
                                                  double g, FluxDen den, double lam_x, double lam_y, int nbx) {
    const int b = blockIdx.x;
    dep_begin();
    if (b < nbx) uface<0>(G, cur, Fx, g, den, lam_x, b * 64 + threadIdx.x);
    else uface<1>(G, cur, Fy, g, den, lam_y, (b - nbx) * 64 + threadIdx.x);
}

// the cell's value (the operations of k_cells)
template <class D>
__device__ __forceinline__ CellValue ucell(const Grid2 &G, const double4 *__restrict__ cur, const double4 *un,
                                           const double4 *__restrict__ Fx, const double4 *__restrict__ Fy, double g,
                                           const FluxDen &den, const CellCoef &k, double tstep, int krk, int r, int i) {
    const int row = 3 + r, col = 3 + i;
    const int64_t self = G.at(row, col), fx = (int64_t)r * (G.nx + 1) + i, fy = (int64_t)r * G.nx + i;
    return cell_update<D>(load_prim(cur, self), load_prim(cur, G.at(row, col + 1)), load_prim(cur, G.at(row, col - 1)),
                          load_prim(cur, G.at(row + 1, col)), load_prim(cur, G.at(row - 1, col)), load_record(Fx + fx + 1),
                          load_record(Fx + fx), load_record(Fy + fy + G.nx), load_record(Fy + fy), k, un + self, tstep,
                          krk, 0, g, den);
}
// a cell that DivNR refuses, out of line
__device__ __noinline__ CellValue ucell_again(const Grid2 &G, const double4 *cur, const double4 *un, const double4 *Fx,
                                              const double4 *Fy, double g, const FluxDen &den, const CellCoef &k,
                                              double tstep, int krk, int r, int i) {
    return ucell<DivIEEE>(G, cur, un, Fx, Fy, g, den, k, tstep, krk, r, i);
}

// LXL + updateRK for every interior cell, and its periodic images among the
// ghosts (BC_cyc at level 0, src/solution.F90:116-136): the thread that makes
// a value stores its copies.  The corners are left alone, as the reference
// never refills them; at stage 3 the threads past the cells copy them from
// the input.
__global__ void __launch_bounds__(128) k_ucells(const __grid_constant__ Grid2 G, const double4 *__restrict__ cur,
                                                const double4 *un, double4 *next, const double4 *__restrict__ Fx,
                                                const double4 *__restrict__ Fy, double g,
                                                const __grid_constant__ FluxDen den,
                                                const __grid_constant__ CellCoef k, double tstep, int krk) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int ncell = G.nx * G.ny;
    dep_begin();
    if (t >= ncell) {
        const int c = (int)t - ncell;   // corner record c of 36: 3 x 3 at each end of both sides
        if (krk == 3 && c < 36) {
            const int a = c / 6, b = c % 6;
            const int64_t at = G.at(a < 3 ? a : G.ny + a, b < 3 ? b : G.nx + b);
            next[at] = un[at];
        }
        return;
    }
    const int r = (int)t / G.nx, i = (int)t - r * G.nx;
    const int row = 3 + r, col = 3 + i;
    CellValue v = ucell<DivNR>(G, cur, un, Fx, Fy, g, den, k, tstep, krk, r, i);
    if (!v.ok) v = ucell_again(G, cur, un, Fx, Fy, g, den, k, tstep, krk, r, i);
    store_record(next + G.at(row, col), v.o);
    if (col >= G.nx) store_record(next + G.at(row, col - G.nx), v.o);
    if (col <= 5) store_record(next + G.at(row, col + G.nx), v.o);
    if (row >= G.ny) store_record(next + G.at(row - G.ny, col), v.o);
    if (row <= 5) store_record(next + G.at(row + G.ny, col), v.o);
}

static inline unsigned nb(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace uniform_static
}  // namespace fdm

extern "C" int fdm_time_advance_rk_uniform_static(const double *prim_in, double *prim_out, int32_t nx,
                                                  int32_t ny, double h, double x_factor, double gama,
                                                  double lambda_x, double lambda_y, double tstep,
                                                  void *stream) {
    using namespace fdm::uniform_static;
    if (!prim_in || !prim_out) return FDM_ERR_ARG;
    if (nx < 3 || ny < 3 || nx > FDM_STATIC_MAX_SIDE || ny > FDM_STATIC_MAX_SIDE ||
        (int64_t)nx * ny > FDM_STATIC_MAX_CELLS)
        return FDM_ERR_ARG;   // outside the fixed scratch: nothing was enqueued
    const int64_t ngrid = (int64_t)(nx + 6) * (ny + 6);
    const int64_t nface = std::max((int64_t)(nx + 1) * ny, (int64_t)nx * (ny + 1));
    if (ngrid > GRID_CAP || nface > FACE_CAP) return FDM_ERR_ARG;
    if (((uintptr_t)prim_in | (uintptr_t)prim_out) & 31) return FDM_ERR_ARG;   // 32-byte records
    // stage 3 reads prim_in while it writes prim_out, and the corners are
    // copied from prim_in last: the two ranges must not share a byte
    const uintptr_t ia = (uintptr_t)prim_in, oa = (uintptr_t)prim_out, nbytes = (uintptr_t)ngrid * 32;
    if (ia < oa + nbytes && oa < ia + nbytes) return FDM_ERR_ARG;
    // an error left pending by earlier, unrelated work is the caller's, not
    // this call's: refuse before enqueueing anything rather than report it
    if (cudaPeekAtLastError() != cudaSuccess) return FDM_ERR_CUDA;
    double4 *base = nullptr;
    if (scratch_address(&base) != cudaSuccess) return FDM_ERR_CUDA;
    double4 *U1 = base, *U2 = base + GRID_CAP, *Fx = base + 2 * GRID_CAP, *Fy = Fx + FACE_CAP;
    cudaStream_t s = (cudaStream_t)stream;
    Grid2 G{nx, ny, nx + 6};
    const double dy = h, dx = x_factor * dy;
    const double cxa = 4.0 / (3.0 * dx), cxb = 1.0 / (6.0 * dx);
    const double cya = 4.0 / 3.0 / dy, cyb = 1.0 / 6.0 / dy;
    const fdm::CellCoef k{cxa, cxb, cya, cyb, dx, dy};
    const double4 *in = (const double4 *)prim_in;
    double4 *out = (double4 *)prim_out;
    const double4 *cur[3] = {in, U1, U2};
    double4 *next[3] = {U1, U2, out};
    const fdm::FluxDen den = fdm::flux_den(gama);
    const unsigned nbx = nb((int64_t)(nx + 1) * ny, 32), nby = nb((int64_t)nx * (ny + 1), 32);
    for (int krk = 1; krk <= 3; ++krk) {
        // the first launch waits for all of the caller's work before it, the
        // later ones' threads for the kernel before
        if (krk == 1)
            k_ufaces<<<nbx + nby, 64, 0, s>>>(G, cur[0], Fx, Fy, gama, den, lambda_x, lambda_y, (int)nbx);
        else
            fdm::launch_after(s, nbx + nby, 64, k_ufaces, G, cur[krk - 1], Fx, Fy, gama, den, lambda_x, lambda_y,
                              (int)nbx);
        fdm::launch_after(s, nb((int64_t)nx * ny + 36, 128), 128, k_ucells, G, cur[krk - 1], in, next[krk - 1], Fx, Fy,
                          gama, den, k, tstep, krk);
    }
    return cudaGetLastError() == cudaSuccess ? FDM_OK : FDM_ERR_CUDA;
}
