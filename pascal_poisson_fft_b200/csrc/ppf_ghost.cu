// ppf_ghost.cu -- ghost-cell update of the ghosted solution (sm_100a), and
// the device-side refinement gate.
//
// The reference fills the ghost cells in a fixed order: quadratic Neumann
// extrapolation along every non-periodic axis (apply_bc_on_direction,
// 01_Fortran/src/fft_3d_poisson.f90:798-852, x then y then z), then the
// periodic copies along every periodic axis (ghostcell_update_on_direction
// at one rank, :709-796, x then y then z).  Each step covers the whole face
// including the other axes' ghost lines, so later steps read values written
// by earlier ones.  Here one launch computes every ghost cell from interior
// cells alone: a cell's value is the one of the last step that writes it,
// evaluated with the earlier steps' values of its neighbours substituted (an
// edge or corner nests two or three steps, up to eight interior cells, in the
// same order of operations).  Bound by launch latency on small grids: three
// launches took 11 us of a 64^3 solve.
#include "ppf_misc_dev.cuh"

#include <algorithm>
#include <math.h>

namespace ppf {

struct GhostArgs {
    double* P;
    int n[3];                 // cells
    int per[3];               // periodic axes
    long st[3];               // strides of P
    const double* dmx[3];
    int faces[3];             // faces to fill (1 lower, 2 upper)
    int ord[3];               // axes in the order of the steps
    long count[3];            // ghost cells of each axis's faces (both): x with every y and z,
                              // y with interior x, z with interior x and y
};

// One axis of a ghost cell's evaluation: value = c0 v(o0) - c1 v(o1), or v(o0)
struct GhostAxis {
    long o0, o1;
    double c0, c1;
    bool two;
};

__device__ __forceinline__ GhostAxis ghost_axis_of(const GhostArgs& g, int d, int i)
{
    GhostAxis a;
    a.two = false;
    a.o1 = 0;
    a.c0 = a.c1 = 0.0;
    const int n = g.n[d];
    const bool lo = i == 0 && (g.faces[d] & 1), hi = i == n + 1 && (g.faces[d] & 2);
    if (!lo && !hi) {
        a.o0 = i * g.st[d];
    } else if (g.per[d]) {
        a.o0 = (lo ? n : 1) * g.st[d];
    } else {
        const double* dmx = g.dmx[d];
        const double e = lo ? dmx[1] : dmx[n + 1], e2 = lo ? dmx[2] : dmx[n];
        const double s = e + e2;
        a.two = true;
        a.c0 = (s * s) / ((s * s) - e * e);
        a.c1 = (e * e) / ((s * s) - e * e);
        a.o0 = (lo ? 1 : n) * g.st[d];
        a.o1 = (lo ? 2 : n - 1) * g.st[d];
    }
    return a;
}

__global__ void __launch_bounds__(256) k_ghosts(const __grid_constant__ GhostArgs g)
{
    pdl_wait();
    const long total = g.count[0] + g.count[1] + g.count[2];
    for (long q = threadIdx.x + (long)blockIdx.x * blockDim.x; q < total; q += (long)blockDim.x * gridDim.x) {
        int c[3];
        if (q < g.count[2]) {                       // z faces, interior x and y (coalesced)
            const unsigned r = (unsigned)q, nx = g.n[0];
            const unsigned row = r / nx;
            c[0] = (int)(r - row * nx) + 1;
            c[1] = (int)(row % (unsigned)g.n[1]) + 1;
            const int face = (int)(row / (unsigned)g.n[1]);
            c[2] = (g.faces[2] == 3 ? face == 0 : g.faces[2] == 1) ? 0 : g.n[2] + 1;
        } else if (q < g.count[2] + g.count[1]) {   // y faces, interior x, every z
            const unsigned r = (unsigned)(q - g.count[2]), nx = g.n[0];
            const unsigned row = r / nx;
            c[0] = (int)(r - row * nx) + 1;
            c[2] = (int)(row >> 1);
            c[1] = (row & 1) ? g.n[1] + 1 : 0;
        } else {                                    // x faces, every y and z
            const unsigned r = (unsigned)(q - g.count[2] - g.count[1]), row = r >> 1, ny = g.n[1] + 2;
            c[2] = (int)(row / ny);
            c[1] = (int)(row - (unsigned)c[2] * ny);
            c[0] = (r & 1) ? g.n[0] + 1 : 0;
        }
        const long at = c[0] * g.st[0] + c[1] * g.st[1] + c[2] * g.st[2];
        const GhostAxis a = ghost_axis_of(g, g.ord[0], c[g.ord[0]]);
        const GhostAxis b = ghost_axis_of(g, g.ord[1], c[g.ord[1]]);
        const GhostAxis e = ghost_axis_of(g, g.ord[2], c[g.ord[2]]);
        auto first = [&](long o) {
            return a.two ? a.c0 * g.P[o + a.o0] - a.c1 * g.P[o + a.o1] : g.P[o + a.o0];
        };
        auto second = [&](long o) { return b.two ? b.c0 * first(o + b.o0) - b.c1 * first(o + b.o1) : first(o + b.o0); };
        g.P[at] = e.two ? e.c0 * second(e.o0) - e.c1 * second(e.o1) : second(e.o0);
    }
}

cudaError_t launch_ghosts(double* P, const Geom& g, const double* dmx1, const double* dmx2, const double* dmx3,
                          LStream st, int zfaces)
{
    GhostArgs a{};
    a.P = P;
    const int n[3] = { g.nx, g.ny, g.nz }, per[3] = { g.px, g.py, g.pz };
    const long str[3] = { 1, g.pstride_y, g.pstride_z };
    const double* dmx[3] = { dmx1, dmx2, dmx3 };
    int k = 0;
    for (int pass = 0; pass < 2; ++pass)            // Neumann axes first, then periodic axes
        for (int d = 0; d < 3; ++d)
            if ((pass == 0) == !per[d]) a.ord[k++] = d;
    for (int d = 0; d < 3; ++d) {
        a.n[d] = n[d];
        a.per[d] = per[d];
        a.st[d] = str[d];
        a.dmx[d] = dmx[d];
        // z of a slab: walls only at the global ends (zfaces), the planes
        // between slabs hold the neighbouring ranks' values
        a.faces[d] = d == 2 ? zfaces : 3;
    }
    a.count[0] = 2L * (g.ny + 2) * (g.nz + 2);
    a.count[1] = 2L * g.nx * (g.nz + 2);
    a.count[2] = (long)((zfaces & 1) + (zfaces >> 1)) * g.nx * g.ny;
    const long want = (a.count[0] + a.count[1] + a.count[2] + 255) / 256;
    int sms = 0;
    const cudaError_t e = device_sms(&sms);
    if (e != cudaSuccess) return e;
    return launch_on(k_ghosts, dim3((unsigned)std::min(want, 64L * sms)), 256, 0, st, a);
}

__global__ void __launch_bounds__(512) k_sweep_gate(const double* partials, long nblocks, double ncell,
                                                    double* mean_prev, int* skip, int* sweeps_done, double* last_rel,
                                                    double tol, int initial)
{
    pdl_enter();
    sweep_gate(partials, nblocks, ncell, mean_prev, skip, sweeps_done, last_rel, tol, initial);
}

cudaError_t launch_sweep_gate(const double* partials, long nblocks, double ncell, double* mean_prev, int* skip_flag,
                              int* sweeps_done, double* last_rel, double tol, int initial, LStream st)
{
    return launch_on(k_sweep_gate, dim3(1), 512, 0, st, partials, nblocks, ncell, mean_prev, skip_flag, sweeps_done, last_rel, tol, initial);
}

}  // namespace ppf
