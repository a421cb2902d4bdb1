// darcy.cu -- Darcy flow through the packing (src/darcy.cuh:169-779, launched
// at src/device.cu:913-1021) and its host-side initialisation
// (src/darcy.cpp:69-798).
//
// The reference runs six kernels per step, each over the fluid grid (the
// cell grid): porosity, transmissivity, ghost nodes, explicit pressure step,
// pressure gradient, velocity.  Here they are four:
//   k_darcy_porosity  porosity of every node from the cell list of the
//                     step's start positions, and from it the node's
//                     conductivity and transmissivity (a per-node function,
//                     so fusing changes no value);
//   k_darcy_ghosts    the boundary nodes copied onto the opposite ghost
//                     nodes, over the face nodes instead of the whole grid;
//   k_darcy_explicit  the explicit step of the pressure;
//   k_darcy_grad_vel  pressure gradient and pore velocity (per node again).
// Every expression keeps the reference's operands and order (FP64, no
// contraction), so the results are the reference's bit for bit.  The
// kernels read the step's start positions and the cell list, which the
// contact-force kernel leaves untouched, and write only the fluid grid.
#include "sphk_internal.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

#include "sphk.h"

namespace sphk {

constexpr int DARCY_BLOCK = 128;
constexpr double D_PI = 3.14159265358979323846;   // M_PI, which src/darcy.cuh uses

// node (x, y, z) with ghost nodes at -1 and num (src/darcy.cuh:125-135)
__host__ __device__ __forceinline__ size_t dnode(uint32_t nx, uint32_t ny, int x, int y, int z)
{
    const size_t nx2 = (size_t)nx + 2, ny2 = (size_t)ny + 2;
    return (size_t)(x + 1) + nx2 * (size_t)(y + 1) + nx2 * ny2 * (size_t)(z + 1);
}

// findPorositiesSphericalDev (src/darcy.cuh:338-477) and
// findDarcyTransmissivitiesDev (src/darcy.cuh:480-538).  The void fraction of
// a sphere of radius min(dx,dy,dz)/2 at the cell centre (measured from the
// origin, as the reference does, not from origo), less the lens-shaped parts
// of the particles of the 27 neighbour cells, which are visited z, y, x
// outermost to innermost and in cell-list order within a cell; clamped to
// [0.1, 0.9].  Its change is zero in the first step.
//
// Most particles of the 27 cells miss the cell sphere.  They are ruled out
// from the float position copy in cell-list order (xs, the one contact
// detection culls with): one 16-byte load at the list position and a few
// float operations.  The cull is conservative: it skips a particle only
// when its float distance exceeds (R + r)(1 + 1e-5) plus a bound on the
// float rounding of the positions (1e-6 of the coordinates' magnitudes), so
// every particle the reference's test (dd < R + r) would take goes through
// the exact FP64 path, in order.
//
// Three warps share 32 nodes, one z-plane of the 27 cells each.  The lanes of
// a warp first collect the particles that pass the cull, each for its node,
// and then evaluate them together, one a lane.  (Evaluated where they are
// found, the ~7 of ~108 that pass come at different places in every lane, and
// the warp ran the FP64 path for nearly every candidate.)  The planes' terms
// meet in shared memory, where one lane a node subtracts them in the
// reference's order.  A lane whose DP_CAP places are full waits until its
// terms have been subtracted and goes on from where it was.  Bound by
// instructions and the latency of the cull's loads at 27 warps an SM: 62,500
// nodes of 250k grains 64.7 -> 42.6 us.
constexpr int DP_CAP = 12;
constexpr int DP_BATCH = 8;   // candidates whose positions are in flight together

// The grid's constants, the same for every node.
struct PoroConsts {
    double dx, dy, dz, R, cell_volume;
};

// Run idx (0..8) of a plane's candidates, in visiting order: for each of its
// three x-rows, the cell through the periodic boundary before it, cells x - 1,
// x, x + 1 as far as they are in the grid (one run of the cell list), and the
// cell through the boundary after it.  Empty where there is none.
__device__ __forceinline__ uint2 poro_run(const Dev &d, const Params &P, int x, int y, int cz,
                                          int idx)
{
    const int nx = (int)P.num[0], ny = (int)P.num[1];
    const int part = idx % 3;
    int cy = y + idx / 3 - 1;
    if ((cy < 0 || cy >= ny) && P.periodic != 1) return make_uint2(0u, 0u);
    if (cy < 0) cy = ny - 1;
    else if (cy >= ny) cy = 0;
    int c0 = max(x - 1, 0), c1 = min(x + 1, nx - 1);
    if (part != 1) {
        if ((P.periodic != 1 && P.periodic != 2) || x != (part == 0 ? 0 : nx - 1)) return make_uint2(0u, 0u);
        c0 = c1 = part == 0 ? nx - 1 : 0;
    }
    const uint32_t row = (uint32_t)cy * (uint32_t)nx + (uint32_t)(nx * ny) * (uint32_t)cz;
    return make_uint2(d.cell_start[row + (uint32_t)c0], d.cell_start[row + (uint32_t)c1 + 1u]);
}
// The periodic shift code of run idx's cells (findDistMod, one wrap an axis).
__device__ __forceinline__ uint32_t poro_code(const Params &P, int y, int idx)
{
    const int part = idx % 3, cy = y + idx / 3 - 1;
    return (part == 0 ? 1u : (part == 2 ? 2u : 0u)) |
           (cy < 0 ? 4u : (cy >= (int)P.num[1] ? 8u : 0u));
}

__global__ void __launch_bounds__(96, 9)
k_darcy_porosity(const __grid_constant__ Dev d, const __grid_constant__ DarcyDev f,
                 const __grid_constant__ PoroConsts G, int A)
{
    constexpr uint32_t FULL = 0xffffffffu;
    __shared__ double term[3][DP_CAP][32];
    __shared__ uint32_t hits[3][DP_CAP][32];
    __shared__ uint16_t expand[3][32 * DP_CAP];   // a warp's hits to evaluate: lane | number << 5
    __shared__ uint2 runs[9][96];        // the plane's runs of each lane
    __shared__ uint8_t cnt[3][32], fin[3][32], curs[32];
    const Params &P = *d.prm;
    const uint32_t nx = P.num[0], ny = P.num[1], nz = P.num[2];
    const uint32_t lane = threadIdx.x & 31u, plane = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    const uint32_t i = blockIdx.x * 32u + lane;
    const bool node = i < nx * ny * nz;
    const uint32_t x = i % nx, y = (i / nx) % ny, z = i / (nx * ny);
    const double dx = G.dx, dy = G.dy, dz = G.dz, R = G.R;
    const d3 X = mk(x * dx + 0.5 * dx, y * dy + 0.5 * dy, z * dz + 0.5 * dz);
    const double4 *__restrict__ xr = d.xr[A];
    const float4 *__restrict__ xs = d.xs[A];
    const float Xx = (float)X.x, Xy = (float)X.y, Xz = (float)X.z;
    const float Rf = (float)R, L0 = (float)P.L[0], L1 = (float)P.L[1];
    const float err = 1e-6f * (2.0f * (fabsf(Xx) + fabsf(Xy) + fabsf(Xz)) + L0 + L1 + (float)P.L[2] + Rf);
    const int cz = (int)z + (int)plane - 1;
    // the bounds of all runs, their loads in flight together
    const bool in = node && cz >= 0 && cz < (int)nz;
    if (in) {
        uint2 b[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) b[q] = poro_run(d, P, (int)x, (int)y, cz, q);
#pragma unroll
        for (int q = 0; q < 9; ++q) runs[q][threadIdx.x] = b[q];
    }
    int idx = in ? 0 : 9;        // the plane's next run
    uint32_t k = 0, end = 0, code = 0;   // next candidate of the present run
    uint32_t n = 0;              // terms in shared memory
    double void_volume = G.cell_volume;   // plane 0's lanes subtract
    uint32_t cur = 0;            // the plane whose terms are subtracted next
    for (;;) {
        // ---- collect up to DP_CAP particles that pass the cull ----
        uint32_t h = n;
        while (h < (uint32_t)DP_CAP) {
            while (k >= end && idx < 9) {
                const uint2 r = runs[idx][threadIdx.x];
                k = r.x;
                end = r.y;
                code = poro_code(P, (int)y, idx);
                ++idx;
            }
            if (k >= end) break;
            const float sx = (code & 1u) ? L0 : ((code & 2u) ? -L0 : 0.0f);
            const float sy = (code & 4u) ? L1 : ((code & 8u) ? -L1 : 0.0f);
            float4 q[DP_BATCH];
#pragma unroll
            for (int j = 0; j < DP_BATCH; ++j) q[j] = __ldg(&xs[min(k + (uint32_t)j, end - 1u)]);
            uint32_t m = 0;
#pragma unroll
            for (int j = 0; j < DP_BATCH; ++j) {
                const float fx = (Xx - q[j].x) + sx, fy = (Xy - q[j].y) + sy, fz = Xz - q[j].z;
                const float thr = __fmaf_rn(Rf + q[j].w, 1.00001f, err);
                if (!(__fmaf_rn(fx, fx, __fmaf_rn(fy, fy, fz * fz)) > thr * thr * 1.00001f)) m |= 1u << j;
            }
            uint32_t next = k + DP_BATCH;
            if (end - k < DP_BATCH) {
                m &= (1u << (end - k)) - 1u;
                next = end;
            }
            for (; m; m &= m - 1u) {
                const uint32_t at = k + (uint32_t)__ffs(m) - 1u;
                if (h == (uint32_t)DP_CAP) { next = at; break; }
                hits[plane][h++][lane] = at | (code << 27);
            }
            k = next;
        }
        __syncwarp();
        // ---- evaluate them, the warp's together ----
        const uint32_t mine = h - n, most = __reduce_max_sync(FULL, mine);
        uint32_t total = 0;
        for (uint32_t q = 0; q < most; ++q) {
            const uint32_t has = __ballot_sync(FULL, mine > q);
            if (mine > q) expand[plane][total + __popc(has & lt)] = (uint16_t)(lane | (q << 5));
            total += __popc(has);
        }
        __syncwarp();
        for (uint32_t base = 0; base < total; base += 32u) {
            const uint32_t e = base + lane;
            const uint32_t w = e < total ? expand[plane][e] : 0u, l = w & 31u;
            const uint32_t at = __shfl_sync(FULL, n, l) + (w >> 5);
            const d3 C = mk(__shfl_sync(FULL, X.x, l), __shfl_sync(FULL, X.y, l), __shfl_sync(FULL, X.z, l));
            if (e >= total) continue;
            const uint32_t v = hits[plane][at][l];
            const double4 p = xr[__ldg(&d.cellorder[v & 0x7ffffffu])];
            const double r = p.w;
            // a shift of zero adds +0.0, as findDistMod's distmod does
            const d3 dist = add(mk(C.x - p.x, C.y - p.y, C.z - p.z), decode_dm(v >> 27, P));
            const double dd = flen(dist);
            // a particle that misses the sphere subtracts nothing: +0.0
            // leaves the void volume as it is
            double t = 0.0;
            if ((R - r) < dd && dd < (R + r))
                t = 1.0 / (12.0 * dd) *
                    (D_PI * (R + r - dd) * (R + r - dd) *
                     (dd * dd + 2.0 * dd * r - 3.0 * r * r + 2.0 * dd * R + 6.0 * r * R -
                      3.0 * R * R));
            if (dd <= R - r) t = 4.0 / 3.0 * D_PI * r * r * r;
            term[plane][at][l] = t;
        }
        n = h;
        cnt[plane][lane] = (uint8_t)n;
        fin[plane][lane] = idx >= 9 && k >= end;
        __syncthreads();
        // ---- subtract, plane by plane ----
        if (plane == 0 && node) {
            while (cur < 3u) {
                const uint32_t m = cnt[cur][lane];
                for (uint32_t e = 0; e < m; ++e) void_volume -= term[cur][e][lane];
                if (!fin[cur][lane]) break;
                ++cur;
            }
            curs[lane] = (uint8_t)cur;
        }
        if (!__syncthreads_or(plane == 0 && node && cur < 3u)) break;
        // the terms of the planes up to `cur` have been subtracted; the
        // finished ones among them are not looked at again
        if (node && plane <= curs[lane]) n = 0u;
        __syncthreads();
    }
    if (plane != 0 || !node) return;
    const size_t me = dnode(nx, ny, (int)x, (int)y, (int)z);
    const double phi_0 = f.phi[me];
    const double phi = fmin(0.9, fmax(0.1, void_volume / G.cell_volume));
    f.phi[me] = phi;
    f.dphi[me] = (*f.first) ? 0.0 : phi - phi_0;
    // Kozeny-Carman conductivity and the transmissivity K * (dx, dy, dz)
    const double rho = 1000.0;
    const double kk = phi * phi * phi / ((1.0 - phi) * (1.0 - phi)) * f.d_factor;
    const double K = kk * rho * -P.g[2] / f.nu;
    f.K[me] = K;
    f.T[3 * me + 0] = K * dx;
    f.T[3 * me + 1] = K * dy;
    f.T[3 * me + 2] = K * dz;
}

// Values of a node that copyDarcyValsDev (src/darcy.cuh:137-166) copies, as
// (array, index within the node's row): first those the step's kernels read
// from ghost nodes, then the rest.
constexpr int GHOST_READ = 5, GHOST_ALL = 16;
__device__ __forceinline__ double *node_value(const DarcyDev &f, int q, size_t node)
{
    switch (q) {
    case 0: return f.H[0] + node;
    case 1: return f.H[1] + node;
    case 2: return f.T + 3 * node;
    case 3: return f.T + 3 * node + 1;
    case 4: return f.T + 3 * node + 2;
    case 5: return f.K + node;
    case 6: return f.Ss + node;
    case 7: return f.W + node;
    case 8: return f.phi + node;
    case 9: return f.dphi + node;
    case 10: case 11: case 12: return f.V + 3 * node + (q - 10);
    default: return f.dH + 3 * node + (q - 13);
    }
}

// setDarcyGhostNodesDev (src/darcy.cuh:169-261): a node on a face of the
// grid is copied onto the ghost node beyond the opposite face.  Edge and
// corner ghosts are never written (nor read).  Face nodes [0, ny nz) are the
// x faces', then [.., + nx nz) the y faces', then [.., + nx ny) the z faces';
// a thread copies value blockIdx.y / 2 of face side blockIdx.y % 2.  Every
// ghost node is written by one thread, and no thread reads a ghost.
//
// The kernels read ghosts of H and T only; the other values of a ghost node
// are the last copy's, so they are copied in the last step of a call alone.
// Bound by the latency of strided rows: one thread for both sides and all 16
// values took 21.7 us at 63 x 63 x 66 nodes, a thread a value 5.7 us.
__global__ void __launch_bounds__(DARCY_BLOCK)
k_darcy_ghosts(const Params *prm, const __grid_constant__ DarcyDev f)
{
    const Params &P = *prm;
    const int nx = (int)P.num[0], ny = (int)P.num[1], nz = (int)P.num[2];
    uint32_t t = blockIdx.x * DARCY_BLOCK + threadIdx.x;
    const int side = (int)(blockIdx.y & 1u), q = (int)(blockIdx.y >> 1);
    const uint32_t nyz = (uint32_t)(ny * nz), nxz = (uint32_t)(nx * nz), nxy = (uint32_t)(nx * ny);
    const uint32_t ux = (uint32_t)nx, uy = (uint32_t)ny;
    size_t from, to;
    if (t < nyz) {
        const int y = (int)(t % uy), z = (int)(t / uy);
        from = dnode(ux, uy, side ? nx - 1 : 0, y, z);
        to = dnode(ux, uy, side ? -1 : nx, y, z);
    } else if ((t -= nyz) < nxz) {
        const int x = (int)(t % ux), z = (int)(t / ux);
        from = dnode(ux, uy, x, side ? ny - 1 : 0, z);
        to = dnode(ux, uy, x, side ? -1 : ny, z);
    } else if ((t -= nxz) < nxy) {
        const int x = (int)(t % ux), y = (int)(t / ux);
        from = dnode(ux, uy, x, y, side ? nz - 1 : 0);
        to = dnode(ux, uy, x, y, side ? -1 : nz);
    } else {
        return;
    }
    *node_value(f, q, to) = *node_value(f, q, from);
}

__device__ __forceinline__ double hmean(double a, double b) { return (2.0 * a * b) / (a + b); }

// explDarcyStepDev (src/darcy.cuh:604-725): explicit finite-difference
// step of the pressure from H into Hn, with harmonic-mean transmissivities
// between nodes and no flux through the z faces
__global__ void __launch_bounds__(DARCY_BLOCK)
k_darcy_explicit(const Params *prm, DarcyDev f, const double *__restrict__ H, double *Hn)
{
    const Params &P = *prm;
    const uint32_t nx = P.num[0], ny = P.num[1], nz = P.num[2];
    const uint32_t i = blockIdx.x * DARCY_BLOCK + threadIdx.x;
    if (i >= nx * ny * nz) return;
    const int x = (int)(i % nx), y = (int)((i / nx) % ny), z = (int)(i / (nx * ny));
    const double dx = P.L[0] / nx, dy = P.L[1] / ny, dz = P.L[2] / nz;
    const double *__restrict__ T = f.T;
    const size_t me = dnode(nx, ny, x, y, z);
    const size_t xn = dnode(nx, ny, x - 1, y, z), xp = dnode(nx, ny, x + 1, y, z);
    const size_t yn = dnode(nx, ny, x, y - 1, z), yp = dnode(nx, ny, x, y + 1, z);
    const size_t zn = dnode(nx, ny, x, y, z - 1), zp = dnode(nx, ny, x, y, z + 1);
    const double Ss = f.Ss[me], Q = f.W[me], dphi = f.dphi[me], Hc = H[me];
    const double TdH_xn = hmean(T[3 * me + 0], T[3 * xn + 0]) * (H[xn] - Hc) / (dx * dx);
    const double TdH_xp = hmean(T[3 * me + 0], T[3 * xp + 0]) * (H[xp] - Hc) / (dx * dx);
    const double TdH_yn = hmean(T[3 * me + 1], T[3 * yn + 1]) * (H[yn] - Hc) / (dy * dy);
    const double TdH_yp = hmean(T[3 * me + 1], T[3 * yp + 1]) * (H[yp] - Hc) / (dy * dy);
    double TdH_zn = hmean(T[3 * me + 2], T[3 * zn + 2]) * (H[zn] - Hc) / (dz * dz);
    double TdH_zp = hmean(T[3 * me + 2], T[3 * zp + 2]) * (H[zp] - Hc) / (dz * dz);
    const double dx_bar = (dx + dy + dz) / 3.0;
    if (z == 0) TdH_zn = 0.0;
    if ((uint32_t)z == nz - 1) TdH_zp = 0.0;
    const double laplacianH = TdH_xn + TdH_xp + TdH_yn + TdH_yp + TdH_zn + TdH_zp;
    const double porevol = -dx_bar * dphi / P.dt;
    const double deltaH = P.dt / (Ss * dx * dy * dz) * (laplacianH + Q + porevol);
    Hn[me] = fmax(0.0, Hc + deltaH);
}

// findDarcyGradientsDev + findDarcyVelocitiesDev (src/darcy.cuh:541-598,
// 728-776): central-difference gradient of the new pressure H (its ghost
// nodes still hold what the ghost copy put there before the step), flux
// -K/nu dH and pore velocity flux / phi
__global__ void __launch_bounds__(DARCY_BLOCK)
k_darcy_grad_vel(const Params *prm, DarcyDev f, const double *__restrict__ H)
{
    const Params &P = *prm;
    const uint32_t nx = P.num[0], ny = P.num[1], nz = P.num[2];
    const uint32_t i = blockIdx.x * DARCY_BLOCK + threadIdx.x;
    if (i >= nx * ny * nz) return;
    if (i == 0) *f.first = 0u;   // the porosity of this step has read it
    const int x = (int)(i % nx), y = (int)((i / nx) % ny), z = (int)(i / (nx * ny));
    const double dx = P.L[0] / nx, dy = P.L[1] / ny, dz = P.L[2] / nz;
    const size_t me = dnode(nx, ny, x, y, z);
    const double gx = (H[dnode(nx, ny, x + 1, y, z)] - H[dnode(nx, ny, x - 1, y, z)]) / (2.0 * dx);
    const double gy = (H[dnode(nx, ny, x, y + 1, z)] - H[dnode(nx, ny, x, y - 1, z)]) / (2.0 * dy);
    const double gz = (H[dnode(nx, ny, x, y, z + 1)] - H[dnode(nx, ny, x, y, z - 1)]) / (2.0 * dz);
    f.dH[3 * me + 0] = gx;
    f.dH[3 * me + 1] = gy;
    f.dH[3 * me + 2] = gz;
    const double nu = f.nu, K = f.K[me], phi = f.phi[me];
    const double qx = -K / nu * gx, qy = -K / nu * gy, qz = -K / nu * gz;
    f.V[3 * me + 0] = qx / phi;
    f.V[3 * me + 1] = qy / phi;
    f.V[3 * me + 2] = qz / phi;
}

// The Darcy block of one step: `a` is the particle buffer of the step's
// start positions, `hs` the pressure buffer they go with, `last` whether the
// step ends a call (the state may be downloaded after it).
void launch_darcy(const Dev &d, const DarcyDev &f, const Params &hp, int a, int hs, int last,
                  cudaStream_t st)
{
    const uint64_t n = (uint64_t)hp.num[0] * hp.num[1] * hp.num[2];
    const uint64_t faces = (uint64_t)hp.num[1] * hp.num[2] + (uint64_t)hp.num[0] * hp.num[2] +
                           (uint64_t)hp.num[0] * hp.num[1];
    PoroConsts G{};
    G.dx = hp.L[0] / hp.num[0];
    G.dy = hp.L[1] / hp.num[1];
    G.dz = hp.L[2] / hp.num[2];
    G.R = std::fmin(G.dx, std::fmin(G.dy, G.dz)) * 0.5;
    G.cell_volume = 4.0 / 3.0 * D_PI * G.R * G.R * G.R;
    k_darcy_porosity<<<div_up(n, 32), 96, 0, st>>>(d, f, G, a);
    k_darcy_ghosts<<<dim3(div_up(faces, DARCY_BLOCK), 2 * (last ? GHOST_ALL : GHOST_READ)), DARCY_BLOCK, 0,
                     st>>>(d.prm, f);
    k_darcy_explicit<<<div_up(n, DARCY_BLOCK), DARCY_BLOCK, 0, st>>>(d.prm, f, f.H[hs], f.H[hs ^ 1]);
    k_darcy_grad_vel<<<div_up(n, DARCY_BLOCK), DARCY_BLOCK, 0, st>>>(d.prm, f, f.H[hs ^ 1]);
}

}  // namespace sphk

// ---- host-side initialisation: DEM::initDarcy (src/darcy.cpp:760-798) ------

namespace {

inline size_t hnode(const sph_config &c, int x, int y, int z)
{
    return sphk::dnode(c.num[0], c.num[1], x, y, z);
}

}  // namespace

extern "C" int sph_darcy_init(const sph_config *cfg, double nu, const double *x,
                              sph_darcy_state *st, double *stability)
{
    if (!cfg || !x || !st || !st->H || !st->phi || !st->dphi || !st->K || !st->T || !st->Ss ||
        !st->W)
        return SPH_ERR_BAD_INPUT;
    // src/darcy.cpp:762-766
    if (!(nu > 0.0)) return SPH_ERR_BAD_INPUT;
    const sph_config &c = *cfg;
    const int nx = (int)c.num[0], ny = (int)c.num[1], nz = (int)c.num[2];
    if (nx <= 0 || ny <= 0 || nz <= 0) return SPH_ERR_BAD_INPUT;
    const double dx = c.L[0] / nx, dy = c.L[1] / ny, dz = c.L[2] / nz;

    // initDarcyVals (src/darcy.cpp:69-104): every node, ghosts included
    for (int ix = -1; ix <= nx; ++ix)
        for (int iy = -1; iy <= ny; ++iy)
            for (int iz = -1; iz <= nz; ++iz) {
                const size_t k = hnode(c, ix, iy, iz);
                st->Ss[k] = 1.0;
                st->W[k] = 0.0;
            }

    // findPorosities / cellPorosity (src/darcy.cpp:600-644): the particles
    // whose centres lie in [x*dx, (x+1)*dx) x ... of a cell, subtracted from
    // its volume one by one in particle order.  The reference loops over all
    // particles per cell; each particle lies in at most one such box (the
    // boxes' bounds are the same products on both sides), so one pass over
    // the particles in order gives every cell the same subtractions.
    const double cell_volume = dx * dy * dz;
    std::vector<double> void_volume((size_t)nx * ny * nz, cell_volume);
    auto box_of = [](double p, double h, int n) {
        // the index b with b*h <= p < (b+1)*h, or -1 when there is none
        if (!(p >= 0.0)) return -1;
        double fb = std::floor(p / h);
        if (fb > (double)n) fb = (double)n;
        int b = (int)fb;
        while (b > 0 && b * h > p) --b;
        while (b < n && (b + 1) * h <= p) ++b;
        return (b < n && b * h <= p && p < (b + 1) * h) ? b : -1;
    };
    for (uint32_t i = 0; i < c.np; ++i) {
        const double *xr = x + 4 * (size_t)i;
        const int bx = box_of(xr[0], dx, nx), by = box_of(xr[1], dy, ny), bz = box_of(xr[2], dz, nz);
        if (bx < 0 || by < 0 || bz < 0) continue;
        double &v = void_volume[(size_t)bx + (size_t)nx * by + (size_t)nx * ny * bz];
        v -= 4.0 / 3.0 * sphk::D_PI * xr[3] * xr[3] * xr[3];
    }
    // meanRadius (src/darcy.cpp:646-653), the sum started from zero, and the
    // host's grain-size factor (src/darcy.cpp:184-187)
    double r_sum = 0.0;
    for (uint32_t i = 0; i < c.np; ++i) r_sum += x[4 * (size_t)i + 3];
    const double r_bar2 = r_sum / (double)c.np * 2.0 * 1.0e-6;
    const double d_factor = r_bar2 * r_bar2 / 180.0;
    // findDarcyTransmissivities (src/darcy.cpp:177-221), dphi := 0
    // (src/darcy.cpp:788-795)
    const double rho = 1000.0;
    for (int ix = 0; ix < nx; ++ix)
        for (int iy = 0; iy < ny; ++iy)
            for (int iz = 0; iz < nz; ++iz) {
                const size_t k = hnode(c, ix, iy, iz);
                const double phi = std::fmin(
                    0.99, std::fmax(0.01, void_volume[(size_t)ix + (size_t)nx * iy +
                                                      (size_t)nx * ny * iz] /
                                              cell_volume));
                st->phi[k] = phi;
                const double kk = phi * phi * phi / ((1.0 - phi) * (1.0 - phi)) * d_factor;
                const double K = kk * rho * -c.g[2] / nu;
                st->K[k] = K;
                st->T[3 * k + 0] = K * dx;
                st->T[3 * k + 1] = K * dy;
                st->T[3 * k + 2] = K * dz;
                st->dphi[k] = 0.0;
            }
    // checkDarcyTimestep (src/darcy.cpp:692-758)
    double T_max = -1.0e13, Ss_min = 1.0e13;
    for (int ix = 0; ix < nx; ++ix)
        for (int iy = 0; iy < ny; ++iy)
            for (int iz = 0; iz < nz; ++iz) {
                const size_t k = hnode(c, ix, iy, iz);
                for (int q = 0; q < 3; ++q)
                    if (st->T[3 * k + q] > T_max) T_max = st->T[3 * k + q];
                if (st->Ss[k] < Ss_min) Ss_min = st->Ss[k];
            }
    const double S_min = Ss_min * dx * dy * dz;
    const double value =
        T_max / S_min * (c.dt / (dx * dx) + c.dt / (dy * dy) + c.dt / (dz * dz));
    if (stability) *stability = value;
    return value > 0.5 ? SPH_ERR_UNSTABLE : SPH_OK;
}
