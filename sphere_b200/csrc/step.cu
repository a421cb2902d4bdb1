// step.cu -- the per-particle DEM step of libsphk: two launches, or one for
// the whole step of a small scene.
//
// k_topo   contact detection into the persistent slots (topology,
//          src/contactsearch.cuh:181-355): a lane's list decisions for one
//          to four particles, then a search for each particle they do not
//          settle.  Candidates come from a float copy of the positions kept
//          in cell-list order (Dev::xs), so the three cells of each x-row of
//          the 27-cell stencil are three adjacent runs of one array and a
//          candidate costs one coalesced 16-byte load; the particle's own slot
//          row is fetched only when an overlap is found.
// k_force_tiles  everything per particle after it (src/device.cu:829-1058):
//          the force laws of the occupied slots (interact's slot loop,
//          src/contactsearch.cuh:468-543), a lane a particle, summed in slot
//          order in registers; the walls (interact,
//          contactsearch.cuh:578-663); the per-bond forces of bondsLinear
//          (cohesion.cuh:8-233, computed by bonds.cu and gathered here in
//          bond order); and the half-step leapfrog (integrate,
//          integration.cuh:9-187).  Warps of a resident grid take tiles of 32
//          particles whose rows arrive by bulk copies.
// k_contact  the slot forces by themselves, where they are timed apart or a
//          block size was asked for; k_force_tiles then reads its sums.
// k_force_diff  the differentiable step's forces and integration.
// k_small  the whole step in one cooperative launch.
// Kinematics of step n are read from buffer A and step n+1 is written to
// buffer B, so neighbours always see start-of-step values.
//
// Parity: every expression keeps the reference's operation order; see
// sphk_internal.cuh.  Candidates are first culled with a conservative FP32
// distance test (Params::cull_eps bounds the float rounding), then the
// reference's own predicate float_sqrt(dot) - (ra + rb) < 0 decides.  The
// visiting order is the reference's: stencil cells z, y, x, members of a cell
// by particle index.
#include <algorithm>

#include "sphk_internal.cuh"
#include "diff_step.cuh"
#include "rebuild.cuh"

namespace sphk {

// Threads per block, and resident blocks per SM that the register
// allocation must allow (the __launch_bounds__ minimum), from sweeps of
// block shapes and caps at 1M spheres.
#ifndef SPHK_FORCE_BLOCK
#define SPHK_FORCE_BLOCK 128
#endif
constexpr int FORCE_BLOCK = SPHK_FORCE_BLOCK;
#ifndef SPHK_FORCE_MIN_BLOCKS
#define SPHK_FORCE_MIN_BLOCKS 6
#endif
// The contact search and the contact forces are compiled in two block
// shapes each, and a context picks one pair (Dev::shape, SPH_OPT_BLOCK_SHAPES;
// the ensemble's autotuner times both).  Shape 0, the default: k_topo in
// blocks of 64 threads, 16 per SM, whose threads leave at different times;
// k_contact in blocks of 4 warps, 4 per SM.  Shape 1: k_topo in 128 x 8,
// k_contact in 2 warps x 8.  The threads resident per SM are the same.
#ifndef SPHK_TOPO_THREADS_PER_SM
#define SPHK_TOPO_THREADS_PER_SM 1024
#endif
constexpr int TOPO_THREADS_PER_SM = SPHK_TOPO_THREADS_PER_SM;
#ifndef SPHK_CONTACT_THREADS_PER_SM
#define SPHK_CONTACT_THREADS_PER_SM 512
#endif
constexpr int CONTACT_THREADS_PER_SM = SPHK_CONTACT_THREADS_PER_SM;
__host__ __device__ constexpr int topo_block(uint32_t shape) { return shape ? 128 : 64; }
__host__ __device__ constexpr int contact_block(uint32_t shape) { return shape ? 64 : 128; }

// What one law adds to a particle's sums.  The laws return their terms by
// value and the caller adds them: each reference update `s += term` is the
// caller's `s + term`, the same operation.  (The wall law is out of line;
// a reference into the caller's sums would put them in local memory for the
// whole kernel.)
struct WallOut {
    d3 f, t;       // F += f, T += t
    double pr;     // p += pr
    double fn;     // the normal force along n (walls_force_pp)
};
struct LawOut {
    d3 f, t;           // F += f, T += t
    double pr, ev;     // p += pr, ev_dot += ev
    double es;         // es_dot += es, where es_set
    bool es_set;
    double4 dt4;       // the slot's new tangential history
};

// contactLinear_wall, src/contactmodels.cuh:10-109.  Inlined into
// wall_forces, its one caller.
__device__ __forceinline__ WallOut contact_wall(const Params &P, double ra, double4 vel_a,
                                             double4 angvel_a, d3 n, double delta, double wvel)
{
    const d3 linvel = xyz(vel_a), angvel = xyz(angvel_a);
    const d3 vel = adds(add(linvel, smul(ra, cross(n, angvel))), wvel);
    const double vel_n = dot(vel, n);
    const d3 vel_t = sub(vel, muls(n, dot(vel, n)));
    const double vel_t_length = flen(vel_t);
    d3 f_n = smul(-P.k_n * delta - P.gamma_wn * vel_n, n);
    if (dot(f_n, n) < 0.0f) f_n = mk(0.0, 0.0, 0.0);
    const double f_n_length = flen(f_n);
    d3 f_t = mk(0.0, 0.0, 0.0);
    const d3 T_res = mk(0.0, 0.0, 0.0);
    if (vel_t_length > 0.f) {
        const double f_t_visc = P.gamma_wt * vel_t_length;
        double f_t_limit;
        if (vel_t_length > 0.001f) f_t_limit = P.mu_wd * f_n_length;
        else f_t_limit = P.mu_ws * f_n_length;
        if (f_t_visc < f_t_limit) f_t = divs(smul(-1.0f * f_t_visc, vel_t), vel_t_length);
        else f_t = divs(smul(-1.0f * f_t_limit, vel_t), vel_t_length);
    }
    WallOut o;
    o.f = add(f_n, f_t);
    o.t = add(smul(-ra, cross(n, f_t)), T_res);
    o.pr = f_n_length / (4.0f * REF_PI * ra * ra);
    o.fn = dot(f_n, n);
    return o;
}

// The walls interact visits, in its order (src/contactsearch.cuh:578-663,
// defaults :416-427): 0 the top wall (dynamic wall 0, else z = L.z), 1 the
// floor at origo.z, then with periodic == 0 the x walls (dynamic walls 1 and
// 2, else x = L.x and x = 0), and with periodic == 0 or 2 the y walls
// (dynamic walls 3 and 4, else y = L.y and y = 0).  Wall k's gap, normal and
// velocity; a dynamic wall replaces the default in order.
template <class PS>
__device__ __forceinline__ double wall_gap(const PS &P, const Walls &W, int k, double4 xa)
{
    auto wpos = [&](int j, double dflt) { return ((uint32_t)j < P.nw) ? W.nx[j].w : dflt; };
    const double ra = xa.w;
    switch (k) {
    case 0: return wpos(0, P.L[2]) - (xa.z + ra);
    case 1: return xa.z - ra - P.origo[2];
    case 2: return wpos(1, P.L[0]) - (xa.x + ra);
    case 3: return xa.x - ra - wpos(2, 0.0);
    case 4: return wpos(3, P.L[1]) - (xa.y + ra);
    default: return xa.y - ra - wpos(4, 0.0);
    }
}

// Bit k: the particle touches wall k (its gap is negative).
template <class PS>
__device__ __forceinline__ uint32_t wall_touch(const PS &P, const Walls &W, double4 xa)
{
    const int nwall = (P.periodic == 0) ? 6 : ((P.periodic == 2) ? 6 : 2);
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        if (k >= nwall || (P.periodic == 2 && (k == 2 || k == 3))) continue;
        if (wall_gap(P, W, k, xa) < 0.0f) m |= 1u << k;
    }
    return m;
}

struct WallSums {
    d3 F, T;
    double p;
    double w0f;   // the normal force of wall 0 (walls_force_pp)
};

// The wall terms of the touched walls, added in interact's order to the slot
// sums (F, T, p).  Out of line: only particles touching a wall call it.
__device__ __noinline__ WallSums wall_forces(const Params &P, const Walls &W, uint32_t touch,
                                             double4 xa, double4 vel_a, double4 angvel_a, d3 F,
                                             d3 T, double p)
{
    WallSums r{F, T, p, 0.0};
    for (int k = 0; k < 6; ++k) {
        if (!((touch >> k) & 1u)) continue;
        const int j = (k == 0) ? 0 : k - 1;    // the dynamic wall that replaces wall k
        const bool dyn = k != 1 && (uint32_t)j < P.nw;
        d3 n;
        switch (k) {
        case 0: n = mk(0.0, 0.0, -1.0); break;
        case 1: n = mk(0.0, 0.0, 1.0); break;
        case 2: n = mk(-1.0, 0.0, 0.0); break;
        case 3: n = mk(1.0, 0.0, 0.0); break;
        case 4: n = mk(0.0, -1.0, 0.0); break;
        default: n = mk(0.0, 1.0, 0.0); break;
        }
        if (dyn) n = xyz(W.nx[j]);
        const double wv = dyn ? W.mvfd[j].y : ((k == 1) ? (double)0.0f : 0.0);
        const WallOut o = contact_wall(P, xa.w, vel_a, angvel_a, n, wall_gap(P, W, k, xa), wv);
        r.F = add(r.F, o.f);
        r.T = add(r.T, o.t);
        r.p += o.pr;
        if (k == 0) r.w0f = o.fn;
    }
    return r;
}

// Whether flen(a) > 0, without the square root.
__device__ __forceinline__ bool has_length(d3 a) { return __double2float_rn(dot(a, a)) > 0.0f; }

// The pressure term of a contact: only a call's last step stores it.
__device__ __forceinline__ double contact_pressure(double f_n_length, double ra)
{
    return f_n_length / (4.0f * REF_PI * ra * ra);
}

// contactLinear, src/contactmodels.cuh:283-493 (contact model 2).
//
// What it does not evaluate: the pressure where it is not stored (want_p), the
// lengths that are only compared with zero, and the capillary force f_c where
// it is a zero vector, which changes no sum (they start at +0) and no length.
// f_c is one where kappa is 0 and its other factors are finite: radii in
// [0, 2^62) and centres apart (n is finite).  k_force_tiles on the jammed 1M
// column 237 -> 218 us, on 64 jammed scenes 109 -> 103; k_small on 500
// colliding grains 24 -> 21.
template <class PR>
__device__ __forceinline__ LawOut contact_linear(const PR &P, double4 vel_a, d3 angvel_a,
                                              double4 vel_b4, double4 angvel_b4, double ra,
                                              double rb, d3 x, double x_length, double delta,
                                              double4 dt4, bool want_p)
{
    LawOut o;
    o.es = 0.0;
    o.es_set = false;
    const double dt = P.dt;
    const d3 vel_b = xyz(vel_b4), angvel_b = xyz(angvel_b4);
    const d3 dt0u = xyz(dt4);
    const bool no_f_c = P.kappa == 0.0 && (uint32_t)__double2hiint(ra) < 0x43d00000u &&
                        (uint32_t)__double2hiint(rb) < 0x43d00000u && __double2hiint(x_length) > 0;
    const d3 n = divs(x, x_length);
    const d3 vel_linear = mk(vel_a.x - vel_b.x, vel_a.y - vel_b.y, vel_a.z - vel_b.z);
    const d3 vel = add(add(vel_linear, smul(ra + delta / 2.0, cross(n, angvel_a))),
                       smul(rb + delta / 2.0, cross(n, angvel_b)));
    const double vel_n = -dot(vel_linear, n);
    const d3 vel_t = sub(vel, muls(n, dot(n, vel)));
    const d3 delta_t0 = sub(dt0u, muls(n, dot(n, dt0u)));
    d3 delta_t = mk(0.0, 0.0, 0.0);   // the reference leaves it unset when unused
    d3 f_n = smul(-P.k_n * delta - P.gamma_n * vel_n, n);
    o.ev = P.gamma_n * vel_n * vel_n;
    if (dot(f_n, n) < 0.0f) f_n = mk(0.0, 0.0, 0.0);
    d3 f_c = mk(0.0, 0.0, 0.0), f_nc = f_n;   // f_n - f_c
    if (!no_f_c) {
        f_c = smul(-P.kappa * fsqrt_of(ra * rb), n);
        f_nc = sub(f_n, f_c);
    }
    d3 f_t = mk(0.0, 0.0, 0.0);
    if (has_length(delta_t0) || has_length(vel_t)) {
        delta_t = add(delta_t0, muls(vel_t, dt));
        const d3 f_t_elast = smul(-P.k_t, delta_t);
        const d3 f_t_visc = smul(-P.gamma_t, vel_t);
        f_t = add(f_t_elast, f_t_visc);
        const double f_t_length = flen(f_t);
        const double f_nc_length = flen(f_nc);
        const double f_t_limit = P.mu_s * f_nc_length;
        if (f_t_length > f_t_limit) {
            const d3 t = divs(f_t, f_t_length);
            f_t = smul(f_t_limit, t);
            delta_t = smul(-1.0 / P.k_t,
                           add(smul(P.mu_d * f_nc_length, t), smul(P.gamma_t, vel_t)));
            o.es = flen(muls(smul(flen(f_t), vel_t), dt)) / dt;
            o.es_set = true;
        }
    }
    o.f = add(f_n, f_t);
    if (!no_f_c) o.f = add(o.f, f_c);
    o.t = cross(smul(-(ra + delta * 0.5), n), f_t);
    o.pr = want_p ? contact_pressure(flen(f_n), ra) : 0.0;
    o.dt4 = make_double4(delta_t.x, delta_t.y, delta_t.z, 0.0f);
    return o;
}

// The FP32 transcendentals of the force laws (expf in capillaryCohesion_exp,
// powf in contactHertz), evaluated as the float nearest to the
// double-precision result.  The reference's GPU build used its fast-math
// intrinsics and its host build the C library's functions; neither is
// correctly rounded, so these are the one place where this path follows
// neither bit for bit (the oracle computes the same nearest float).
__device__ __forceinline__ double f32_expf(double x)
{
    return (double)__double2float_rn(exp((double)__double2float_rn(x)));
}
__device__ __forceinline__ double f32_powf(double x, float y)
{
    return (double)__double2float_rn(pow((double)__double2float_rn(x), (double)y));
}

// contactLinearViscous, src/contactmodels.cuh:114-253 (contact model 1): no
// tangential history, and the torque is left alone (its update is commented
// out in the reference, :244).  Returns the force on a; pr: the pressure.
__device__ __forceinline__ d3 contact_viscous(const Params &P, double &pr, d3 vel_a, d3 vel_b,
                                              d3 angvel_a, d3 angvel_b, double ra, double rb,
                                              d3 x_ab, double x_ab_length, double delta)
{
    const d3 n = divs(x_ab, x_ab_length);
    const d3 vel_linear = mk(vel_a.x - vel_b.x, vel_a.y - vel_b.y, vel_a.z - vel_b.z);
    const d3 vel = add(add(vel_linear, smul(ra + delta / 2.0, cross(n, angvel_a))),
                       smul(rb + delta / 2.0, cross(n, angvel_b)));
    const double vel_n = dot(vel_linear, n);
    const d3 vel_t = sub(vel, muls(n, dot(vel, n)));
    const double vel_t_length = flen(vel_t);
    d3 f_n = smul(-P.k_n * delta - P.gamma_n * vel_n, n);
    if (dot(f_n, n) < 0.0f) f_n = mk(0.0, 0.0, 0.0);
    const double f_n_length = flen(f_n);
    const d3 f_c = smul(-P.kappa * fsqrt_of(ra * rb), n);
    d3 f_t = mk(0.0, 0.0, 0.0);
    if (vel_t_length > 0.0) {
        const double f_t_visc = P.gamma_t * vel_t_length;
        double f_t_limit;
        if (vel_t_length > 0.001f) f_t_limit = P.mu_d * flen(sub(f_n, f_c));
        else f_t_limit = P.mu_s * flen(sub(f_n, f_c));
        if (f_t_visc < f_t_limit) f_t = divs(smul(-f_t_visc, vel_t), vel_t_length);
        else f_t = divs(smul(-f_t_limit, vel_t), vel_t_length);
    }
    pr = f_n_length / (4.0f * REF_PI * ra * ra);
    return add(add(f_n, f_t), f_c);
}

// capillaryCohesion_exp, src/cohesion.cuh:314-350
__device__ __forceinline__ d3 capillary_exp(const Params &P, double ra, double rb, double delta,
                                            d3 x_ab, double x_ab_length)
{
    const d3 n = divs(x_ab, x_ab_length);
    double r;
    if ((ra / rb) > (rb / ra)) r = ra / rb;
    else r = rb / ra;
    const double h = -fsqrt_of(r);
    const double R_har = (2.0f * ra * rb) / (ra + rb);
    const double R_geo = fsqrt_of(ra * rb);
    const double lambda = 0.9f * h * fsqrt_of(P.V_b / R_har);
    return smul(-P.kappa * R_geo * f32_expf(-delta / lambda), n);
}

// contactHertz, src/contactmodels.cuh:499-666 (contact model 3).  As in the
// reference, delta is the (negative) overlap, so its fractional powers are
// NaN and so are the forces of every touching pair.  Inlined into k_contact.
template <class PR>
__device__ __forceinline__ LawOut contact_hertz(const PR &P, double4 vel_a, d3 angvel_a,
                                             double4 vel_b4, double4 angvel_b4, double ra,
                                             double rb, d3 x, double x_length, double delta,
                                             double4 dt4, bool want_p)
{
    LawOut o;
    o.es = 0.0;
    o.es_set = false;
    const double dt = P.dt;
    const d3 vel_b = xyz(vel_b4), angvel_b = xyz(angvel_b4);
    const d3 dt0u = xyz(dt4);
    const d3 n = divs(x, x_length);
    const d3 vel_linear = mk(vel_a.x - vel_b.x, vel_a.y - vel_b.y, vel_a.z - vel_b.z);
    const d3 vel = add(add(vel_linear, smul(ra + delta / 2.0, cross(n, angvel_a))),
                       smul(rb + delta / 2.0, cross(n, angvel_b)));
    const d3 angvel_ab = sub(angvel_a, angvel_b);
    const double angvel_ab_length = flen(angvel_ab);
    const double vel_n = dot(vel_linear, n);
    const d3 vel_t = sub(vel, muls(n, dot(vel, n)));
    const double vel_t_length = flen(vel_t);
    const d3 delta_t0 = sub(dt0u, muls(n, dot(dt0u, n)));
    const double delta_t0_length = flen(delta_t0);
    d3 delta_t = mk(0.0, 0.0, 0.0);   // the reference leaves it unset when unused
    d3 f_n = smul(-P.k_n * f32_powf(delta, 3.0f / 2.0f)
                      - P.gamma_n * f32_powf(delta, 1.0f / 4.0f) * vel_n, n);
    o.ev = P.gamma_n * vel_n * vel_n;
    if (dot(f_n, n) < 0.0f) f_n = mk(0.0, 0.0, 0.0);
    const double f_n_length = flen(f_n);
    const d3 f_c = smul(-P.kappa * fsqrt_of(ra * rb), n);
    d3 f_t = mk(0.0, 0.0, 0.0);
    d3 T_res = mk(0.0, 0.0, 0.0);
    if (delta_t0_length > 0.f || vel_t_length > 0.f) {
        const d3 f_t_elast = smul(-P.k_t * f32_powf(delta, 1.0f / 2.0f), delta_t0);
        const d3 f_t_visc = smul(-P.gamma_t * f32_powf(delta, 1.0f / 4.0f), vel_t);
        double f_t_limit;
        if (vel_t_length > 0.001f) f_t_limit = P.mu_d * flen(sub(f_n, f_c));
        else f_t_limit = P.mu_s * flen(sub(f_n, f_c));
        f_t = add(f_t_elast, f_t_visc);
        const double f_t_length = flen(f_t);
        if (f_t_length > f_t_limit) {
            f_t = muls(f_t, f_t_limit / f_t_length);
            delta_t = divs(add(f_t, smul(P.gamma_t * f32_powf(delta, 1.0f / 4.0f), vel_t)),
                           -P.k_t * f32_powf(delta, 1.0f / 2.0f));
            o.es = flen(sub(delta_t0, delta_t)) * P.k_t / dt;
            o.es_set = true;
        } else {
            delta_t = add(delta_t0, muls(vel_t, dt));
        }
    }
    if (angvel_ab_length > 0.f) {
        T_res = divs(smul(-1.0f * fmin(P.gamma_r * ra * angvel_ab_length,
                                       P.mu_r * ra * f_n_length),
                          angvel_ab),
                     angvel_ab_length);
    }
    o.f = add(add(f_n, f_t), f_c);
    o.t = add(smul(-(ra + delta / 2.0), cross(n, f_t)), T_res);
    o.pr = want_p ? contact_pressure(f_n_length, ra) : 0.0;
    o.dt4 = make_double4(delta_t.x, delta_t.y, delta_t.z, 0.0f);
    return o;
}

__device__ __forceinline__ uint32_t dm_get(unsigned long long lo, unsigned long long hi, int i)
{
    return (uint32_t)((i < 16 ? (lo >> (4 * i)) : (hi >> (4 * (i - 16)))) & 0xFull);
}
__device__ __forceinline__ void dm_set(unsigned long long &lo, unsigned long long &hi, int i,
                                       uint32_t code)
{
    if (i < 16) {
        lo = (lo & ~(0xFull << (4 * i))) | ((unsigned long long)code << (4 * i));
    } else {
        hi = (hi & ~(0xFull << (4 * (i - 16)))) | ((unsigned long long)code << (4 * (i - 16)));
    }
}


// findDistMod for one axis that may be periodic (src/contactsearch.cuh:12-74):
// wraps -1 -> num-1 (shift +L, code bit lo) and num -> 0 (shift -L, bit hi).
// far: a cell beyond the stencil, which only the candidate lists look at.
__device__ __forceinline__ void wrap_axis(int32_t &c, uint32_t num, uint32_t &code,
                                          uint32_t bit_lo, uint32_t bit_hi, bool far)
{
    if (far && c == -2) { c += (int32_t)num; code |= bit_lo; return; }
    if (far && c == (int32_t)num + 1) { c = 1; code |= bit_hi; return; }
    if (c < 0) { c = (int32_t)(num - 1); code |= bit_lo; }
    if ((uint32_t)c == num) { c = 0; code |= bit_hi; }
}
// Whether a stencil cell lies past an axis that is not periodic.
__device__ __forceinline__ bool past_axis(int32_t c, uint32_t num, bool far)
{
    return c < 0 || (uint32_t)c == num || (far && (uint32_t)c > num);
}

// Slot state of one particle during contact detection.
struct TopoSlots {
    uint32_t occ;                    // occupied-slot mask
    uint32_t occ0;                   // the mask before this step's search
    uint32_t err;
    unsigned long long dm_lo, dm_hi; // periodic shift code of each slot
    int nc;                          // contacts found this step
    bool loaded;                     // row copied to shared memory
    bool dirty;                      // row changed
};

// Copies the partners of the particle's occupied slots to shared memory and
// its shift codes to registers (once); the other entries are neither
// searched nor written back.
template <int TB>
__device__ __forceinline__ void topo_load_row(const Dev &d, uint32_t *srow, int tid, uint32_t s,
                                              TopoSlots &ts)
{
    if (ts.loaded) return;
    if (ts.occ) {
        for (uint32_t m = ts.occ; m; m &= m - 1u) {
            const uint32_t i = (uint32_t)(__ffs(m) - 1);
            srow[i * TB + tid] = d.contacts[tile_at(s, i, NC)];
        }
        const ulonglong2 c2 = d.dmc[s];
        ts.dm_lo = c2.x;
        ts.dm_hi = c2.y;
    }
    ts.loaded = true;
}

// The slot of the (loaded) row that candidate t holds, or -1.
template <int TB>
__device__ __forceinline__ int slot_of(const uint32_t *srow, int tid, const TopoSlots &ts, uint32_t t)
{
    for (uint32_t m = ts.occ; m; m &= m - 1) {
        const int i = __ffs(m) - 1;
        if (srow[i * TB + tid] == t) return i;
    }
    return -1;
}

// Overlapping candidate t (storage index) reached through a stencil cell
// with shift `code`: the slot choice.  Returns false once nc > NC, which ends
// the current cell (the reference returns from findContactsInCell).  Kept
// out of line: it runs for the few overlaps of a particle, and inlining it
// would raise the register count of the whole candidate loop.
template <int TB>
__device__ __noinline__ bool topo_insert(const Dev &d, uint32_t *srow, int tid, uint32_t s,
                                         uint32_t t, uint32_t code, TopoSlots &ts)
{
    topo_load_row<TB>(d, srow, tid, s, ts);
    // slot choice, src/contactsearch.cuh:252-271: a slot already holding t
    // wins, else the last empty slot, else position nc
    int cpos = -1;
    for (uint32_t m = ts.occ; m; m &= m - 1) {
        const int i = __ffs(m) - 1;
        if (srow[i * TB + tid] == t) { cpos = i; break; }
    }
    if (cpos >= 0) {
        // already in its slot: the reference writes the slot again, which
        // changes the row only where the partner is now seen through
        // another periodic image
        if (dm_get(ts.dm_lo, ts.dm_hi, cpos) != code) {
            dm_set(ts.dm_lo, ts.dm_hi, cpos, code);
            ts.dirty = true;
        }
    } else {
        const uint32_t empty = ~ts.occ;
        cpos = empty ? 31 - __clz(empty) : ts.nc;
        if (cpos < NC) {
            ts.occ |= 1u << cpos;
            srow[cpos * TB + tid] = t;
            dm_set(ts.dm_lo, ts.dm_hi, cpos, code);
            ts.dirty = true;
        } else {
            ts.err |= ST_NC_OVERFLOW;
        }
    }
    return ++ts.nc <= NC;
}

// The reference's overlap, float_sqrt(dot) - (ra + rb), of candidate row xb
// through a stencil cell with shift `code` (src/contactsearch.cuh:233-248);
// it overlaps where this is below 0.0f.
__device__ __forceinline__ double pair_gap(const Params &P, double4 xb, uint32_t code, double4 xa,
                                           double &len)
{
    const d3 dm = decode_dm(code, P);
    const d3 xab = add(mk(xa.x - xb.x, xa.y - xb.y, xa.z - xb.z), dm);
    len = flen(xab);
    return len - (xa.w + xb.w);
}

// The periodic image through which the candidate at xb of a list entry is seen
// from xa: the entry's, or (with Params::one_image) the nearest, which is the one
// of any near pair, whatever boundaries the two have crossed since.
// one: whether it may have changed since it was recorded.
__device__ __forceinline__ uint32_t list_code(const Params &P, bool one, double4 xa, double4 xb, uint32_t meta)
{
    if (!one) return vl_code(meta);
    const double dx = xa.x - xb.x, hx = 0.5 * P.L[0];
    uint32_t code = dx < -hx ? 1u : (dx > hx ? 2u : 0u);
    if (P.periodic == 1) {
        const double dy = xa.y - xb.y, hy = 0.5 * P.L[1];
        code |= dy < -hy ? 4u : (dy > hy ? 8u : 0u);
    }
    return code;
}

// Contact model 1 processes each candidate as soon as it is found
// (findAndProcessContactsInCell, src/contactsearch.cuh:81-175): overlap ->
// contactLinearViscous, else a gap below db -> capillaryCohesion_exp.  One
// pair's force on s in f (where the return is not 0), and its pressure in pr
// (where the return is 2).
__device__ __forceinline__ int visc_pair(const Dev &d, const Params &P, int A, uint32_t s, uint32_t t,
                                         uint32_t code, d3 &f, double &pr)
{
    const double4 xa = d.xr[A][s], xb = d.xr[A][t];
    const d3 va = xyz(ld4(d.vel[A], s)), vb = xyz(ld4(d.vel[A], t));
    const d3 wa = xyz(ld4(d.angvel[A], s)), wb = xyz(ld4(d.angvel[A], t));
    const d3 dm = decode_dm(code, P);
    const d3 xab = add(mk(xa.x - xb.x, xa.y - xb.y, xa.z - xb.z), dm);
    const double len = flen(xab);
    const double delta = len - (xa.w + xb.w);
    if (delta < 0.0f) {
        f = contact_viscous(P, pr, va, vb, wa, wb, xa.w, xb.w, xab, len, delta);
        return 2;
    }
    if (delta < P.db) {
        f = capillary_exp(P, xa.w, xb.w, delta, xab, len);
        return 1;
    }
    return 0;
}

// The pairs of model 1 that a particle's search found, in visiting order, are
// kept as (storage index | shift code << 27) in its column of shared memory
// (act) and worked on by the whole warp (visc_warp).  A particle with more
// than VISC_CAP of them works them off itself, out of line.
constexpr uint32_t VISC_CAP = 32;
struct ViscAct {
    uint32_t n;      // pairs in the column
    d3 F;            // what has been summed up already
    double p;
};
__device__ __noinline__ void visc_spill(const Dev &d, const Params &P, int A, uint32_t s,
                                        const uint32_t *col, uint32_t stride, ViscAct &v)
{
    for (uint32_t k = 0; k < v.n; ++k) {
        const uint32_t e = col[k * stride];
        d3 f;
        double pr;
        const int does = visc_pair(d, P, A, s, e & 0x7ffffffu, e >> 27, f, pr);
        if (does) v.F = add(v.F, f);
        if (does == 2) v.p += pr;
    }
    v.n = 0u;
}

// A warp's shared memory for the pairs of its lanes' particles.
struct ViscWarp {
    double terms[4][64];          // force terms held, pressure
    uint32_t smask[VISC_CAP];     // the lanes with a k-th pair
    uint32_t hitw[2], touchw[2];  // which held pairs act, overlap
    uint16_t expand[32 * VISC_CAP];
    uint16_t sbase[VISC_CAP];
};

// The pairs of the warp's particles (lane's particle s, its column act),
// evaluated 32 at a time, one a lane, and added up by each particle's own lane
// in visiting order.  All lanes.
__device__ __forceinline__ void visc_warp(const Dev &d, int A, uint32_t s, const uint32_t *act,
                                          uint32_t stride, ViscWarp &vs, ViscAct &v)
{
    constexpr uint32_t FULL = 0xffffffffu;
    const Params &P = *d.prm;
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    const uint32_t total = __reduce_add_sync(FULL, v.n);
    uint32_t most = __reduce_max_sync(FULL, v.n);
    for (uint32_t k = 0, at = 0; k < most; ++k) {
        const uint32_t m = __ballot_sync(FULL, v.n > k);
        if (v.n > k) vs.expand[at + __popc(m & lt)] = (uint16_t)(lane | (k << 5));
        if (lane == 0) {
            vs.sbase[k] = (uint16_t)at;
            vs.smask[k] = m;
        }
        at += __popc(m);
    }
    __syncwarp();
    uint32_t done = 0;   // of this lane's pairs
    for (uint32_t base = 0; base < total; base += 32u) {
        const uint32_t c = base + lane, pb = base - base % 64u;
        const uint32_t x = c < total ? vs.expand[c] : 0u;
        const uint32_t sq = __shfl_sync(FULL, s, x & 31u);
        int does = 0;
        if (c < total) {
            const uint32_t e = act[(x >> 5) * stride + (x & 31u)];
            d3 f;
            double pr = 0.0;
            does = visc_pair(d, P, A, sq, e & 0x7ffffffu, e >> 27, f, pr);
            if (does) {
                const uint32_t k = c - pb;
                vs.terms[0][k] = f.x;
                vs.terms[1][k] = f.y;
                vs.terms[2][k] = f.z;
                vs.terms[3][k] = pr;
            }
        }
        const uint32_t hb = __ballot_sync(FULL, does != 0), tb = __ballot_sync(FULL, does == 2);
        if (lane == 0) {
            vs.hitw[(base - pb) >> 5] = hb;
            vs.touchw[(base - pb) >> 5] = tb;
        }
        const uint32_t pe = min(total, pb + 64u);
        if (base + 32u < pe) continue;
        __syncwarp();
        while (done < v.n) {
            const uint32_t j = vs.sbase[done] + __popc(vs.smask[done] & lt);
            if (j >= pe) break;
            const uint32_t k = j - pb;
            ++done;
            if ((vs.hitw[k >> 5] >> (k & 31u)) & 1u)
                v.F = add(v.F, mk(vs.terms[0][k], vs.terms[1][k], vs.terms[2][k]));
            if ((vs.touchw[k >> 5] >> (k & 31u)) & 1u) v.p += vs.terms[3][k];
        }
        __syncwarp();
    }
}

// A moment on the epoch's clock (Verlet::moved) before which a pair whose
// gap is `gap` now, at moment S, cannot overlap: each of the two moves at
// most as far as the clock advances.  `slack` covers the float roundings of
// this length and of the later one.  Rounded down.
__device__ __forceinline__ float pair_when(float S, double gap, double slack)
{
    const float g = __double2float_rd(gap - slack);
    return g > 0.0f ? __fadd_rd(S, __fmul_rd(0.5f, g)) : S;
}

// The stencil slot (0..26, z y x) through which the search of a particle in
// grid cell gp reaches a candidate at xb through image `code`, or -1 where its
// stencil does not.  The candidate's cell is computed from its start-of-step
// position: in k_small, Dev::cell may be the next step's by now.
__device__ __forceinline__ int stencil_slot(const Params &P, const int32_t gp[3], double4 xb,
                                            uint32_t code)
{
    uint32_t c;
    if (!grid_cell(P, xb.x, xb.y, xb.z, c)) return -1;
    const uint32_t nx = P.num[0], ny = P.num[1];
    int32_t x = (int32_t)(c % nx) - gp[0], y = (int32_t)((c / nx) % ny) - gp[1];
    const int32_t z = (int32_t)(c / (nx * ny)) - gp[2];
    if (code & 1u) x -= (int32_t)nx;
    if (code & 2u) x += (int32_t)nx;
    if (code & 4u) y -= (int32_t)ny;
    if (code & 8u) y += (int32_t)ny;
    if (x < -1 || x > 1 || y < -1 || y > 1 || z < -1 || z > 1) return -1;
    return (z + 1) * 9 + (y + 1) * 3 + (x + 1);
}

// The entry of `set` (a mask over s's candidate list) that the reference's
// search visits first: by stencil cell, then by particle index.  Entries
// outside the stencil are dropped from `set`; returns -1 when none is left.
// `slot`: the stencil slot of the entry.
__device__ __noinline__ int first_visited(const Dev &d, const Params &P, int A, const int32_t gp[3],
                                          uint32_t s, uint32_t &set, int &slot)
{
    int best = -1;
    uint64_t bkey = ~0ull;
    for (uint32_t m = set; m; m &= m - 1u) {
        const int e = __ffs(m) - 1;
        const size_t at = vl_at(s, (uint32_t)e);
        const uint32_t t = d.vl[at];
        const int k = stencil_slot(P, gp, d.xr[A][t], vl_code(d.vl_meta[at]));
        if (k < 0) { set &= ~(1u << e); continue; }
        const uint64_t key = ((uint64_t)k << 32) | d.uid[t];
        if (key < bkey) { bkey = key; best = e; slot = k; }
    }
    if (best >= 0) set &= ~(1u << best);
    return best;
}

// What a sweep found: the particle's next moment, the entries known to hold a
// slot, the entries recorded and whether they are a list.
struct Swept {
    float due;
    uint32_t held, nlist;
    bool listed;
};

// The sweep of particle s in grid cell gp (which need not be in the grid), for
// topo_search: the 27 stencil cells are scanned as in the reference (z, y, x;
// members by particle index) and the list is recorded on the way, together
// with the near candidates two cells away where cells are that small
// (Params::wide), or with `record` not set only searched.  What bounds it is latency, a chain of loads a row and one an
// overlap: an x-row is one run of the cell list (a run a cell: 25 rows took 50
// more), and the overlaps are tested when the sweep is over (where they are found
// they come at different places in every lane).  k_topo sweeping in every step,
// 50,000 grains in contact: 96 us -> 55.
//
// Out of line: few steps sweep, and the decision and the lists' path keep their
// registers (k_topo on 97,778 loose grains 5.9 us inline, 5.7 so; without lists, where
// every particle sweeps, 500,000 grains take 276 us a step inline, 298 so).
template <bool VISC, int TB>
__device__ __noinline__ Swept topo_sweep(const Dev &d, const Params &P, int A, uint32_t s, int tid,
                                         uint32_t *srow, float S, double4 xa, const int32_t gp[3],
                                         bool record, TopoSlots &ts, ViscAct &va)
{
    const double ra = xa.w;
    const double4 *__restrict__ xr = d.xr[A];
    const uint32_t nx = P.num[0], ny = P.num[1], nz = P.num[2];
    const bool gp_in = gp[0] >= 0 && (uint32_t)gp[0] < nx && gp[1] >= 0 && (uint32_t)gp[1] < ny &&
                       gp[2] >= 0 && (uint32_t)gp[2] < nz;
    // one more acting pair of model 1
    auto act_on = [&](uint32_t t, uint32_t code) {
        if (va.n == VISC_CAP) visc_spill(d, P, A, s, srow + tid, TB, va);
        srow[va.n++ * TB + tid] = t | (code << 27);
    };
    uint32_t held = 0;
    float due = 3.0e38f;
    const float4 *xs = d.xs[A];
    const uint32_t k = d.pos[s];
    const float4 xaf = xs[k];
    const float Lf0 = (float)P.L[0], Lf1 = (float)P.L[1];
    const float eps = P.cull_eps;
    const double skin = record ? P.skin : 0.0;
    const float skinf = (float)skin;
    const float extraf = (float)P.reach_extra;
    uint32_t nlist = 0;
    bool list_overflow = false;

    // Cell-level pruning: a stencil cell whose box lies farther from the
    // particle than ra + rmax + skin (plus the float slack of the
    // predicate) holds neither a contact nor a list candidate; skipping
    // it leaves the visiting order of the others unchanged.  Used only
    // while the particle's own cell is inside the grid and every
    // particle sits inside its cell's box (alias_any clear).
    const bool prune = gp_in && (__ldcg(d.alias_any) == 0u);
    // squared distances to the cells one and two away on each axis
    float lo1[3], hi1[3], lo2[3], hi2[3];
    {
        const double xc[3] = {xa.x, xa.y, xa.z};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double lo = xc[q] - (P.origo[q] + (double)gp[q] * P.cellsize[q]);
            const double hi = (P.origo[q] + (double)(gp[q] + 1) * P.cellsize[q]) - xc[q];
            const double l2 = lo + P.cellsize[q], h2 = hi + P.cellsize[q];
            lo1[q] = lo > 0.0 ? (float)(lo * lo) * 0.99999f : 0.0f;
            hi1[q] = hi > 0.0 ? (float)(hi * hi) * 0.99999f : 0.0f;
            lo2[q] = l2 > 0.0 ? (float)(l2 * l2) * 0.99999f : 0.0f;
            hi2[q] = h2 > 0.0 ? (float)(h2 * h2) * 0.99999f : 0.0f;
        }
    }
    auto dist2 = [&](int q, int o) {
        return o == 0 ? 0.0f : (o < 0 ? (o == -1 ? lo1[q] : lo2[q]) : (o == 1 ? hi1[q] : hi2[q]));
    };
    const double extra = VISC ? P.reach_extra : 0.0;
    const float reach = (float)((ra + P.rmax + skin + extra) * (1.0 + 1e-5) + P.prune_pad);
    // (cells two away, which the reference does not visit, are only looked into for
    // the list: their distance counts in any case)
    const float far2 = reach * reach, reach2 = prune ? far2 : 3.0e38f;
    const int R = (P.wide && record) ? 2 : 1;

    // A run of the cell list: cells c0, c0 + 1, ..., through image `code`;
    // [in0, in1) is its part in the stencil, the rest, two cells away, is
    // only recorded.
    struct Run {
        uint32_t beg, end, in0, in1, c0, code;
    };
    // The overlaps of the first VL_CAP near candidates are tested after the
    // sweep, from the list: found here and there in a warp's lanes, each
    // would make the whole warp wait for its two loads and its slot.  (With
    // Params::one_image the list of a particle outside the grid may have to stay.)
    const bool room = gp_in || !P.one_image;
    uint32_t later = 0;
    auto test_later = [&]() {
        for (; later; later &= later - 1u) {
            const uint32_t e = (uint32_t)(__ffs(later) - 1);
            const size_t at = vl_at(s, e);
            const uint32_t t = d.vl[at], code = vl_code(d.vl_meta[at]);
            double ln;
            if (pair_gap(P, xr[t], code, xa, ln) < 0.0f) {
                topo_insert<TB>(d, srow, tid, s, t, code, ts);   // nc <= VL_CAP: no cell ends
                held |= 1u << e;
            } else {
                due = fminf(due, S);
            }
        }
    };

    // A run's candidates, culled four at a time so that their loads are in
    // flight together; hits are handled in list order.
    auto scan_run = [&](const Run &r) {
        const float sx = (r.code & 1u) ? Lf0 : ((r.code & 2u) ? -Lf0 : 0.0f);
        const float sy = (r.code & 4u) ? Lf1 : ((r.code & 8u) ? -Lf1 : 0.0f);
        uint32_t base = r.beg;
        while (base < r.end) {
            const uint32_t last = r.end - 1;
            float4 c[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) c[j] = xs[min(base + (uint32_t)j, last)];
            uint32_t near = 0, hit = 0;
            float gj[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float fx = (xaf.x - c[j].x) + sx;
                const float fy = (xaf.y - c[j].y) + sy;
                const float fz = xaf.z - c[j].z;
                const float d2 = __fmaf_rn(fx, fx, __fmaf_rn(fy, fy, fz * fz));
                const float rsum = VISC ? (xaf.w + c[j].w + extraf) : (xaf.w + c[j].w);
                const float rr = rsum * 1.000004f + eps;
                const float rs = (rsum + skinf) * 1.000004f + eps;
                const uint32_t k2 = base + (uint32_t)j;
                const bool ok = k2 < r.end && k2 != k;
                if (ok && d2 < rs * rs) {
                    near |= 1u << j;
                    // the gap, with the cull's float slack taken against it
                    gj[j] = __fsub_rd(__fmul_rd(__fsqrt_rd(d2), 0.999996f), rr);
                }
                if (ok && k2 >= r.in0 && k2 < r.in1 && d2 < rr * rr) hit |= 1u << j;
            }
            uint32_t next = base + 4;
            while (near) {
                const int j = __ffs(near) - 1;
                near &= near - 1;
                const uint32_t t = d.cellorder[base + (uint32_t)j];
                const float g = j < 2 ? (j == 0 ? gj[0] : gj[1]) : (j == 2 ? gj[2] : gj[3]);
                // when it can overlap (a hit's gap is not positive)
                float w = g > 0.0f ? __fadd_rd(S, __fmul_rd(0.5f, g)) : S;
                if (VISC) {
                    if ((hit >> j) & 1u) {
                        act_on(t, r.code);
                        w = -1.0f;
                    }
                } else if ((hit >> j) & 1u) {
                    if (room && nlist < VL_CAP) {
                        later |= 1u << nlist;
                        w = 3.0e38f;
                    } else {
                        test_later();   // in visiting order
                        double ln;
                        if (pair_gap(P, xr[t], r.code, xa, ln) < 0.0f) {
                            if (!topo_insert<TB>(d, srow, tid, s, t, r.code, ts)) {
                                // nc > NC: skip the rest of this cell; the list
                                // would not describe the skipped part
                                uint32_t e = r.c0 + 1u;
                                while (d.cell_start[e] <= base + (uint32_t)j) ++e;
                                next = d.cell_start[e];
                                near = 0;
                                list_overflow = true;
                            }
                            w = 3.0e38f;
                        }
                    }
                }
                due = fminf(due, w);
                if (room && nlist < VL_CAP) {
                    const size_t at = vl_at(s, nlist);
                    d.vl[at] = t;
                    // a held entry that loses its slot is due at once
                    d.vl_meta[at] = vl_meta_of(r.code, w > 1.0e38f ? S : fmaxf(w, 0.0f));
                    ++nlist;
                } else {
                    list_overflow = true;
                }
            }
            base = next;
        }
    };

    // The cells in visiting order, of each x-row in up to three runs: those
    // through the periodic boundary before it, those in the grid, those
    // through the boundary after it (of a particle outside the grid its
    // three cells one by one, as the reference's stencil names them).
    for (int oz = -R; oz <= R; ++oz) {
        const int32_t cz = (int32_t)((uint32_t)gp[2] + (uint32_t)oz);
        if (past_axis(cz, nz, R == 2)) continue;
        const float dz2 = dist2(2, oz);
        if (dz2 > (oz < -1 || oz > 1 ? far2 : reach2)) continue;
        for (int oy = -R; oy <= R; ++oy) {
            const float dyz2 = dz2 + dist2(1, oy);
            const bool far_row = oz < -1 || oz > 1 || oy < -1 || oy > 1;
            const float most = far_row ? far2 : reach2;
            if (dyz2 > most) continue;
            int32_t cy = (int32_t)((uint32_t)gp[1] + (uint32_t)oy);
            uint32_t ycode = 0;
            if (P.periodic == 1) wrap_axis(cy, ny, ycode, 4u, 8u, R == 2);
            else if (past_axis(cy, ny, R == 2)) continue;
            const uint32_t rowbase = (uint32_t)cy * nx + (nx * ny) * (uint32_t)cz;
            for (int part = 0; part < 3; ++part) {
                int32_t a, b, cx;   // cells gp + a .. gp + b; the first one's x
                Run r;
                r.code = ycode;
                if (gp_in) {
                    const int32_t g = gp[0], n = (int32_t)nx;
                    if (part == 1) {
                        a = max(-R, -g);
                        b = min(R, n - 1 - g);
                    } else {
                        if (P.periodic != 1 && P.periodic != 2) continue;
                        a = part == 0 ? -R : n - g;
                        b = part == 0 ? -g - 1 : R;
                    }
                    if (a == -2 && a <= b && dyz2 + lo2[0] > far2) ++a;
                    if (a == -1 && a <= b && dyz2 + lo1[0] > most) ++a;
                    if (b == 2 && a <= b && dyz2 + hi2[0] > far2) --b;
                    if (b == 1 && a <= b && dyz2 + hi1[0] > most) --b;
                    if (a > b) continue;
                    cx = g + a + (part == 0 ? n : (part == 2 ? -n : 0));
                    if (part != 1) r.code |= part == 0 ? 1u : 2u;
                } else {
                    a = b = part - 1;
                    cx = (int32_t)((uint32_t)gp[0] + (uint32_t)a);
                    if (P.periodic == 1 || P.periodic == 2) wrap_axis(cx, nx, r.code, 1u, 2u, false);
                    else if (past_axis(cx, nx, false)) continue;
                }
                const uint32_t cid = (uint32_t)cx + rowbase;
                if (cid >= P.ncells) { ts.err |= ST_OUT_OF_GRID; continue; }
                r.c0 = cid + P.cell_base;
                const uint32_t *const bounds = d.cell_start + r.c0;
                r.beg = bounds[0];
                r.end = bounds[b - a + 1];
                // the stencil's part: cells max(a, -1) .. min(b, 1)
                r.in0 = a < -1 ? bounds[-1 - a] : r.beg;
                r.in1 = far_row || a > 1 || b < -1 ? r.in0 : (b > 1 ? bounds[2 - a] : r.end);
                scan_run(r);
            }
        }
    }
    if (!VISC) test_later();
    return Swept{due, held, nlist, record && !list_overflow};
}

// The contact search of one particle s that is due (k_topo); sweep: its
// candidate list cannot be used; S: the epoch's clock; step, crossed: as in
// Verlet.
//
// List mode: the list holds every candidate that can overlap while the epoch
// lasts, each with the earliest moment it can (vl_when).  Candidates known to
// hold their slot (Dev::vl_held) need no test: the reference leaves such a
// slot as it is, and a separated one is freed by the force pass.  The others
// that are due are measured, and either overlap or get a new moment.  The
// order of new overlaps is the reference's visiting order, taken from their
// present cells; with one, the usual case, there is no order to find.  The
// reference's count nc matters only once a row can fill up: while the
// occupied slots plus the list length stay within NC none can (`simple`);
// otherwise every overlap is walked in order, as the reference does.
//
// Sweep mode: topo_sweep.
//
// VISC (contact model 1): no slots; every candidate within ra + rb + db acts,
// in visiting order: they are left in `va` and the lane's column of srow.
template <bool VISC, bool BATCH, int TB>
__device__ __forceinline__ void topo_search(const Dev &d, int A, uint32_t s, int tid, uint32_t *srow,
                                            bool sweep, bool crossed, uint32_t step, float S, ViscAct &va)
{
    const Params &P = prm_at<BATCH>(d, s);
    const uint32_t len = d.vl_len[s];
    // After a position left the grid (the step reports SPH_ERR_OUT_OF_GRID)
    // the scene has come apart: saturated cell ids pile its particles into
    // the edge cells, where the stencil sweep grows with the square of their
    // count.  The search stays off until an upload clears the status.  A
    // batch goes on, since its other scenes are still sound.  Tested only
    // here, past the decision, and from the word the last step's end left
    // (k_small's integration may be setting the status already).  The slot
    // mask and the position are loaded with it, so the three wait out one
    // memory latency together.
    const uint32_t occ_in = d.cmask[s];
    const double4 xa = d.xr[A][s];
    uint32_t held = VISC ? 0u : d.vl_held[s];
    const bool one = crossed && P.one_image != 0u;   // else an entry's image is as recorded
    if (!BATCH && __ldcg(&d.vs->came_apart) != 0u) return;
    const double4 *__restrict__ xr = d.xr[A];
    TopoSlots ts{occ_in, occ_in, 0u, 0ull, 0ull, 0, false, false};
    const uint32_t nx = P.num[0], ny = P.num[1], nz = P.num[2];
    int32_t gp[3];
    gp[0] = __double2int_rz(cell_floor(P, 0, xa.x));
    gp[1] = __double2int_rz(cell_floor(P, 1, xa.y));
    gp[2] = __double2int_rz(cell_floor(P, 2, xa.z));
    const bool gp_in = gp[0] >= 0 && (uint32_t)gp[0] < nx && gp[1] >= 0 && (uint32_t)gp[1] < ny &&
                       gp[2] >= 0 && (uint32_t)gp[2] < nz;
    const bool use_lists = P.skin > 0.0 && gp_in;
    // around a particle that is back from outside a periodic boundary every entry
    // is looked at; a list that was recorded while it stood outside is not used
    auto new_list = [&]() { return d.vl_tag[s] == (uint8_t)(step - 1u); };
    if (crossed && __ldcg(&d.vs->look_step) == step && __ldcg(&d.look[d.cell[s]]) == step) {
        held = 0u;
        if (new_list()) sweep = true;
    }
    float due = 3.0e38f;         // the particle's next moment

    if (use_lists && !sweep && len < VL_OVER) {
        const bool simple = VISC || len + (uint32_t)__popc(ts.occ) <= (uint32_t)NC;
        if (!simple) held = 0u;
        const bool rows = !VISC && simple && held == 0u && ts.occ != 0u;
        uint32_t act = 0;   // entries that overlap (or act, model 1)
        // the list is read four entries at a time, so that their loads are
        // in flight together
        uint32_t tv[4], mv[4];
        auto load4 = [&](uint32_t e0) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const size_t at = vl_at(s, min(e0 + (uint32_t)j, (uint32_t)len - 1u));
                tv[j] = d.vl[at];
                mv[j] = d.vl_meta[at];
            }
        };
        if (len) load4(0);   // the first four entries are in flight with the slot row
        if (rows) topo_load_row<TB>(d, srow, tid, s, ts);
        for (uint32_t e0 = 0; e0 < len; e0 += 4) {
            if (e0) load4(e0);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t e = e0 + (uint32_t)j;
                if (e >= len) break;
                if ((held >> e) & 1u) continue;
                const uint32_t t = tv[j];
                if (rows) {
                    const int i = slot_of<TB>(srow, tid, ts, t);
                    if (i >= 0 && dm_get(ts.dm_lo, ts.dm_hi, i) == list_code(P, one, xa, xr[t], mv[j])) {
                        held |= 1u << e;
                        continue;
                    }
                }
                const float w = vl_when(mv[j]);
                // (a pair of model 1 acts in every step, at rest too)
                if (VISC ? !(S >= w) : !(S > w)) { due = fminf(due, w); continue; }
                double ln;
                const double4 xb = xr[t];
                const uint32_t code = list_code(P, one, xa, xb, mv[j]);
                const double gap = pair_gap(P, xb, code, xa, ln);
                if (VISC ? (gap < 0.0f || gap < P.db) : (gap < 0.0f)) {
                    act |= 1u << e;
                    if (code != vl_code(mv[j])) d.vl_meta[vl_at(s, e)] = (mv[j] & ~0xfu) | code;
                } else {
                    const uint32_t meta =
                        vl_meta_of(code, pair_when(S, gap, 1e-6 * ln + (VISC ? P.reach_extra : 0.0)));
                    d.vl_meta[vl_at(s, e)] = meta;
                    due = fminf(due, vl_when(meta));
                }
            }
        }
        if (act) {
            uint32_t left = act;
            int slot = 0, skip_slot = -1;
            if constexpr (VISC) {
                // by stencil cell, then particle index: the keys sorted in the
                // column (slot << 27 | uid, both fit), then the pairs they name
                for (; left; left &= left - 1u) {
                    const size_t at = vl_at(s, (uint32_t)(__ffs(left) - 1));
                    const uint32_t t = d.vl[at];
                    const int k = stencil_slot(P, gp, xr[t], vl_code(d.vl_meta[at]));
                    if (k < 0) continue;   // not in the stencil: not visited
                    const uint32_t key = ((uint32_t)k << 27) | d.uid[t];
                    uint32_t q = va.n++;
                    for (; q > 0u && srow[(q - 1u) * TB + tid] > key; --q)
                        srow[q * TB + tid] = srow[(q - 1u) * TB + tid];
                    srow[q * TB + tid] = key;
                }
                for (uint32_t q = 0; q < va.n; ++q) {
                    const uint32_t key = srow[q * TB + tid], k = key >> 27;
                    const int32_t cx = gp[0] + (int32_t)(k % 3u) - 1, cy = gp[1] + (int32_t)(k / 3u % 3u) - 1;
                    const uint32_t code = (cx < 0 ? 1u : (cx == (int32_t)nx ? 2u : 0u)) |
                                          (cy < 0 ? 4u : (cy == (int32_t)ny ? 8u : 0u));
                    srow[q * TB + tid] = d.sidx[key & 0x7ffffffu] | (code << 27);
                }
                due = -1.0f;
            } else if (simple && (act & (act - 1u)) == 0u) {
                // one new overlap: its slot does not depend on any order
                const size_t at = vl_at(s, (uint32_t)(__ffs(act) - 1));
                const uint32_t t = d.vl[at], code = vl_code(d.vl_meta[at]);
                if (stencil_slot(P, gp, xr[t], code) >= 0) {
                    topo_insert<TB>(d, srow, tid, s, t, code, ts);
                    held |= act;
                } else {
                    due = -1.0f;   // not in the stencil yet: looked at again next step
                }
            } else {
                for (int e; (e = first_visited(d, P, A, gp, s, left, slot)) >= 0;) {
                    const size_t at = vl_at(s, (uint32_t)e);
                    const uint32_t t = d.vl[at], code = vl_code(d.vl_meta[at]);
                    if (slot == skip_slot) continue;   // nc > NC: rest of that cell
                    if (!topo_insert<TB>(d, srow, tid, s, t, code, ts)) skip_slot = slot;
                    held |= 1u << e;
                }
                if ((held & act) != act) due = -1.0f;
            }
        }
        if (!simple) {
            held = 0u;
            due = -1.0f;
        }
    } else {
        // a list that had too many entries is tried again with the cells around
        // or in the next epoch; until then the reference's stencil is enough
        const bool record = use_lists && (sweep || len != VL_OVER);
        const Swept w = topo_sweep<VISC, TB>(d, P, A, s, tid, srow, S, xa, gp, record, ts, va);
        due = w.due;
        held = w.held;
        const bool listed = w.listed;
        if (!listed) {
            // searched again next step, over a cell list of that step.  The list of
            // a particle that stands outside a periodic boundary stays for its
            // return, unless it may miss another one that is back.
            due = -1.0f;
            const bool stays = one && !gp_in && !sweep && !new_list() && __ldcg(&d.vs->dirty_step) != step;
            if (!stays) d.vl_len[s] = gp_in ? VL_OVER : VL_NONE;
            if (P.skin > 0.0 && gp_in) d.vs->want_cells = 1u;   // (outside: particle_tail asks)
        } else {
            d.vl_len[s] = (uint8_t)w.nlist;
            d.vl_tag[s] = (uint8_t)step;
        }
    }

    d.due[s] = due;
    if (!VISC) d.vl_held[s] = held;
    if (ts.dirty) {
        // the search only fills empty slots (and may change a code): the
        // partners of the newly occupied slots are the entries to write;
        // an empty slot's entry is never read
        const uint32_t occ = ts.occ;
        for (uint32_t m = occ & ~ts.occ0; m; m &= m - 1u) {
            const uint32_t i = (uint32_t)(__ffs(m) - 1);
            d.contacts[tile_at(s, i, NC)] = srow[i * TB + tid];
        }
        d.cmask[s] = occ;
        d.dmc[s] = make_ulonglong2(ts.dm_lo, ts.dm_hi);
        if (occ) d.cflag[s >> 5] = 1;
    }
    if (ts.err) atomicOr(d.status, ts.err);
}

// Most particles whose decision each lane of k_topo makes in one go.
constexpr uint32_t TOPO_SPAN_MAX = 4;

// k_topo: the contact search, one warp per span x 32 consecutive storage
// indices (storage order, which relayout keeps close to cell order), span
// <= TOPO_SPAN_MAX.  First every lane decides for its span particles (particle
// base + 32 j + lane), their loads in flight together: a particle is searched
// only when the epoch's clock has passed the moment Dev::due kept for it, the
// earliest at which anything can change for it.  The particles that are due
// are then dealt to the warp's lanes in order, 32 at a time, each searched by
// topo_search.
//
// What bounds it: the latency of the few searches (three dependent L2 round
// trips in a warp with one), not bytes -- the decision reads 4 a particle.
// The lists used to be tied to the cells (a particle that changed cell made
// the 54 cells around it sweep, and the cell list was sorted anew in each
// such step) and tested against the largest displacement in every step.  Per
// step, search + cell list, then and now: 1M loose grains in motion 44 + 60
// -> 12.0 + 0.1 us; 50k in a rapid flow 36 + 25 -> 15.5 + 0.7 us; 64 jammed
// scenes of 330k grains 233 + 62 -> 5.1 + 0.1 us; the 1M jammed column 13.9
// -> 9.5 us.
template <bool VISC, bool BATCH, int TB>
__global__ void __launch_bounds__(TB, TOPO_THREADS_PER_SM / TB)
k_topo(const __grid_constant__ Dev d, int A, uint32_t span)
{
    constexpr uint32_t FULL = 0xffffffffu;
    __shared__ uint32_t srow[NC * TB];
    __shared__ ViscWarp visc[VISC ? TB / 32 : 1];
    const uint32_t np = d.np_all;
    const int tid = threadIdx.x;
    const uint32_t lane = (uint32_t)tid & 31u;
    const uint32_t base = ((blockIdx.x * TB + (uint32_t)tid) >> 5) * (32u * span);
    const Verlet &V = *d.vs;
    const uint32_t step = V.step;
    const bool all = V.all_rebuild != 0u, dirty = V.dirty_step == step, crossed = V.crossed != 0u;
    const bool look = crossed && V.look_step == step;
    const float S = V.moved;
    // bit j: particle base + 32 j + lane is searched / must sweep
    uint32_t need = 0, swp = 0;
#pragma unroll
    for (uint32_t j = 0; j < TOPO_SPAN_MAX; ++j) {
        const uint32_t s = base + 32u * j + lane;
        if (j >= span) break;
        if (s >= np) continue;
        const float due = d.due[s];
        const bool sw = all || (dirty && d.dirty[d.cell[s]] == step);
        if (!sw && !(S > due) && !(look && d.look[d.cell[s]] == step)) {
            if (VISC) d.c1acc[s] = make_double4(0.0, 0.0, 0.0, 0.0);
            continue;
        }
        need |= 1u << j;
        if (sw) swp |= 1u << j;
    }
    // the warp's particles that need the search, in (j, lane) order: the
    // k-th goes to lane k % 32 in round k / 32
    uint32_t m[TOPO_SPAN_MAX], ms[TOPO_SPAN_MAX];
    uint32_t total = 0;
#pragma unroll
    for (uint32_t j = 0; j < TOPO_SPAN_MAX; ++j) {
        // need and swp have no bit j >= span: those masks are zero
        m[j] = __ballot_sync(FULL, (need >> j) & 1u);
        ms[j] = __ballot_sync(FULL, (swp >> j) & 1u);
        total += (uint32_t)__popc(m[j]);
    }
    for (uint32_t k0 = 0; k0 < total; k0 += 32u) {
        const uint32_t k = k0 + lane;
        uint32_t s = 0;
        ViscAct va{0u, mk(0.0, 0.0, 0.0), 0.0};
        if (k < total) {
            uint32_t rem = k, sel = 0, selj = 0, sel_s = 0;
            bool got = false;
#pragma unroll
            for (uint32_t j = 0; j < TOPO_SPAN_MAX; ++j) {
                const uint32_t c = (uint32_t)__popc(m[j]);
                if (!got) {
                    if (rem < c) {
                        sel = m[j];
                        sel_s = ms[j];
                        selj = j;
                        got = true;
                    } else {
                        rem -= c;
                    }
                }
            }
            const uint32_t bit = __fns(sel, 0, (int)rem + 1);
            s = base + 32u * selj + bit;
            topo_search<VISC, BATCH, TB>(d, A, s, tid, srow, (sel_s >> bit) & 1u, crossed, step, S, va);
        }
        if constexpr (VISC) {
            __syncwarp();
            visc_warp(d, A, s, srow + (tid & ~31), TB, visc[tid >> 5], va);
            if (k < total) d.c1acc[s] = make_double4(va.F.x, va.F.y, va.F.z, va.p);
        }
    }
}

struct ForceArgs {
    Dev d;
    int a;              // read buffer (start of step); the kernel writes buffer 1-a
    int write_outputs;  // store force/torque/acc/angacc/edp of this step
    int tape_step;      // differentiable step: tape row to record, or -1
    ForceConsts fc;     // single-scene contexts: the scene's constants
    LawParams lp;
};

// The epoch's clock and the decision for the next step: the lists hold every
// pair that can overlap while 2 moved < skin; otherwise (a clock that is not a
// number included) every particle sweeps and a new epoch starts.  One thread,
// after everything else of the step's force kernel.
__device__ void step_tail(const Dev &d)
{
    const Params &P = *d.prm;
    Verlet &V = *d.vs;
    float moved = __ldcg(&V.moved);
    const float inc = __fmul_ru(__fsqrt_ru(__uint_as_float(atomicExch(&V.inc2_bits, 0u))), 1.00001f);
    if (inc != 0.0f) moved = __fadd_ru(moved, __fadd_ru(inc, 1e-15f));
    const bool restart = P.skin > 0.0 && !(2.02 * (double)moved < 0.999 * P.skin);
    V.all_rebuild = restart ? 1u : 0u;
    V.moved = restart ? 0.0f : moved;
    // a sweep needs the cell list of its own step
    const bool want = atomicExch(&V.want_cells, 0u) != 0u;
    const bool next = atomicExch(&d.rebuild[REBUILD_NEXT], 0u) != 0u;
    d.rebuild[REBUILD_NOW] = (restart || want || next) ? 1u : 0u;
    V.came_apart = *(volatile const uint32_t *)d.status & ST_OUT_OF_GRID;
    V.step = __ldcg(&V.step) + 1u;
}
// Large scenes end a step in a launch of their own: in the force kernel's
// last block it took longer (the fence of every block behind its stores, 4 us
// at 1M against 1.8 for the launch).
__global__ void k_tail(const __grid_constant__ Dev d)
{
    if (threadIdx.x == 0) step_tail(d);
}
void launch_tail(const Dev &d, cudaStream_t st)
{
    k_tail<<<1, 32, 0, st>>>(d);
}

// The last block of a kernel ends the step.  Called by all threads of every
// block.
__device__ __forceinline__ void end_of_step(const Dev &d)
{
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&d.vs->done_blocks, 1u) != gridDim.x - 1u) return;
    __threadfence();
    d.vs->done_blocks = 0u;
    step_tail(d);
}

// Where the force kernels read a particle's own start-of-step rows: global
// memory (GlobalRows) or a tile of rows staged in shared memory (TileRows).
struct GlobalRows {
    const Dev &d;
    int A;
    uint32_t s;
    __device__ double4 xr() const { return d.xr[A][s]; }
    __device__ double4 vel() const { return ld4(d.vel[A], s); }
    __device__ double4 angvel() const { return ld4(d.angvel[A], s); }
    __device__ P3 angpos() const { return d.angpos[s]; }
    __device__ P3 angvel0() const { return d.angvel0[s]; }
    __device__ P3 vel0() const { return d.vel0[s]; }
    __device__ double2 xysum() const { return d.xysum[s]; }
    __device__ uint32_t cell() const { return d.cell[s]; }
    __device__ uint8_t fixed() const { return d.fixed[s]; }
    __device__ uint8_t wtouch() const { return d.wtouch[s]; }
};

// The tiled force kernel: blocks of FORCE_WARPS warps, each with tiles of its
// own, a chunk of 32 particles (one lane each); the per-particle arrays it
// stages are allocated in whole tiles.
constexpr uint32_t FT_TILE = 32;
static_assert(ROW_PAD % FT_TILE == 0, "force tiles are whole chunks of a padded array");
constexpr int FORCE_WARPS = 4;
// Resident blocks per SM: two stages of a warp's tile are 11 KB of shared memory.
#ifndef SPHK_FORCE_TILE_BLOCKS
#define SPHK_FORCE_TILE_BLOCKS 4
#endif

// The start-of-step rows of FT_TILE consecutive particles, each array one
// bulk copy (every member a multiple of 16 bytes).
struct __align__(16) ForceTile {
    double4 xr[FT_TILE];
    P3 vel[FT_TILE], angvel[FT_TILE], angpos[FT_TILE], angvel0[FT_TILE], vel0[FT_TILE];
    double2 xysum[FT_TILE];
    uint32_t cell[FT_TILE];
    uint8_t fixed[FT_TILE], wtouch[FT_TILE];
};
static_assert(sizeof(ForceTile) % 16 == 0 && (FT_TILE % 16) == 0, "bulk copies are multiples of 16 bytes");

struct TileRows {
    const ForceTile &T;
    uint32_t r;
    __device__ double4 xr() const { return T.xr[r]; }
    __device__ double4 vel() const
    {
        const P3 v = T.vel[r];
        return make_double4(v.x, v.y, v.z, 0.0);
    }
    __device__ double4 angvel() const
    {
        const P3 v = T.angvel[r];
        return make_double4(v.x, v.y, v.z, 0.0);
    }
    __device__ P3 angpos() const { return T.angpos[r]; }
    __device__ P3 angvel0() const { return T.angvel0[r]; }
    __device__ P3 vel0() const { return T.vel0[r]; }
    __device__ double2 xysum() const { return T.xysum[r]; }
    __device__ uint32_t cell() const { return T.cell[r]; }
    __device__ uint8_t fixed() const { return T.fixed[r]; }
    __device__ uint8_t wtouch() const { return T.wtouch[r]; }
};

// Whether every component is a zero; whether v is a positive normal number.
__device__ __forceinline__ bool is_zero(d3 a)
{
    return ((__double_as_longlong(a.x) | __double_as_longlong(a.y) | __double_as_longlong(a.z)) << 1) == 0;
}
__device__ __forceinline__ bool positive(double v)
{
    return (uint32_t)__double2hiint(v) - 0x00100000u < 0x7fe00000u;
}

// MODEL: the contact model (1, 2 or 3), a template argument so that each
// model's kernel carries only its own force law.
// DIFF: the differentiable step (contact model 2 in exact FP64 with
// per-particle friction, implicit walls only, no bonds), recording the tape
// row args.tape_step when it is >= 0.  Energy rates and pressure are not
// computed in this variant.
// Everything per particle after the slot sums (F, T, p, ev_dot, es_dot):
// the walls, the bonds, the energy sums, the half-step leapfrog, the
// displacement bound and the cell of the new position.  xa, vel_a and
// angvel_a4 are the particle's start-of-step rows of buffer A, R reads its
// other rows; the new state goes to buffer 1 - A.
// P: the particle's scene constants (Params, or a launch's ForceConsts);
template <bool BATCH, bool DIFF, class Rows, class PS>
__device__ __forceinline__ void particle_tail(const Dev &d, const PS &P, uint32_t s, int A,
                                              int write_outputs, double4 xa,
                                              double4 vel_a, double4 angvel_a4, d3 F, d3 T,
                                              double p, double ev_dot, double es_dot,
                                              const Rows &R)
{
    const int B = 1 - A;
    const double ra = xa.w;
    uint32_t err = 0;
    // ---- walls, src/contactsearch.cuh:578-663 (defaults :416-427) ----------
    double w0f = 0.0;
    if constexpr (DIFF) {
        WallHits wh;
        implicit_walls(P, xa, wh);
        const dl::WallLaw wl{P.k_n, P.gamma_wn, P.gamma_wt, P.mu_ws, P.mu_wd};
        for (int k = 0; k < wh.count; ++k) {
            dl::V3 fw, tw;
            dl::wall_fwd(wl, ra, dl::v3(vel_a.x, vel_a.y, vel_a.z),
                         dl::v3(angvel_a4.x, angvel_a4.y, angvel_a4.z), wh.n[k], wh.delta[k], 0.0,
                         fw, tw);
            F = add(F, mk(fw.x, fw.y, fw.z));
            T = add(T, mk(tw.x, tw.y, tw.z));
        }
    } else {
        // the six wall gaps first, inline; a particle touching no wall
        // (nearly all) takes no call
        const uint32_t touch = wall_touch(P, *d.walls, xa);
        if (touch) {
            const WallSums ws = wall_forces(prm_at<BATCH>(d, s), *d.walls, touch, xa, vel_a,
                                            angvel_a4, F, T, p);
            F = ws.F;
            T = ws.T;
            p = ws.p;
            w0f = ws.w0f;
        }
    }

    // ---- bonds: per-bond contributions in bond order (bondsLinear's serial
    // scatter order, cohesion.cuh:220-226) ------------------------------------
    if (P.nb0 > 0) {
        const uint32_t u = d.uid[s];
        const uint32_t e0 = d.bond_ptr[u], e1 = d.bond_ptr[u + 1];
        for (uint32_t e = e0; e < e1; ++e) {
            const uint32_t ent = d.bond_list[e];
            const uint32_t b = ent >> 1;
            const uint32_t xu = d.bond_xu[b];
            if (xu == 0xffffffffu) continue;
            const double4 f = d.bond_f[b];
            const double4 tj = d.bond_t[b];
            if ((ent & 1u) == 0u) {
                if (xu != u) continue;
                F = mk(F.x + f.x, F.y + f.y, F.z + f.z);
                T = mk(T.x - tj.x, T.y - tj.y, T.z - tj.z);
            } else {
                F = mk(F.x - f.x, F.y - f.y, F.z - f.z);
                T = mk(T.x + tj.x, T.y + tj.y, T.z + tj.z);
            }
        }
    }

    const double dt = P.dt;
    // es += es_dot dt, ev += ev_dot dt; a zero rate adds +0.0, which leaves
    // the sums unchanged unless one is -0.0 (esv_skip clear)
    if (es_dot != 0.0 || ev_dot != 0.0 || !P.esv_skip) {
        const double2 e = d.esv[s];
        d.esv[s] = make_double2(e.x + es_dot * dt, e.y + ev_dot * dt);
    }
    // the outputs of the call's last step, each stored once it is final, so
    // that no sum stays live through the integration for them
    if (write_outputs) {
        d.force[s] = make_double4(F.x, F.y, F.z, 0.0f);
        d.edp[s] = make_double4(es_dot, ev_dot, p, 0.0);
    }
    if (P.nw > 0) {
        const uint8_t touched = R.wtouch();
        if (w0f != 0.0 || touched) {
            const uint32_t u = d.uid[s];
            d.wf_pp[u] = w0f;
            d.wf_flag[u / 256u] = 1;
            d.wtouch[s] = (w0f != 0.0) ? 1 : 0;
        }
    }

    // ---- integrate, src/integration.cuh:9-187 -------------------------------
    // The rotation and the translation are independent; each is finished and
    // stored before the other starts, so fewer values are live at once.
    // Every expression keeps the reference's operands and order; a zero over
    // a positive number is that zero, which a warp of particles without a
    // contact finds without dividing.
    const double radius = xa.w;
    const double m = 4.0 / 3.0 * REF_PI * radius * radius * radius * P.rho;
    const bool fixed = R.fixed() != 0;   // fixvel > 0
    {
        P3 angpos = R.angpos(), angvel0 = R.angvel0();
        const double I = 2.0 / 5.0 * m * radius * radius;
        double4 angacc = make_double4(T.x, T.y, T.z, 0.0);
        if (!(is_zero(T) && positive(I))) {
            angacc.x = T.x * 1.0 / I;
            angacc.y = T.y * 1.0 / I;
            angacc.z = T.z * 1.0 / I;
        }
        if (fixed) angacc = make_double4(0.0f, 0.0f, 0.0f, 0.0f);
        angvel0.x += angacc.x * dt;
        angvel0.y += angacc.y * dt;
        angvel0.z += angacc.z * dt;
        angpos.x += angvel0.x * dt;
        angpos.y += angvel0.y * dt;
        angpos.z += angvel0.z * dt;
        P3 angvel;
        angvel.x = angvel0.x + 0.5 * angacc.x * dt;
        angvel.y = angvel0.y + 0.5 * angacc.y * dt;
        angvel.z = angvel0.z + 0.5 * angacc.z * dt;
        d.angvel[B][s] = angvel;
        d.angvel0[s] = angvel0;
        d.angpos[s] = angpos;
        if (write_outputs) {
            d.torque[s] = make_double4(T.x, T.y, T.z, 0.0f);
            d.angacc[s] = angacc;
        }
    }
    double4 x = xa, vel = vel_a;
    P3 vel0 = R.vel0();
    double4 acc = make_double4(F.x, F.y, F.z, 0.0);
    if (!(is_zero(F) && positive(m))) {
        acc.x = F.x / m;
        acc.y = F.y / m;
        acc.z = F.z / m;
    }
    acc.x += P.g[0];
    acc.y += P.g[1];
    acc.z += P.g[2];
    if (fixed) {
        acc.x = 0.0;
        acc.y = 0.0;
        acc.z -= P.g[2];
    }
    if (write_outputs) d.acc[s] = acc;
    if (P.periodic == 1) {
        if (x.x < P.origo[0]) x.x += P.L[0];
        if (x.x > P.L[0]) x.x -= P.L[0];
        if (x.y < P.origo[1]) x.y += P.L[1];
        if (x.y > P.L[1]) x.y -= P.L[1];
    } else if (P.periodic == 2) {
        if (x.x < P.origo[0]) x.x += P.L[0];
        if (x.x > P.L[0]) x.x -= P.L[0];
    }
    const uint32_t wrapped = (x.x != xa.x ? 1u : 0u) | (x.y != xa.y ? 2u : 0u);   // axes
    vel0.x += acc.x * dt;
    vel0.y += acc.y * dt;
    vel0.z += acc.z * dt;
    x.x += vel0.x * dt;
    x.y += vel0.y * dt;
    x.z += vel0.z * dt;
    vel.x = vel0.x + 0.5 * acc.x * dt;
    vel.y = vel0.y + 0.5 * acc.y * dt;
    vel.z = vel0.z + 0.5 * acc.z * dt;
    double2 xys = make_double2(0.0f, 0.0f);
    xys.x += vel.x * dt;
    xys.y += vel.y * dt;
    {
        const double2 o = R.xysum();
        d.xysum[s] = make_double2(o.x + xys.x, o.y + xys.y);
    }
    d.xr[B][s] = x;
    d.vel[B][s] = p3of(vel);
    d.vel0[s] = vel0;
    // float copy in cell-list order, where every step needs it
    if (P.eager) d.xs[B][d.pos[s]] = make_float4((float)x.x, (float)x.y, (float)x.z, (float)x.w);

    // ---- the largest displacement of the step, squared, rounded up ---------
    Verlet &V = *d.vs;
    if (P.skin > 0.0) {
        const float fx = __double2float_ru(fabs(vel0.x * dt)), fy = __double2float_ru(fabs(vel0.y * dt)),
                    fz = __double2float_ru(fabs(vel0.z * dt));
        const float d2 = __fmaf_ru(fx, fx, __fmaf_ru(fy, fy, __fmul_ru(fz, fz)));
        // one mask for both: a warp that is split here has a publishing lane in
        // each part, whatever joins again between the two
        const uint32_t on = __activemask();
        const uint32_t bits = __reduce_max_sync(on, __float_as_uint(d2) & 0x7fffffffu);
        if ((threadIdx.x & 31u) == (uint32_t)(__ffs(on) - 1) &&
            bits > *(volatile uint32_t *)&V.inc2_bits)
            atomicMax(&V.inc2_bits, bits);
    }

    // ---- cell of the new position, for the next step's cell list -----------
    // a position that is not finite (NaN forces, contact model 3) is
    // outside the grid whatever its float-to-integer conversion gives
    uint32_t c;
    bool out;
    if (!cell_at(P, x.x, x.y, x.z, c, out)) { err |= ST_OUT_OF_GRID; c = d.ncells_all; }
    else c += P.cell_base;
    const uint32_t c_old = R.cell();
    if (out) {
        // outside its cell's box: its own search sweeps, over a fresh list
        // (past the last cell its stencil is empty)
        if (c != d.ncells_all || c != c_old) d.rebuild[REBUILD_NEXT] = 1u;
        d.due[s] = -1.0f;
        // (a store by every such particle holds up the readers of V)
        if (*(volatile uint32_t *)&V.crossed == 0u) V.crossed = 1u;
        d.outside[d.uid[s]] = cell_outside(P, xa.x, xa.y, xa.z) ? 2 : 1;
    }
    // (out through one side and into the next cell on another axis, a particle
    // can come back into the cell that its id aliased)
    if (c != c_old || (wrapped != 0u && c != d.ncells_all)) {
        d.cell[s] = c;
        // A move between neighbouring cells inside the grid leaves every
        // candidate list as it is (the lists are sets of near pairs, ordered
        // by their cells only when needed), and so does one out through a
        // periodic boundary.  One back in by a period has the lists around
        // looked at.  Any other -- or where axes are too short for that -- changes
        // images or what a stencil reaches: the cells around sweep again.
        // While a particle stays outside nobody's list changes: below the grid it
        // is found in the cell next to it all along, above it nowhere near.
        const uint32_t was = outside_axes(P, xa.x, xa.y, xa.z), is = out ? outside_axes(P, x.x, x.y, x.z) : 0u;
        bool hard = !P.set_lists || c == d.ncells_all || c_old == d.ncells_all, look = false;
        if (!hard && (was | is | wrapped)) {
            const uint32_t sides = P.periodic == 1 ? 033u : 011u;   // with one_image
            const bool leaves = P.one_image && !was && !wrapped && (is & ~sides) == 0u;
            const bool stays = was && is && !wrapped && !((was >> 3) && !(is >> 3));
            look = P.one_image && !is && wrapped == ((was | was >> 3) & 7u) && d.outside[d.uid[s]] == 1;
            hard = !look && !leaves && !stays;
        }
        if (!hard && !(was | is)) {
            const uint32_t p = c_old - P.cell_base, q = c - P.cell_base;
            const uint32_t nx = P.num[0], ny = P.num[1];
            const int dx = (int)(q % nx) - (int)(p % nx), dy = (int)(q / nx % ny) - (int)(p / nx % ny),
                      dz = (int)(q / (nx * ny)) - (int)(p / (nx * ny));
            hard = dx < -1 || dx > 1 || dy < -1 || dy > 1 || dz < -1 || dz > 1;
        }
        if (hard || look || P.eager) d.rebuild[REBUILD_NEXT] = 1u;
        if (look) V.crossed = 1u;   // (outside since the upload)
        if ((hard || look) && P.skin > 0.0) {
            const uint32_t m = atomicAdd(&V.nmovers, 1u);
            if (m < MOVER_CAP) d.movers[m] = make_uint2(hard ? c_old : LOOK, c);
            else V.movers_overflow = 1u;
        }
    }
    if (err) atomicOr(d.status, err);
}

// A particle's slot sums.
struct SlotSums {
    d3 F, T;
    double p, ev, es;
};

// interact's slot loop (src/contactsearch.cuh:468-543) for particle s, whose
// occupied slots are occ0: the sums of the laws' terms in slot order, the
// slots' new history, and in occ the slots still held.  A slot whose partner
// no longer overlaps is freed and its history zeroed, as in the reference.
// xa, vel_a and angvel_a are its own rows; want_p: the pressure is stored.
template <int MODEL, class PR>
__device__ __forceinline__ void contact_slots(const Dev &d, int A, const PR &P, uint32_t s,
                                              double4 xa, double4 vel_a, d3 angvel_a,
                                              uint32_t occ0, uint32_t &occ, SlotSums &o,
                                              bool want_p)
{
    const ulonglong2 dmw = d.dmc[s];
    o = SlotSums{mk(0.0, 0.0, 0.0), mk(0.0, 0.0, 0.0), 0.0, 0.0, 0.0};
    occ = occ0;
    // the partner of the next slot, loaded a slot ahead
    uint32_t i = (uint32_t)(__ffs(occ0) - 1);
    uint32_t t = d.contacts[tile_at(s, i, NC)];
    for (uint32_t m = occ0; m;) {
        const size_t e = tile_at(s, i, NC);
        const double4 xb = d.xr[A][t];
        const double4 vel_b = ld4(d.vel[A], t), angvel_b = ld4(d.angvel[A], t);
        const P3 dtp = d.delta_t[e];
        const uint32_t bit = m & (0u - m), slot = i;
        m &= m - 1u;
        if (m) {
            i = (uint32_t)(__ffs(m) - 1);
            t = d.contacts[tile_at(s, i, NC)];
        }
        const double ra = xa.w, rb = xb.w;
        const d3 dm = decode_dm(dm_get(dmw.x, dmw.y, (int)slot), P);
        const d3 xab = mk(xa.x - xb.x + dm.x, xa.y - xb.y + dm.y, xa.z - xb.z + dm.z);
        const double xlen = flen(xab);
        const double delta_n = xlen - (ra + rb);
        if (delta_n < 0.0f) {
            const double4 dt0 = make_double4(dtp.x, dtp.y, dtp.z, 0.0);
            const LawOut l = (MODEL == 2)
                ? contact_linear(P, vel_a, angvel_a, vel_b, angvel_b, ra, rb, xab, xlen, delta_n, dt0,
                                 want_p)
                : contact_hertz(P, vel_a, angvel_a, vel_b, angvel_b, ra, rb, xab, xlen, delta_n, dt0,
                                 want_p);
            d.delta_t[e] = P3{l.dt4.x, l.dt4.y, l.dt4.z};
            o.F = add(o.F, l.f);
            o.T = add(o.T, l.t);
            o.p += l.pr;
            o.ev += l.ev;
            if (l.es_set) o.es += l.es;
        } else {
            // separated: free the slot and zero its history
            d.contacts[e] = d.np_all;
            d.delta_t[e] = P3{0.0, 0.0, 0.0};
            occ &= ~bit;
        }
    }
    if (occ != occ0) {
        d.cmask[s] = occ;
        d.vl_held[s] = 0u;   // a listed candidate left its slot: the next
        d.due[s] = -1.0f;    // search looks at the list
    }
}

// Everything of one particle s after the contact search: its slot sums and
// particle_tail.  The sums are k_topo's for model 1; with SLOTS they are made
// here; otherwise they are k_contact's, in Dev::csum_* for the chunks it
// visited.  f: the chunk flag of s (Dev::cflag[s / 32], read by the caller
// ahead of the rows, the same for the warp); fc, lp: the constants of s's
// scene; occ: with SLOTS, the slots still held.
template <int MODEL, bool BATCH, bool SLOTS, class Rows>
__device__ __forceinline__ void force_row(const ForceArgs &args, const ForceConsts &fc,
                                          const LawParams &lp, uint32_t s, const Rows &R, uint8_t f,
                                          uint32_t &occ)
{
    const Dev &d = args.d;
    const double4 xa = R.xr();
    const double4 vel_a = R.vel();
    const double4 angvel_a4 = R.angvel();
    SlotSums o{mk(0.0, 0.0, 0.0), mk(0.0, 0.0, 0.0), 0.0, 0.0, 0.0};
    if constexpr (MODEL == 1) {
        const double4 c = d.c1acc[s];
        o.F = mk(c.x, c.y, c.z);
        o.p = c.w;
    } else if constexpr (SLOTS) {
        if (f != 0) {
            const uint32_t occ0 = d.cmask[s];
            if (occ0)
                contact_slots<MODEL>(d, args.a, lp, s, xa, vel_a, xyz(angvel_a4), occ0, occ, o,
                                     args.write_outputs != 0);
        }
    } else if (f >= 2 && d.cmask[s] != 0u) {
        // the sums of a particle that still holds a slot (with every slot
        // freed nothing was added: the sums are zero)
        const double4 cf = d.csum_f[s], ct = d.csum_t[s];
        o = SlotSums{mk(cf.x, cf.y, cf.z), mk(ct.x, ct.y, ct.z), cf.w, ct.w, d.csum_es[s]};
    }
    particle_tail<BATCH, false>(d, fc, s, args.a, args.write_outputs, xa, vel_a, angvel_a4, o.F, o.T,
                                o.p, o.ev, o.es, R);
}

// The differentiable step's force kernel: one thread per particle, rows
// read from global memory, its own slot laws (contact model 2 in exact FP64
// with per-particle friction), recording the tape.
__global__ void __launch_bounds__(FORCE_BLOCK, SPHK_FORCE_MIN_BLOCKS)
k_force_diff(ForceArgs args)
{
    const Dev &d = args.d;
    const uint32_t np = d.np_all;
    const uint32_t s = blockIdx.x * FORCE_BLOCK + threadIdx.x;
    if (s >= np) return;
    // The state the integration reads comes after the contact work and
    // after stores the compiler may not move loads across, so each of its
    // loads would wait out a full DRAM latency in turn.  Lane 0 of every
    // warp whose 32 rows all exist asks for the warp's rows of it up front.
    if ((threadIdx.x & 31u) == 0 && s + 32 <= np) {
        bulk_prefetch_l2(d.angpos + s, 32 * sizeof(P3));
        bulk_prefetch_l2(d.angvel0 + s, 32 * sizeof(P3));
        bulk_prefetch_l2(d.vel0 + s, 32 * sizeof(P3));
        bulk_prefetch_l2(d.xysum + s, 32 * sizeof(double2));
        bulk_prefetch_l2(d.cell + s, 32 * sizeof(uint32_t));
        bulk_prefetch_l2(d.fixed + s, 32);
        bulk_prefetch_l2(d.wtouch + s, 32);
    }
    const GlobalRows R{d, args.a, s};
    {
        const Params &P = *d.prm;
        const int A = args.a;
        const double4 xa = d.xr[A][s];
        const double ra = xa.w;
        const double4 vel_a = ld4(d.vel[A], s);
        const double4 angvel_a4 = ld4(d.angvel[A], s);
        d3 F = mk(0.0, 0.0, 0.0), T = mk(0.0, 0.0, 0.0);
        double es_dot = 0.0f, ev_dot = 0.0f, p = 0.0f;
        // ---- interact: occupied slots in slot order ----------------------
        uint32_t occ = d.cmask[s];
        const int j = args.tape_step;
        const size_t row = (j >= 0) ? ((size_t)j * np + s) : 0;
        uint32_t lawmask = 0;
        const ulonglong2 dmw = d.dmc[s];
        const uint32_t occ0 = occ;
        for (uint32_t m = occ0; m; m &= m - 1) {
            const int i = __ffs(m) - 1;
            const size_t at = tile_at(s, (uint32_t)i, NC);
            const uint32_t t = d.contacts[at];
            const d3 dm = decode_dm(dm_get(dmw.x, dmw.y, i), P);
            const double4 xb = d.xr[A][t];
            dl::PairIn in;
            in.xab = dl::v3(xa.x - xb.x + dm.x, xa.y - xb.y + dm.y, xa.z - xb.z + dm.z);
            in.ra = ra;
            in.rb = xb.w;
            if (dl::len(in.xab) - (ra + xb.w) < 0.0) {
                const P3 d0p = d.delta_t[at];
                const double4 vb = ld4(d.vel[A], t), wb = ld4(d.angvel[A], t);
                const double4 d0 = make_double4(d0p.x, d0p.y, d0p.z, 0.0);
                in.va = dl::v3(vel_a.x, vel_a.y, vel_a.z);
                in.vb = dl::v3(vb.x, vb.y, vb.z);
                in.wa = dl::v3(angvel_a4.x, angvel_a4.y, angvel_a4.z);
                in.wb = dl::v3(wb.x, wb.y, wb.z);
                in.d0u = dl::v3(d0.x, d0.y, d0.z);
                const dl::Law law{P.k_n, P.k_t, P.gamma_n, P.gamma_t,
                                  0.5 * (d.mu_p[s] + d.mu_p[t]), P.kappa, P.dt};
                dl::PairOut o;
                dl::pair_fwd(law, in, o);
                F = add(F, mk(o.F.x, o.F.y, o.F.z));
                T = add(T, mk(o.T.x, o.T.y, o.T.z));
                d.delta_t[at] = P3{o.dtn.x, o.dtn.y, o.dtn.z};
                lawmask |= 1u << i;
                if (j >= 0) {
                    const size_t ts = tape_slot_at((uint32_t)j, np, s, (uint32_t)i);
                    d.tp_partner[ts] = t;
                    d.tp_dt0[ts] = d0p;
                }
            } else {
                occ &= ~(1u << i);
                d.contacts[at] = np;
                d.delta_t[at] = P3{0.0, 0.0, 0.0};
            }
        }
        if (occ != occ0) {
            d.cmask[s] = occ;
            d.vl_held[s] = 0u;   // a listed candidate left its slot: the
            d.due[s] = -1.0f;    // next search looks at the list
        }
        if (j >= 0) {
            d.tp_x[row] = xa;
            d.tp_v[row] = make_double4(vel_a.x, vel_a.y, vel_a.z, d.fixed[s] ? 1.0 : 0.0);
            d.tp_w[row] = angvel_a4;
            d.tp_mask[row] = lawmask;
            d.tp_dmc[row] = dmw;
        }
        particle_tail<false, true>(d, P, s, A, args.write_outputs, xa, vel_a, angvel_a4, F,
                                   T, p, ev_dot, es_dot, R);
    }
}

// Asks for the slot rows of chunk t, if it may hold a contact, so that they
// are in L2 when its turn comes: its slot tiles are contiguous, and the top
// PF_SLOTS slots are the ones in use.  Only a whole chunk, so that no request
// passes an array's end.
__device__ __forceinline__ void prefetch_slots(const Dev &d, uint32_t t)
{
    const uint32_t b = t * FT_TILE;
    if (b + FT_TILE > d.np_all || d.cflag[t] == 0) return;
    bulk_prefetch_l2(d.cmask + b, 32 * sizeof(uint32_t));
    bulk_prefetch_l2(d.dmc + b, 32 * sizeof(ulonglong2));
    bulk_prefetch_l2(d.contacts + tile_at(b, NC - PF_SLOTS, NC), PF_SLOTS * 32 * sizeof(uint32_t));
    bulk_prefetch_l2(d.delta_t + tile_at(b, NC - PF_SLOTS, NC), PF_SLOTS * 32 * sizeof(P3));
}

// Issues the bulk copies of tile t's rows into T, completing on `bar`.
__device__ __forceinline__ void stage_force_tile(const Dev &d, int A, uint32_t t, ForceTile &T,
                                                 uint64_t *bar)
{
    const size_t s0 = (size_t)t * FT_TILE;
    mbar_expect_tx(bar, (uint32_t)sizeof(ForceTile));
    bulk_load(T.xr, d.xr[A] + s0, sizeof(T.xr), bar);
    bulk_load(T.vel, d.vel[A] + s0, sizeof(T.vel), bar);
    bulk_load(T.angvel, d.angvel[A] + s0, sizeof(T.angvel), bar);
    bulk_load(T.angpos, d.angpos + s0, sizeof(T.angpos), bar);
    bulk_load(T.angvel0, d.angvel0 + s0, sizeof(T.angvel0), bar);
    bulk_load(T.vel0, d.vel0 + s0, sizeof(T.vel0), bar);
    bulk_load(T.xysum, d.xysum + s0, sizeof(T.xysum), bar);
    bulk_load(T.cell, d.cell + s0, sizeof(T.cell), bar);
    bulk_load(T.fixed, d.fixed + s0, sizeof(T.fixed), bar);
    bulk_load(T.wtouch, d.wtouch + s0, sizeof(T.wtouch), bar);
}

// Calls `run` for the lanes of the (converged) warp with `on` set, the
// constants of their scene in `slot`, the warp's own place in shared memory:
// scene by scene, which is once for nearly every warp (storage is in scene
// order).  `have`: the scene in the slot.  Read through their pointer the
// constants would be loaded again after every store to global memory, which
// might alias them.
template <class Consts, class Fill, class Run>
__device__ __forceinline__ void by_scene(Consts &slot, uint32_t &have, uint32_t inst, bool on,
                                         Fill fill, Run run)
{
    uint32_t left = __ballot_sync(0xffffffffu, on);
    while (left) {
        const uint32_t i = __shfl_sync(0xffffffffu, inst, __ffs(left) - 1);
        const bool mine = on && inst == i;
        if (i != have) {
            __syncwarp();
            if ((threadIdx.x & 31u) == 0) fill(slot, i);
            have = i;
            __syncwarp();
        }
        left &= ~__ballot_sync(0xffffffffu, mine);
        if (mine) run(slot);
        __syncwarp();
    }
}

// Shared-memory stages of k_force_tiles: tiles a warp has in flight.
#ifndef SPHK_FORCE_STAGES
#define SPHK_FORCE_STAGES 2
#endif
constexpr uint32_t FT_STAGES = SPHK_FORCE_STAGES;

// k_force_tiles: force_row over tiles of 32 particles (SLOTS: with the slot
// forces, which the graphs of a step use; profile mode and the second block
// shapes run them as k_contact), a resident grid whose warps each take tiles
// g, g + W, g + 2 W, ... of the W warps.  The particles' own rows (364 of the
// 364 + 172 bytes a particle moves) arrive by bulk copies into a ring of
// FT_STAGES shared-memory stages of the warp: while it integrates one tile,
// the copy engine fetches its next ones, so the bytes in flight do not depend
// on how many threads are resident.  A stage is refilled, FT_STAGES tiles
// ahead, once the warp is past its tile.  The per-particle arrays are
// allocated in whole tiles (ROW_PAD), so every copy is a whole tile.  A copy
// that has not landed after BULK_WAIT_NS stops the warp with ST_TIMEOUT, after
// the copies it issued have landed.
//
// The warps of a block wait for nothing of one another: with tiles of the
// block a chunk with contacts held up the three beside it (64 jammed scenes
// 113 us a step, 109 so; the 1M scenes the same).
template <int MODEL, bool BATCH, bool SLOTS>
__global__ void __launch_bounds__(32 * FORCE_WARPS, SPHK_FORCE_TILE_BLOCKS)
k_force_tiles(const __grid_constant__ ForceArgs args)
{
    struct Scene {
        ForceConsts fc;
        LawParams lp;
    };
    __shared__ ForceTile tiles[FORCE_WARPS][FT_STAGES];
    __shared__ uint64_t full[FORCE_WARPS][FT_STAGES];
    __shared__ Scene scene[BATCH ? FORCE_WARPS : 1];   // a batch's, one a warp
    constexpr uint32_t FULL = 0xffffffffu;
    uint32_t have = 0xffffffffu;
    const Dev &d = args.d;
    const uint32_t np = d.np_all;
    const uint32_t ntiles = (np + FT_TILE - 1) / FT_TILE;
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t first = blockIdx.x * FORCE_WARPS + w, stride = gridDim.x * FORCE_WARPS;
    const int A = args.a;
    if (lane == 0) {
        for (uint32_t k = 0; k < FT_STAGES; ++k) mbar_init(&full[w][k], 1);
        mbar_init_fence();
        // the warp's first FT_STAGES tiles
        for (uint32_t k = 0; k < FT_STAGES; ++k) {
            const uint32_t tk = first + k * stride;
            if (tk >= ntiles) continue;
            stage_force_tile(d, A, tk, tiles[w][k], &full[w][k]);
            if (SLOTS) prefetch_slots(d, tk);
        }
    }
    __syncwarp();
    uint32_t t = first;
    for (uint32_t it = 0; t < ntiles; t += stride, ++it) {
        const uint32_t k = it % FT_STAGES;
        const uint32_t s = t * FT_TILE + lane;
        // the chunk flag comes from global memory: asked for before the wait
        const uint8_t f = MODEL != 1 ? d.cflag[t] : (uint8_t)0;
        const bool ready = mbar_wait(&full[w][k], (it / FT_STAGES) & 1u, BULK_WAIT_NS);
        if (!__all_sync(FULL, ready)) {
            if (lane == 0) {
                atomicOr(d.status, ST_TIMEOUT);
                // this tile's copies and those issued for the next ones land
                // before the warp leaves
                for (uint32_t q = 0; q < FT_STAGES; ++q) {
                    const uint32_t iq = it + q;
                    if (t + q * stride < ntiles)
                        mbar_wait(&full[w][iq % FT_STAGES], (iq / FT_STAGES) & 1u, BULK_WAIT_NS);
                }
            }
            return;
        }
        uint32_t occ = 0u;   // slots that the particle still holds
        if constexpr (BATCH) {
            const uint32_t inst = s < np ? d.inst[s] : 0u;
            by_scene(scene[w], have, inst, s < np,
                     [&](Scene &c, uint32_t i) { c = Scene{force_consts(d.prm[i]), law_params(d.prm[i])}; },
                     [&](const Scene &c) {
                         force_row<MODEL, true, SLOTS>(args, c.fc, c.lp, s, TileRows{tiles[w][k], lane}, f, occ);
                     });
        } else if (s < np) {
            force_row<MODEL, false, SLOTS>(args, args.fc, args.lp, s, TileRows{tiles[w][k], lane}, f, occ);
        }
        // the chunk's flag for the next step's search: 1 while it holds a
        // contact (k_contact left 2 for that, 3 for none)
        if (MODEL != 1 && f >= (SLOTS ? 1 : 2)) {
            const bool held = SLOTS ? __any_sync(FULL, occ != 0u) : f == 2;
            if (lane == 0) d.cflag[t] = held ? 1 : 0;
        }
        // every lane is past its reads of stage k: it takes the tile
        // FT_STAGES rounds ahead
        __syncwarp();
        const uint32_t tn = t + FT_STAGES * stride;
        if (lane == 0 && tn < ntiles) {
            fence_proxy_async_smem();
            stage_force_tile(d, A, tn, tiles[w][k], &full[w][k]);
            if (SLOTS) prefetch_slots(d, tn);
        }
    }
}

struct ContactArgs {
    Dev d;
    int a;               // read buffer (start of step)
    int write_outputs;   // the pressure is read after this step
    LawParams lp;        // single-scene contexts; a batch reads each scene's Params
};

// k_contact: the slot forces of contact models 2 and 3.
//
// The unit of work is a chunk of 32 consecutive storage indices, a lane a
// particle, and a chunk is visited only while its flag (Dev::cflag) says it
// may hold a contact: the contact search sets the flag when it writes a row
// with an occupied slot, and this kernel clears it when the chunk ends without
// one.  The grid is resident (a few blocks per SM); warp g takes chunks g,
// g + W, g + 2W, ... of the W warps, reading the flags of 32 of them in one
// load, so a contact-free scene costs about one memory latency.  A chunk's
// rows are contiguous, its slot tiles too, and its lanes mostly walk the same
// slots, so their loads coalesce.
//
// What bounds it: the laws' FP64 chains at 16 warps an SM and L1, 54 B of
// history and 80 B of the partner's rows a contact.  A lane a contact, which
// kept every lane busy whatever the spread of contact counts, loaded the
// particle's own rows again for each of its contacts and passed nine terms
// through shared memory (L1 79% busy): the jammed 1M column 189 -> 166 us.
template <int MODEL, bool BATCH, int CB>
__global__ void __launch_bounds__(CB, CONTACT_THREADS_PER_SM / CB)
k_contact(ContactArgs args)
{
    constexpr uint32_t FULL = 0xffffffffu;
    constexpr int WARPS = CB / 32;
    __shared__ LawParams law[BATCH ? WARPS : 1];   // a batch's scene, one a warp
    uint32_t have = 0xffffffffu;
    const Dev &d = args.d;
    const int A = args.a;
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t np = d.np_all;
    const uint32_t nchunk = (np + 31u) >> 5;
    const uint32_t gw = blockIdx.x * WARPS + w, nwarps = gridDim.x * WARPS;
    // A chunk's rows are contiguous (its slot tiles too), so one lane asks
    // the copy engine to bring a chunk that is coming up into L2 while the
    // warp works: the chain of loads of each round then waits on L2, not on
    // DRAM.  Only whole chunks, so that no request passes an array's end.
    auto prefetch_chunk = [&](uint32_t ch) {
        const uint32_t b = ch << 5;
        if (lane != 0 || b + 32u > np) return;
        bulk_prefetch_l2(d.cmask + b, 32 * sizeof(uint32_t));
        bulk_prefetch_l2(d.dmc + b, 32 * sizeof(ulonglong2));
        bulk_prefetch_l2(d.xr[A] + b, 32 * sizeof(double4));
        bulk_prefetch_l2(d.vel[A] + b, 32 * sizeof(P3));
        bulk_prefetch_l2(d.angvel[A] + b, 32 * sizeof(P3));
        bulk_prefetch_l2(d.contacts + tile_at(b, NC - PF_SLOTS, NC), PF_SLOTS * 32 * sizeof(uint32_t));
        bulk_prefetch_l2(d.delta_t + tile_at(b, NC - PF_SLOTS, NC), PF_SLOTS * 32 * sizeof(P3));
    };

    for (uint32_t g = gw; g < nchunk; g += 32u * nwarps) {
        // the flags of this warp's next 32 chunks: g, g + W, ..., one a lane
        const uint32_t mine = g + lane * nwarps;
        uint32_t todo = __ballot_sync(FULL, mine < nchunk && d.cflag[mine] != 0);
        if (todo) prefetch_chunk(g + (uint32_t)(__ffs(todo) - 1) * nwarps);
        while (todo) {
            const uint32_t chunk = g + (uint32_t)(__ffs(todo) - 1) * nwarps;
            todo &= todo - 1u;
            if (todo) prefetch_chunk(g + (uint32_t)(__ffs(todo) - 1) * nwarps);
            const uint32_t s0 = chunk << 5;
            const uint32_t s = s0 + lane;
            const uint32_t occ0 = (s < np) ? d.cmask[s] : 0u;
            uint32_t occ = 0u;
            auto slots = [&](const auto &P) {
                SlotSums o;
                contact_slots<MODEL>(d, A, P, s, d.xr[A][s], ld4(d.vel[A], s), xyz(ld4(d.angvel[A], s)),
                                     occ0, occ, o, args.write_outputs != 0);
                d.csum_f[s] = make_double4(o.F.x, o.F.y, o.F.z, o.p);
                d.csum_t[s] = make_double4(o.T.x, o.T.y, o.T.z, o.ev);
                d.csum_es[s] = o.es;
            };
            if constexpr (BATCH) {
                by_scene(law[w], have, s < np ? d.inst[s] : 0u, occ0 != 0u,
                         [&](LawParams &l, uint32_t i) { l = law_params(d.prm[i]); }, slots);
            } else if (occ0) {
                slots(args.lp);
            }
            const bool held = __any_sync(FULL, occ != 0u);
            // visited (2: a slot is still held, 3: none is); k_force_tiles reads
            // the sums of a visited chunk and sets its flag back to 1 or 0
            // for the next step's search
            if (lane == 0) d.cflag[chunk] = held ? 2 : 3;
        }
    }
}

// A particle's rows, loaded together.
struct RegRows {
    double4 x;
    P3 v, w, ap, w0, v0;
    double2 xy;
    uint32_t c;
    uint8_t fx, wt;
    __device__ RegRows(const Dev &d, int A, uint32_t s)
        : x(d.xr[A][s]), v(d.vel[A][s]), w(d.angvel[A][s]), ap(d.angpos[s]), w0(d.angvel0[s]),
          v0(d.vel0[s]), xy(d.xysum[s]), c(d.cell[s]), fx(d.fixed[s]), wt(d.wtouch[s])
    {
    }
    __device__ P3 angpos() const { return ap; }
    __device__ P3 angvel0() const { return w0; }
    __device__ P3 vel0() const { return v0; }
    __device__ double2 xysum() const { return xy; }
    __device__ uint32_t cell() const { return c; }
    __device__ uint8_t fixed() const { return fx; }
    __device__ uint8_t wtouch() const { return wt; }
};

// k_small: the step of a scene small enough that every chunk of 32 particles
// has a warp of its own on the device at once.  A particle's search, contact
// forces and integration need its neighbours' start-of-step rows (buffer A)
// and its own results only, so the warp of a chunk runs all three, and the
// step is one launch: the slot sums stay in registers, the last block ends
// the step.
//
// What bounds it: latency, one chain of the search, the laws' rounds and the
// integration.  As three kernels each of their launches, ramps and drains
// stood in that chain: whole runs of 500 grains 7.05 -> 6.45 ms (200 steps), of
// 10,000 10.8 -> 8.4 ms (500 steps).
//
// Blocks of 128 threads: with 64, twice as many meet at the barriers of a cell
// list (50,000 grains in a flow 37.4 us a step, 36.1 with 128).
constexpr int SMALL_BLOCK = 128, SMALL_BLOCKS_PER_SM = 4;
template <int MODEL, bool BATCH>
__global__ void __launch_bounds__(SMALL_BLOCK, SMALL_BLOCKS_PER_SM)
k_small(const __grid_constant__ ForceArgs args, int own_list)
{
    constexpr uint32_t FULL = 0xffffffffu;
    constexpr int WARPS = SMALL_BLOCK / 32;
    constexpr bool VISC = MODEL == 1;
    __shared__ uint32_t srow[WARPS][NC * 32];   // the search's slot rows; model 1's acting pairs
    __shared__ ViscWarp visc[VISC ? WARPS : 1];
    __shared__ LawParams law[BATCH ? WARPS : 1];
    __shared__ ForceConsts scene[BATCH ? WARPS : 1];
    const Dev &d = args.d;
    const int A = args.a;
    const uint32_t np = d.np_all, lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t chunk = blockIdx.x * WARPS + w, s0 = chunk * 32u, s = s0 + lane;
    // the cell list first, where this step needs it (REBUILD_NOW does not
    // change before the step ends)
    if (own_list && *(volatile const uint32_t *)&d.rebuild[REBUILD_NOW] != 0u) {
        if (lists_given_up(d)) return;
        GridBar bar{&d.vs->bar_small, 0};
        if (!rebuild_grid<SMALL_BLOCK>(d, A, bar) || !grid_barrier(d, bar)) return;
    }
    if (s0 < np) {
        ViscAct va{0u, mk(0.0, 0.0, 0.0), 0.0};   // model 1's sums
        // ---- the search (k_topo) ----
        {
            // past L1: the rebuild above may have changed them
            const Verlet &V = *d.vs;
            const uint32_t step = __ldcg(&V.step);
            const float S = __ldcg(&V.moved);
            const bool crossed = __ldcg(&V.crossed) != 0u;
            const bool look = crossed && __ldcg(&V.look_step) == step;
            bool need = false, sweep = false;
            if (s < np) {
                sweep = __ldcg(&V.all_rebuild) != 0u ||
                        (__ldcg(&V.dirty_step) == step && __ldcg(&d.dirty[d.cell[s]]) == step);
                need = sweep || S > d.due[s] || (look && __ldcg(&d.look[d.cell[s]]) == step);
            }
            if (need) topo_search<VISC, BATCH, 32>(d, A, s, (int)lane, srow[w], sweep, crossed, step, S, va);
            __syncwarp();
            if constexpr (VISC) visc_warp(d, A, s, srow[w], 32u, visc[w], va);
        }
        // ---- the slot forces (k_contact) ----
        const uint32_t inst = (BATCH && s < np) ? d.inst[s] : 0u;
        uint32_t have = 0xffffffffu, occ = 0u;
        SlotSums o{mk(0.0, 0.0, 0.0), mk(0.0, 0.0, 0.0), 0.0, 0.0, 0.0};
        if constexpr (!VISC) {
            if (d.cflag[chunk] != 0) {
                const uint32_t occ0 = (s < np) ? d.cmask[s] : 0u;
                auto slots = [&](const auto &P) {
                    contact_slots<MODEL>(d, A, P, s, d.xr[A][s], ld4(d.vel[A], s),
                                         xyz(ld4(d.angvel[A], s)), occ0, occ, o,
                                         args.write_outputs != 0);
                };
                if constexpr (BATCH) {
                    by_scene(law[w], have, inst, occ0 != 0u,
                             [&](LawParams &l, uint32_t i) { l = law_params(d.prm[i]); }, slots);
                } else if (occ0) {
                    slots(args.lp);
                }
                const bool held = __any_sync(FULL, occ != 0u);
                if (lane == 0) d.cflag[chunk] = held ? 1 : 0;
            }
        }
        // ---- the rest of the step (k_force_tiles) ----
        auto integrate = [&](const ForceConsts &fc) {
            const RegRows R(d, A, s);
            d3 F = mk(0.0, 0.0, 0.0), T = mk(0.0, 0.0, 0.0);
            double es_dot = 0.0f, ev_dot = 0.0f, p = 0.0f;
            if constexpr (VISC) {
                F = va.F;
                p = va.p;
            } else if (occ != 0u) {
                F = o.F;
                T = o.T;
                p = o.p;
                ev_dot = o.ev;
                es_dot = o.es;
            }
            particle_tail<BATCH, false>(d, fc, s, A, args.write_outputs, R.x,
                                        make_double4(R.v.x, R.v.y, R.v.z, 0.0),
                                        make_double4(R.w.x, R.w.y, R.w.z, 0.0), F, T, p, ev_dot,
                                        es_dot, R);
        };
        if constexpr (BATCH) {
            have = 0xffffffffu;
            by_scene(scene[w], have, inst, s < np,
                     [&](ForceConsts &c, uint32_t i) { c = force_consts(d.prm[i]); }, integrate);
        } else if (s < np) {
            integrate(args.fc);
        }
    }
    end_of_step(d);
}

// Blocks of k_small that the device holds at once.
template <int MODEL, bool BATCH>
static uint32_t small_blocks()
{
    return std::min(resident_blocks<k_small<MODEL, BATCH>, SMALL_BLOCK>(), sm_count() * SMALL_BLOCKS_PER_SM);
}
static uint32_t small_blocks(const Dev &d, int model)
{
    if (d.inst) return small_blocks<2, true>();
    return model == 1 ? small_blocks<1, false>()
                      : (model == 3 ? small_blocks<3, false>() : small_blocks<2, false>());
}

// Whether a context's steps run as k_small: its chunks have a resident warp
// each (75,776 particles on 148 SMs), and no shape or span of the split
// kernels was asked for.  Above, the split kernels balance the work over the
// device and stream the integration.  Microseconds a step, one kernel against
// split, on a B200: in a flow 20.0 / 24.0 at 1,000 grains, 25.3 / 30.7 at
// 10,000, 30.3 / 36.0 at 50,000, 36.0 / 42.0 at 75,000; in a jammed packing
// 20.9 / 20.7 at 1,000, 22.8 / 23.2 at 29,791, 28.8 / 27.0 at 74,088.
//
// Beside a Darcy flow (with_flow) up to a block an SM: its blocks start all
// together, so beyond that k_small waits for the porosity's to leave, which runs
// at the same time.  One kernel against split, cells of 2.5 and 4 radii: 42.9 /
// 47.0 and 60.6 / 60.9 at 10,000 grains, 66.0 / 54.1 and 108.8 / 69.0 at 20,000,
// 69.5 / 60.5 and 113.0 / 73.1 at 50,000.
bool small_step(const Dev &d, uint32_t np, int model, bool with_flow)
{
    const uint32_t blocks = div_up(np, SMALL_BLOCK);
    return d.shape == 0 && d.topo_span == 0 && blocks <= small_blocks(d, model) &&
           !(with_flow && blocks > sm_count());
}

// own_list: the kernel makes the cell list itself when it is due.
cudaError_t launch_small(const Dev &d, const Params &hp, uint32_t np, int model, int a, int write_outputs,
                         bool own_list, cudaStream_t st)
{
    const ForceArgs args{d, a, write_outputs, -1, force_consts(hp), law_params(hp)};
    // more blocks than chunks need where the cells are many: they share the list
    const unsigned grid = std::min(small_blocks(d, model),
                                   std::max(div_up(np, SMALL_BLOCK), div_up(d.ncells_all, 32 * SMALL_BLOCK)));
    const int own = own_list ? 1 : 0;
    if (d.inst) return launch_together(k_small<2, true>, grid, SMALL_BLOCK, st, args, own);
    if (model == 1) return launch_together(k_small<1, false>, grid, SMALL_BLOCK, st, args, own);
    if (model == 3) return launch_together(k_small<3, false>, grid, SMALL_BLOCK, st, args, own);
    return launch_together(k_small<2, false>, grid, SMALL_BLOCK, st, args, own);
}

// A resident grid of k_contact: the blocks of this instantiation that the
// device holds at once.
template <int MODEL, bool BATCH, int CB>
static unsigned contact_grid(uint32_t np)
{
    const uint64_t chunks = div_up(np, 32);
    return (unsigned)std::min<uint64_t>(resident_blocks<k_contact<MODEL, BATCH, CB>, CB>(), div_up(chunks, CB / 32));
}

// Particles per lane of k_topo's list decisions: 4 once the scene is four
// times the threads the device holds at once (one decision round then
// hides the latency of four), 2 from twice, else 1, so that a smaller
// scene's searches run on as many lanes as it has particles.
static uint32_t topo_span(uint32_t np)
{
    const uint64_t resident = (uint64_t)sm_count() * TOPO_THREADS_PER_SM;
    return (uint64_t)np >= 4 * resident ? 4u : ((uint64_t)np >= 2 * resident ? 2u : 1u);
}

template <int TB>
static void launch_topo_as(const Dev &d, uint32_t np, bool visc, int a, cudaStream_t st)
{
    // one warp per span x 32 particles
    const uint32_t span = d.topo_span ? d.topo_span : topo_span(np);
    const unsigned grid = div_up(div_up(np, 32u * span), (uint32_t)TB / 32u);
    if (d.inst)   // batched contexts: contact model 2 only
        k_topo<false, true, TB><<<grid, TB, 0, st>>>(d, a, span);
    else if (visc)
        k_topo<true, false, TB><<<grid, TB, 0, st>>>(d, a, span);
    else
        k_topo<false, false, TB><<<grid, TB, 0, st>>>(d, a, span);
}

template <int CB>
static void launch_contact_as(const ContactArgs &args, uint32_t np, int model, cudaStream_t st)
{
    if (args.d.inst)   // batched contexts: contact model 2 only
        k_contact<2, true, CB><<<contact_grid<2, true, CB>(np), CB, 0, st>>>(args);
    else if (model == 3)
        k_contact<3, false, CB><<<contact_grid<3, false, CB>(np), CB, 0, st>>>(args);
    else
        k_contact<2, false, CB><<<contact_grid<2, false, CB>(np), CB, 0, st>>>(args);
}

void launch_topo(const Dev &d, uint32_t np, bool visc, int a, cudaStream_t st)
{
    if (d.shape) launch_topo_as<topo_block(1)>(d, np, visc, a, st);
    else launch_topo_as<topo_block(0)>(d, np, visc, a, st);
}

// Blocks of k_force_tiles: as many as fit on the device at once, no more
// than there are tiles.
template <int MODEL, bool BATCH, bool SLOTS>
static void launch_force_tiles(const ForceArgs &args, uint32_t np, cudaStream_t st)
{
    const uint32_t grid = std::min(div_up(np, FT_TILE * FORCE_WARPS),
                                   resident_blocks<k_force_tiles<MODEL, BATCH, SLOTS>, 32 * FORCE_WARPS>());
    if (grid) k_force_tiles<MODEL, BATCH, SLOTS><<<grid, 32 * FORCE_WARPS, 0, st>>>(args);
}

template <bool SLOTS>
static void launch_force_as(const ForceArgs &args, uint32_t np, int model, cudaStream_t st)
{
    if (args.d.inst)   // batched contexts: contact model 2 only
        launch_force_tiles<2, true, SLOTS>(args, np, st);
    else if (model == 1)
        launch_force_tiles<1, false, false>(args, np, st);
    else if (model == 3)
        launch_force_tiles<3, false, SLOTS>(args, np, st);
    else
        launch_force_tiles<2, false, SLOTS>(args, np, st);
}

// slots: the kernel does k_contact's work too.
void launch_force(const Dev &d, const Params &hp, uint32_t np, int model, int a, int write_outputs,
                  bool slots, cudaStream_t st)
{
    const ForceArgs args{d, a, write_outputs, -1, force_consts(hp), law_params(hp)};
    if (d.mu_p)   // the differentiable step
        k_force_diff<<<div_up(np, FORCE_BLOCK), FORCE_BLOCK, 0, st>>>(args);
    else if (slots)
        launch_force_as<true>(args, np, model, st);
    else
        launch_force_as<false>(args, np, model, st);
}

// The differentiable step, recording tape row `tape_step`.
void launch_force_tape(const Dev &d, uint32_t np, int a, int tape_step, cudaStream_t st)
{
    ForceArgs args{d, a, 0, tape_step, ForceConsts{}, LawParams{}};
    k_force_diff<<<div_up(np, FORCE_BLOCK), FORCE_BLOCK, 0, st>>>(args);
}

// The slot forces of contact models 2 and 3; model 1 has no slots (k_topo
// sums its forces) and the differentiable step evaluates its own law in
// k_force_diff, recording the tape.
void launch_contact(const Dev &d, const Params &hp, uint32_t np, int model, int a, int write_outputs,
                    cudaStream_t st)
{
    if (model == 1 || d.mu_p) return;
    ContactArgs args{d, a, write_outputs, law_params(hp)};
    if (d.shape) launch_contact_as<contact_block(1)>(args, np, model, st);
    else launch_contact_as<contact_block(0)>(args, np, model, st);
}

}  // namespace sphk
