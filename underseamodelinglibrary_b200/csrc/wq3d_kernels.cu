/*
 * wq3d_kernels.cu -- FP64 WaveQ3D propagation kernels for sm_100a.
 *
 * One step of wave_queue::step() (waveq3d/wave_queue.cc:155-192) is five
 * launches (four under the inline reflection schedule):
 *   k_reflect   one thread per ray on the worklist of rays that reflect in
 *               this step: the surface/bottom reflection chain with the RK3
 *               re-initialisation (reflect_chain), on a private copy of the
 *               ray written to its shadow slot.  It only reads the fronts,
 *               so it runs on a side stream beside the previous step's
 *               k_cpa / k_eigenray.
 *   k_advance   one thread per ray: caustic hand-off (for a reflecting ray
 *               on its states before the reflection) and vertices,
 *               wave_front::find_edges (reflecting rays read from their
 *               shadow slots), the queue rotation, the AB3 step and
 *               wave_front::update of the new front, and the next step's
 *               reflection worklist; k_advance_inline runs the next step's
 *               reflection chains itself instead.
 *   k_commit    writes the reflected rays' slots and the caustic and vertex
 *               counts into the fronts, on the eigenray stream.
 *   k_cpa       closest-point-of-approach test (detect_eigenrays +
 *               is_closest_ray), a warp of neighbouring rays against
 *               clusters of targets, with distance2 recomputed from
 *               per-front terms and the targets that no ray of the warp
 *               can keep dropped by FP32 bounds; k_cpa_items decides the
 *               rest in FP64.
 *   k_eigenray  one warp per CPA found: build_eigenray, compute_offsets,
 *               hybrid Gaussian or classic spreading, target angles.
 *
 * Compiled with --fmad=false: every add and multiply rounds as in the
 * reference, so the FP64 form differs from the CPU oracle only through the
 * last-place differences between CUDA's and the host's sin/cos/exp.
 *
 * The file is compiled twice.  The full build defines every kernel, with
 * the stepping kernels in namespace "gridded" (all ocean model kinds).  The
 * second build (WQ3D_WITH_GRID=0, WQ3D_KERNEL_NS=analytic,
 * WQ3D_STEP_KERNELS_ONLY=1) defines only the stepping kernels, in
 * namespace "analytic", without the gridded models.
 */
#ifndef WQ3D_KERNEL_NS
#define WQ3D_KERNEL_NS gridded
#endif
#ifndef WQ3D_STEP_KERNELS_ONLY
#define WQ3D_STEP_KERNELS_ONLY 0
#endif
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "wq3d_engine.cuh"

namespace wq3d {

namespace {

struct RayS {
    double pos[3];
    double pg[3];
    double nd[3];
    double ng[3];
    double c;
    double sg[3];
    double dist;
};

struct Roles {
    const FrontPtrs* P;
    const FrontPtrs* V;
    const FrontPtrs* C;
    const FrontPtrs* X;
};

__device__ __forceinline__ void roles_at(const QueueDev& q, int64_t s,
                                         Roles& r) {
    r.P = &q.F[ring_slot(s + 4)];
    r.V = &q.F[ring_slot(s + 1)];
    r.C = &q.F[ring_slot(s + 2)];
    r.X = &q.F[ring_slot(s + 3)];
}

__device__ __forceinline__ void set_err(const QueueDev& q, uint32_t bit) {
    atomicOr(q.err, bit);
}

/* profile evaluation for one point (profile_model::sound_speed) */
__device__ __forceinline__ void profile_at(const QueueDev& q, const double* pos,
                                           double* c, double* sg) {
    sound_speed(q.oc.prof, q.R, pos[0], pos[1], pos[2], c, sg);
}

/* wave_front::update on a 1x1 front without targets */
__device__ __forceinline__ void update1(const QueueDev& q, RayS& y) {
    profile_at(q, y.pos, &y.c, y.sg);
    double st;
    ray_derivs<!WQ3D_WITH_GRID>(y.c, y.sg[0], y.sg[1], y.sg[2], y.pos, y.nd, y.pg, y.ng, &st);
}

/* wave_front::update of the FP32 propagation form (no distance terms) */
__device__ __forceinline__ void update1_f32(const QueueDev& q, RayS& y) {
    float c, g[3];
    sound_speed_f32(q.oc.prof, q.R, y.pos[0], y.pos[1], y.pos[2], &c, g);
    y.c = (double)c;
    y.sg[0] = (double)g[0];
    y.sg[1] = (double)g[1];
    y.sg[2] = (double)g[2];
    ray_derivs_f32(c, g, y.pos, y.nd, y.pg, y.ng);
}

/* ode_integ.cc:20-126 */
__device__ __forceinline__ void rk1(double h, const RayS& y0, RayS& y1) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        y1.pos[k] = y0.pos[k] + 0.5 * h * y0.pg[k];
        y1.nd[k] = y0.nd[k] + 0.5 * h * y0.ng[k];
    }
}
__device__ __forceinline__ void rk2(double h, const RayS& y0, const RayS& y1,
                                    RayS& y2) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        y2.pos[k] = y0.pos[k] + h * (2.0 * y1.pg[k] - y0.pg[k]);
        y2.nd[k] = y0.nd[k] + h * (2.0 * y1.ng[k] - y0.ng[k]);
    }
}
__device__ __forceinline__ void rk3(double h, const RayS& y0, const RayS& y1,
                                    const RayS& y2, RayS& y3) {
    double p[3], d[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        p[k] = y0.pos[k] + h / 6.0 * (y0.pg[k] + 4.0 * y1.pg[k] + y2.pg[k]);
        d[k] = y0.nd[k] + h / 6.0 * (y0.ng[k] + 4.0 * y1.ng[k] + y2.ng[k]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        y3.pos[k] = p[k];
        y3.nd[k] = d[k];
    }
}
/* ode_integ.cc:131-186, including the step distance of ab3_pos */
__device__ __forceinline__ void ab3(double h, const RayS& y0, const RayS& y1,
                                    const RayS& y2, RayS& y3) {
    const double A2 = 23.0 / 12.0, A1 = 16.0 / 12.0, A0 = 5.0 / 12.0;
    double d[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
        d[k] = h * (A2 * y2.pg[k] - A1 * y1.pg[k] + A0 * y0.pg[k]);
    const double b = y2.pos[0] * d[1];
    const double cc = y2.pos[0] * (sin(y2.pos[1]) * d[2]);
    y3.dist = sqrt(d[0] * d[0] + b * b + cc * cc);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        y3.pos[k] = y2.pos[k] + d[k];
        y3.nd[k] = y2.nd[k] + h * (A2 * y2.ng[k] - A1 * y1.ng[k] + A0 * y0.ng[k]);
    }
}

/* one ray's state through the read-only data cache, for kernels that never
 * write the arrays they read this way: the loads may then all be in flight at
 * once instead of waiting behind stores to the caller's copy */
__device__ __forceinline__ void load_ray_ro(const FrontPtrs& f, int r, RayS& y) {
    double v[17];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        v[k] = __ldg(f.pos[k] + r);
        v[3 + k] = __ldg(f.pg[k] + r);
        v[6 + k] = __ldg(f.nd[k] + r);
        v[9 + k] = __ldg(f.ng[k] + r);
        v[12 + k] = __ldg(f.sg[k] + r);
    }
    v[15] = __ldg(f.c + r);
    v[16] = __ldg(f.dist + r);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        y.pos[k] = v[k];
        y.pg[k] = v[3 + k];
        y.nd[k] = v[6 + k];
        y.ng[k] = v[9 + k];
        y.sg[k] = v[12 + k];
    }
    y.c = v[15];
    y.dist = v[16];
}

/* reflection_model::reflection_copy (reflection_model.cc:335-360); the
 * copied path_length of a fresh 1x1 front is zero, so it is left alone */
__device__ __forceinline__ void copy_ray(const FrontPtrs& f, int r, const RayS& y) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        f.pos[k][r] = y.pos[k];
        f.pg[k][r] = y.pg[k];
        f.nd[k][r] = y.nd[k];
        f.ng[k][r] = y.ng[k];
        f.sg[k][r] = y.sg[k];
    }
    f.c[r] = y.c;
    f.dist[r] = y.dist;
}

/* wave_front::update of the main front for one ray: profile, attenuation
 * (attenuation_thorp.cc:14-36 / attenuation_constant.cc:14-25), cleared
 * phase, derivatives and the distance2 terms */
__device__ __forceinline__ void update_main(const QueueDev& q, const FrontPtrs& f,
                                            int r, RayS& y, bool accumulate,
                                            const FrontPtrs* src) {
    profile_at(q, y.pos, &y.c, y.sg);
    double st;
    ray_derivs<!WQ3D_WITH_GRID>(y.c, y.sg[0], y.sg[1], y.sg[2], y.pos, y.nd, y.pg, y.ng, &st);
    copy_ray(f, r, y);
    f.cpa[0][r] = y.pos[0];
    f.cpa[1][r] = y.pos[1];
    f.cpa[2][r] = y.pos[2];
    f.cpa[3][r] = st;
    const double alt = y.pos[0] - q.R;
    for (int k = 0; k < q.nf; ++k) {
        double a;
        if (q.oc.prof.atten == WQ3D_ATTEN_CONSTANT) {
            a = q.oc.prof.atten_coef * y.dist * q.freq[k];
        } else {
            a = y.dist * q.alpha[k] * (1.0 + 5.88264e-6 * alt);
        }
        double p = 0.0;
        if (accumulate) {
            a += src->atten[(size_t)k * q.n + r];
            p += src->phase[(size_t)k * q.n + r];
        }
        f.atten[(size_t)k * q.n + r] = a;
        f.phase[(size_t)k * q.n + r] = p;
    }
}

/* a / r.b, by quot() when the time step's powers are in its range */
__device__ __forceinline__ double div_dt(const QueueDev& q, double a, Recip r) { return q.dt_ok ? quot(a, r) : a / r.b; }

#if !WQ3D_STEP_KERNELS_ONLY
/* wave_queue::collision_location (wave_queue.cc:982-1057) */
__device__ void collision_location(const QueueDev& q, const FrontPtrs& V,
                                   const FrontPtrs& C, const FrontPtrs& X, int i,
                                   double tw, double* pos, double* nd,
                                   double* speed) {
    const double dt = q.dt;
    const Recip time1{2.0 * dt, q.r_2dt}, time2{dt * dt, q.r_dt2};
    const double dtime2 = tw * tw;
    const double drho = div_dt(q, X.c[i] - V.c[i], time1);
    const double d2rho = div_dt(q, X.c[i] + V.c[i] - 2.0 * C.c[i], time2);
    *speed = C.c[i] + drho * tw + 0.5 * d2rho * dtime2;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double v1 = div_dt(q, X.pos[k][i] - V.pos[k][i], time1);
        const double v2 = div_dt(q, X.pos[k][i] + V.pos[k][i] - 2.0 * C.pos[k][i], time2);
        pos[k] = C.pos[k][i] + v1 * tw + 0.5 * v2 * dtime2;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double v1 = div_dt(q, X.nd[k][i] - V.nd[k][i], time1);
        const double v2 = div_dt(q, X.nd[k][i] + V.nd[k][i] - 2.0 * C.nd[k][i], time2);
        nd[k] = C.nd[k][i] + v1 * tw + 0.5 * v2 * dtime2;
    }
}
#endif

/* What a reflection reads of a ray on one front.  The reflection chain
 * keeps these of the prev, curr and next fronts in registers; the whole
 * states go to the ray's shadow slot as they are made, from which k_advance
 * and k_commit take them, so k_cpa / k_eigenray of the previous step can
 * read the fronts at the same time.  (The reference also rewrites the ray's
 * "past" entry, reflection_model.cc:320, but the AB3 step of the same
 * wave_queue::step overwrites that entry before anything reads it.) */
struct RayC {
    double pos[3], nd[3], c;
};

/* a front's or a slot's state (17 doubles), without the slopes */
__device__ __forceinline__ void load_rayc(const FrontPtrs& f, int r, RayC& y) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        y.pos[k] = __ldg(f.pos[k] + r);
        y.nd[k] = __ldg(f.nd[k] + r);
    }
    y.c = __ldg(f.c + r);
}
__device__ __forceinline__ void rayc_from(const double* src, RayC& y) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        y.pos[k] = src[k];
        y.nd[k] = src[6 + k];
    }
    y.c = src[12];
}
__device__ __forceinline__ RayC rayc_of(const RayS& y) {
    RayC o;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        o.pos[k] = y.pos[k];
        o.nd[k] = y.nd[k];
    }
    o.c = y.c;
    return o;
}

/* wave_queue::collision_location (wave_queue.cc:982-1057) from one ray's
 * prev, curr and next states */
__device__ __forceinline__ void collision_rays(const QueueDev& q, const RayC& V, const RayC& Cr, const RayC& X,
                                               double tw, double* pos, double* nd, double* speed) {
    const double dt = q.dt;
    const Recip time1{2.0 * dt, q.r_2dt}, time2{dt * dt, q.r_dt2};
    const double dtime2 = tw * tw;
    const double drho = div_dt(q, X.c - V.c, time1);
    const double d2rho = div_dt(q, X.c + V.c - 2.0 * Cr.c, time2);
    *speed = Cr.c + drho * tw + 0.5 * d2rho * dtime2;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double v1 = div_dt(q, X.pos[k] - V.pos[k], time1);
        const double v2 = div_dt(q, X.pos[k] + V.pos[k] - 2.0 * Cr.pos[k], time2);
        pos[k] = Cr.pos[k] + v1 * tw + 0.5 * v2 * dtime2;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double v1 = div_dt(q, X.nd[k] - V.nd[k], time1);
        const double v2 = div_dt(q, X.nd[k] + V.nd[k] - 2.0 * Cr.nd[k], time2);
        nd[k] = Cr.nd[k] + v1 * tw + 0.5 * v2 * dtime2;
    }
}

/* seq_vector::increment: the index clamps to the last element, and -1
 * (an unsigned index in the reference) clamps there too */
__device__ __forceinline__ double seq_inc(const double* inc, int n, int k) {
    return inc[(k < 0 || k > n - 1) ? n - 1 : k];
}

/* wave_queue::build_eigenverb (wave_queue.cc:1063-1164) for ray i.  C is
 * the stored "curr" front: its path length, attenuation and caustic /
 * upper / lower counts are not changed by reflections.  curr_c is curr's
 * sound speed (re-initialised by an earlier reflection of this step) and
 * surface / bottom the counts at this point of the reflection chain. */
__device__ __noinline__ void build_eigenverb(const QueueDev& q, const FrontPtrs& C, int i, int64_t step,
                                double t_old, double tw, double grazing, double speed,
                                const double* pos, const double* nd, int type, double curr_c,
                                int surface, int bottom, int seq) {
    grazing = fabs(grazing);
    const int d = i / q.naz, a = i % q.naz;
    if (bottom > q.max_bottom || surface > q.max_surface || C.caustic[i] > q.max_caustic ||
        C.upper[i] > q.max_upper || C.lower[i] > q.max_lower)
        return;
    if (t_old <= 0.0 || grazing < 1e-6 || (q.az_boundary && a == q.naz - 1) || fabs(q.de[d]) > 89.9)
        return;
    /* footprint of the ray's share of the fan, half-way to its neighbours */
    const double de_angle = deg2rad(q.de[d]);
    const double de_plus = de_angle + 0.5 * deg2rad(seq_inc(q.de_inc, q.nde, d));
    const double de_minus = de_angle - 0.5 * deg2rad(seq_inc(q.de_inc, q.nde, d - 1));
    const double az_angle = deg2rad(q.az[a]);
    const double az_plus = az_angle + 0.5 * deg2rad(seq_inc(q.az_inc, q.naz, a));
    const int az_index = (a == 0 && q.az_boundary) ? q.naz - 1 : a;
    const double az_minus = az_angle - 0.5 * deg2rad(seq_inc(q.az_inc, q.naz, az_index - 1));
    const double area = (sin(de_plus) - sin(de_minus)) * (az_plus - az_minus);
    const double de_delta = de_plus - de_minus;
    const double az_delta = area / de_delta;
    const double path_length = C.plen[i] + curr_c * tw;
    if (path_length <= 0) return;
    const double sin_grazing = sin(grazing);
    bool above = false;
    for (int f = 0; f < q.nf && !above; ++f)
        above = pow(10.0, -0.1 * C.atten[(size_t)f * q.n + i]) * area / sin_grazing >= q.verb_threshold;
    if (!above) return;
    const uint32_t slot = atomicAdd(q.n_verb, 1u);
    if (slot >= q.cap_verb) {
        set_err(q, ERR_VERB_OVERFLOW);
        return;
    }
    wq3d_eigenverb v;
    v.travel_time = t_old + tw;
    v.length = 0.5 * path_length * de_delta / sin_grazing;
    v.width = 0.5 * path_length * az_delta;
    for (int k = 0; k < 3; ++k) v.position[k] = pos[k];
    /* wvector1::direction (wvector1.cc:79-82), degrees and back */
    v.direction = deg2rad(rad2deg(atan2(nd[2], -nd[1])));
    v.grazing = grazing;
    v.sound_speed = speed;
    v.source_de = deg2rad(q.de[d]);
    v.source_az = deg2rad(q.az[a]);
    v.de = d;
    v.az = a;
    v.surface = surface;
    v.bottom = bottom;
    v.caustic = C.caustic[i];
    v.upper = C.upper[i];
    v.lower = C.lower[i];
    v.interface_num = type;
    v.step = step;
    v.seq = seq;
    v.pad = 0;
    q.verb[slot] = v;
    for (int f = 0; f < q.nf; ++f)
        q.verb_power[(size_t)slot * q.nf + f] =
            pow(10.0, -0.1 * C.atten[(size_t)f * q.n + i]) * area / sin_grazing;
}

/* wave_queue::detect_volume_scattering (wave_queue.cc:297-345) with the
 * ray's prev / curr / next states V, Cr, X.  The collision time is
 * measured to the ocean surface, not to the layer, as in the reference. */
__device__ __noinline__ void volume_scatter(const QueueDev& q, const FrontPtrs& C, int i, int64_t step,
                               double t_old, const RayC& V, const RayC& Cr, const RayC& X,
                               int surface, int bottom, int& seq) {
    if (bottom > q.max_bottom || surface > q.max_surface || C.caustic[i] > q.max_caustic ||
        C.upper[i] > q.max_upper || C.lower[i] > q.max_lower)
        return;
    for (int k = 0; k < q.oc.nvol; ++k) {
        const double height = q.oc.vol_rho[k];
        const double d1 = height - X.pos[0];
        const double d2 = height - Cr.pos[0];
        if (d1 * d2 >= 0) continue;
        double c = Cr.c;
        const double dd = c * c * Cr.nd[0];
        const double tw = (dd == 0.0) ? 0.0 : -(Cr.pos[0] - q.R) / dd;
        double pos[3], nd[3];
        collision_rays(q, V, Cr, X, tw, pos, nd, &c);
        const double grazing = atan2(Cr.nd[0], sqrt(Cr.nd[1] * Cr.nd[1] + Cr.nd[2] * Cr.nd[2]));
        const int type = (d1 > 0) ? WQ3D_VERB_VOLUME_LOWER + 2 * k : WQ3D_VERB_VOLUME_UPPER + 2 * k;
        build_eigenverb(q, C, i, step, t_old, tw, grazing, c, pos, nd, type, Cr.c, surface, bottom, seq++);
    }
}

/* update1_f32 out of line: the FP32 form's path through the one update that
 * the re-initialisation inlines */
__device__ __noinline__ void reinit_update_f32(const QueueDev& q, RayS& y) { update1_f32(q, y); }

/* wave_front::update of the re-initialisation; *st: sin(theta) */
__device__ __forceinline__ void reinit_update(const QueueDev& q, RayS& y, double* st) {
    if (q.precision == WQ3D_FP32) {
        RayS t = y;
        reinit_update_f32(q, t);
        y = t;
        *st = sin(y.pos[1]);
    } else {
        profile_at(q, y.pos, &y.c, y.sg);
        ray_derivs<!WQ3D_WITH_GRID>(y.c, y.sg[0], y.sg[1], y.sg[2], y.pos, y.nd, y.pg, y.ng, st);
    }
}

/* reflection_model::reflection_reinit: from the collision point back to
 * the times of the curr, prev and past fronts by RK3, and forward to the
 * next by AB3.  v, c, x take the new prev, curr and next; "out" takes the
 * whole states (out.put(0 prev / 1 curr / 2 next, state)).
 *
 * Ten updates follow one another and bound the chain of a reflecting ray,
 * and so the step.  They run as ten rounds of one loop with one inlined
 * copy of the update: the states stay in registers, and the code is small
 * enough to stay in the instruction cache.  Per step in k_reflect, against
 * out-of-line updates on states in local memory: 38 for 60 us on the sloped
 * workload, 60 for 108 us on 901 x 45 rays over a gridded ocean, 49 for 88 us
 * on STD14.  (Ten inlined copies of the update waited on instruction
 * fetch.) */
template <class Out>
__device__ __forceinline__ void reinit_ray(const QueueDev& q, RayC& v, RayC& c, RayC& x, double tw, const double* pos,
                                           const double* nd, Out& out) {
    struct Slope {
        double p[3], n[3];
    };
    RayS y;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        y.pos[k] = pos[k];
        y.nd[k] = nd[k];
    }
    y.dist = 0.0;
    double bp[3], bn[3];           /* the state an RK3 run starts from */
    Slope b0, k1, k2, t0, sc, sv;  /* its slopes, the run's, the collision point's, curr's, prev's */
    double h = -tw, st, st_c = 0.0;
    /* rounds: 0 the collision point; 1 2 3 RK3 to curr; 4 5 6 to prev; 7 8
     * to past (whose second slope is the collision point's: the reference
     * does not update there); 9 AB3 to next */
#pragma unroll 1
    for (int r = 0; r < 10; ++r) {
        reinit_update(q, y, &st);
        Slope s;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            s.p[k] = y.pg[k];
            s.n[k] = y.ng[k];
        }
        int next; /* 1, 2, 3: the next state is that RK3 stage; 4: AB3 */
        if (r == 1 || r == 4 || r == 7) {
            k1 = s;
            k2 = t0;
            next = r == 7 ? 3 : 2;
        } else if (r == 2 || r == 5) {
            k2 = s;
            next = 3;
        } else if (r == 8) {
            next = 4;
        } else if (r == 9) {
            out.put(2, y);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                x.pos[k] = y.pos[k];
                x.nd[k] = y.nd[k];
            }
            x.c = y.c;
            return;
        } else {
            /* 0, 3, 6: a run starts here */
            if (r == 0) {
                t0 = s;
            } else {
                RayC& o = r == 3 ? c : v;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    o.pos[k] = y.pos[k];
                    o.nd[k] = y.nd[k];
                }
                o.c = y.c;
                out.put(r == 3 ? 1 : 0, y);
                if (r == 3) {
                    sc = s;
                    st_c = st;
                } else {
                    sv = s;
                }
                h = -q.dt;
            }
            b0 = s;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                bp[k] = y.pos[k];
                bn[k] = y.nd[k];
            }
            next = 1;
        }
        if (next == 1) { /* ode_integ.cc:20-126 */
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                y.pos[k] = bp[k] + 0.5 * h * b0.p[k];
                y.nd[k] = bn[k] + 0.5 * h * b0.n[k];
            }
        } else if (next == 2) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                y.pos[k] = bp[k] + h * (2.0 * k1.p[k] - b0.p[k]);
                y.nd[k] = bn[k] + h * (2.0 * k1.n[k] - b0.n[k]);
            }
        } else if (next == 3) {
            const double h6 = quot(h, Recip{6.0, 1.0 / 6.0});
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                y.pos[k] = bp[k] + h6 * (b0.p[k] + 4.0 * k1.p[k] + k2.p[k]);
                y.nd[k] = bn[k] + h6 * (b0.n[k] + 4.0 * k1.n[k] + k2.n[k]);
            }
        } else { /* ode_integ.cc:131-186; sin(theta) of curr is its update's */
            const double A2 = 23.0 / 12.0, A1 = 16.0 / 12.0, A0 = 5.0 / 12.0;
            const double dt = q.dt;
            double d[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) d[k] = dt * (A2 * sc.p[k] - A1 * sv.p[k] + A0 * s.p[k]);
            const double e = c.pos[0] * d[1];
            const double f = c.pos[0] * (st_c * d[2]);
            y.dist = sqrt(d[0] * d[0] + e * e + f * f);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                y.pos[k] = c.pos[k] + d[k];
                y.nd[k] = c.nd[k] + dt * (A2 * sc.n[k] - A1 * sv.n[k] + A0 * s.n[k]);
            }
        }
    }
}

__device__ void record_reflection(const QueueDev& q, int64_t step, double t_old,
                                  int i, double tw, double grazing, double c,
                                  const double* pos, const double* nd, int type,
                                  int seq) {
    if (!q.want_refl) return;
    const uint32_t slot = atomicAdd(q.n_refl, 1u);
    if (slot >= q.cap_refl) {
        set_err(q, ERR_REFL_OVERFLOW);
        return;
    }
    wq3d_reflection r;
    r.time = t_old + tw;
    r.dt = tw;
    r.grazing = grazing;
    r.speed = c;
    for (int k = 0; k < 3; ++k) {
        r.position[k] = pos[k];
        r.ndirection[k] = nd[k];
    }
    r.de = i / q.naz;
    r.az = i % q.naz;
    r.type = type;
    r.pad = seq;
    r.step = step;
    q.refl[slot] = r;
}

/* one bounce's loss: what every frequency's attenuation and phase gain,
 * or for a wind-driven surface (Eckart) the sine of the grazing angle */
struct Loss {
    double amp, ph, sin_grazing;
    int eckart; /* 0, or the boundary (1 surface, 2 bottom) whose wind sets it */
};

__device__ __forceinline__ void bounce_loss(const LossDev& Lo, double grazing, int which, Loss& o) {
    o.amp = o.ph = o.sin_grazing = 0.0;
    o.eckart = 0;
    if (Lo.kind == WQ3D_LOSS_ECKART) {
        o.eckart = which;
        o.sin_grazing = sin(grazing);
    } else {
        reflect_loss_scalar(Lo, grazing, &o.amp, &o.ph);
    }
}

/* reflection_model::surface_reflection (reflection_model.cc:187-243) up to
 * the re-initialisation, for a ray heading up (the reference's grazing angle
 * is positive exactly when the curr direction's radial part is): collision
 * time, point and reflected direction.  The angle itself is formed only for
 * those who read it. */
template <class Out>
__device__ __forceinline__ void surface_bounce(const QueueDev& q, const FrontPtrs& C, const RayC& v, const RayC& cr,
                                               const RayC& x, int i, int64_t step, double t_old, int surface,
                                               int bottom, int& seq, double* tw_out, double* pos, double* nd,
                                               Out& out) {
    double c = cr.c;
    const double d = c * c * cr.nd[0];
    const double tw = (d == 0.0) ? 0.0 : -(cr.pos[0] - q.R) / d;
    collision_rays(q, v, cr, x, tw, pos, nd, &c);
    const LossDev& Lo = q.oc.surf.loss;
    double grazing = 0.0;
    if (q.want_refl || q.want_verbs || Lo.kind == WQ3D_LOSS_ECKART || Lo.kind == WQ3D_LOSS_RAYLEIGH) {
        const double n1 = cr.nd[1], n2 = cr.nd[2];
        grazing = atan2(cr.nd[0], sqrt(n1 * n1 + n2 * n2));
    }
    record_reflection(q, step, t_old, i, tw, grazing, c, pos, nd, 1, seq);
    if (q.want_verbs)
        build_eigenverb(q, C, i, step, t_old, tw, grazing, c, pos, nd, WQ3D_VERB_SURFACE, cr.c, surface, bottom, seq);
    ++seq;
    if (out.losses()) {
        Loss l;
        bounce_loss(Lo, grazing, 1, l);
        l.ph = -M_PI;
        out.add(l);
    }
    nd[0] = -nd[0];
    *tw_out = tw;
}

/* reflection_model::bottom_reflection (reflection_model.cc:33-182) up to
 * the re-initialisation */
template <class Out>
__device__ __forceinline__ void bottom_bounce(const QueueDev& q, const FrontPtrs& C, const RayC& v, const RayC& cr,
                                              const RayC& x, int i, double depth, int64_t step, double t_old,
                                              int surface, int bottom, int& seq, double* tw_out, double* position,
                                              double* ndir, Out& out) {
    const BoundaryDev& B = q.oc.bot;
    double c = cr.c;
    double c2 = c * c;
    double nrm[3];
    double bottom_rho = boundary_height_normal(B, cr.pos[1], cr.pos[2], nrm);
    double height_water = cr.pos[0] - bottom_rho;
    const double TOO_SHALLOW = 300.0 * q.dt;
    const bool shallow = (q.R - bottom_rho) < TOO_SHALLOW;
    if (shallow) {
        const double N = sqrt(nrm[1] * nrm[1] + nrm[2] * nrm[2]);
        nrm[0] = 0.0;
        nrm[1] = nrm[1] / N;
        nrm[2] = nrm[2] / N;
    }
    double dot_full = nrm[0] * (c2 * cr.nd[0]) + nrm[1] * (c2 * cr.nd[1]) + nrm[2] * (c2 * cr.nd[2]);
    const double MIN_REFLECT = 6.0;
    double max_dot = -fmax(MIN_REFLECT, (height_water + depth) * nrm[0]);
    if (dot_full >= max_dot) dot_full = max_dot;
    const double dot_water = -height_water * nrm[0];
    const double time_water = fmax(0.0, dot_water / dot_full);

    collision_rays(q, v, cr, x, time_water, position, ndir, &c);
    bottom_rho = boundary_height_normal(B, position[1], position[2], nrm);
    if (shallow) {
        const double N = sqrt(nrm[1] * nrm[1] + nrm[2] * nrm[2]);
        nrm[0] = 0.0;
        nrm[1] = nrm[1] / N;
        nrm[2] = nrm[2] / N;
    }
    c2 = c * c;
    height_water = position[0] - bottom_rho;
    ndir[0] = c2 * ndir[0];
    ndir[1] = c2 * ndir[1];
    ndir[2] = c2 * ndir[2];
    dot_full = nrm[0] * ndir[0] + nrm[1] * ndir[1] + nrm[2] * ndir[2];
    max_dot = -fmax(MIN_REFLECT, (height_water + depth) * nrm[0]);
    if (dot_full >= max_dot) dot_full = max_dot;

    double grazing;
    const double sine = dot_full / c;
    if (sine >= 1.0) {
        grazing = -M_PI_2;
    } else if (sine <= -1.0) {
        grazing = M_PI_2;
    } else {
        grazing = asin(-sine);
    }
    record_reflection(q, step, t_old, i, time_water, grazing, c, position, ndir, 0, seq);
    if (q.want_verbs)
        build_eigenverb(q, C, i, step, t_old, time_water, grazing, c, position, ndir, WQ3D_VERB_BOTTOM, cr.c, surface,
                        bottom, seq);
    ++seq;
    if (out.losses()) {
        Loss l;
        bounce_loss(B.loss, grazing, 2, l);
        if (B.loss.kind == WQ3D_LOSS_ECKART) l.ph = M_PI;
        out.add(l);
        if (q.sens) {
            double g[3];
            reflect_loss_rayleigh_grad(B.loss, grazing, g);
            out.tangents(g);
        }
    }
    dot_full *= 2.0;
    ndir[0] = ndir[0] - dot_full * nrm[0];
    ndir[1] = ndir[1] - dot_full * nrm[1];
    ndir[2] = ndir[2] - dot_full * nrm[2];
    const double N = sqrt(ndir[0] * ndir[0] + ndir[1] * ndir[1] + ndir[2] * ndir[2]) * c;
    if (divisor_ok(N) && dividend_ok(ndir[0]) && dividend_ok(ndir[1]) && dividend_ok(ndir[2])) {
        const Recip r = recip(N);
        ndir[0] = quot(ndir[0], r);
        ndir[1] = quot(ndir[1], r);
        ndir[2] = quot(ndir[2], r);
    } else {
        ndir[0] = ndir[0] / N;
        ndir[1] = ndir[1] / N;
        ndir[2] = ndir[2] / N;
    }
    *tw_out = time_water;
}

/* The reference's detect_reflections for one ray (wave_queue.cc:197-256):
 * volume layers, then the surface / bottom chain, volume layers after each
 * reflection.  A ray tries the surface first, else the bottom, and after a
 * bounce the other boundary, until it meets none; out.stop(n) may end the
 * chain after n bounces.  v, c, x: the ray's prev, curr and next states,
 * replaced by the reflected ones. */
template <class Out>
__device__ __forceinline__ void bounce_chain(const QueueDev& q, const FrontPtrs& C, int i, int64_t step, double t_old,
                                             RayC& v, RayC& c, RayC& x, int& surface, int& bottom, Out& out) {
    const bool vol = q.want_verbs && q.oc.nvol > 0;
    int seq = 0; /* orders the ray's events */
    int last = -1; /* 0 the surface, 1 the bottom */
    if (vol) volume_scatter(q, C, i, step, t_old, v, c, x, surface, bottom, seq);
#pragma unroll 1
    for (int n = 0;; ++n) {
        if (n > 0 && out.stop(n)) return;
        const bool surf = last != 0 && x.pos[0] - q.R > 0.0 && !(c.nd[0] <= 0.0);
        double depth = 0.0;
        if (!surf) {
            if (last == 1) return;
            depth = boundary_height(q.oc.bot, x.pos[1], x.pos[2]) - x.pos[0];
            if (!(depth > 0.0)) return;
        }
        double tw, pos[3], nd[3];
        if (surf)
            surface_bounce(q, C, v, c, x, i, step, t_old, surface, bottom, seq, &tw, pos, nd, out);
        else
            bottom_bounce(q, C, v, c, x, i, depth, step, t_old, surface, bottom, seq, &tw, pos, nd, out);
        reinit_ray(q, v, c, x, tw, pos, nd, out);
        out.bounced(!surf);
        if (surf)
            ++surface;
        else
            ++bottom;
        last = surf ? 0 : 1;
        if (vol) volume_scatter(q, C, i, step, t_old, v, c, x, surface, bottom, seq);
    }
}

/* whether the "next" ray reflects at the start of the following step:
 * 1 = surface if above the surface and heading up (surface_reflection's
 * grazing > 0, which is the sign of the direction's radial part), else 2 = bottom if below the bottom (wave_queue.cc:222-256) */
__device__ __forceinline__ uint8_t reflect_decision(const QueueDev& q,
                                                    const double* xpos,
                                                    const double* cnd) {
    if (xpos[0] - q.R > 0.0 && cnd[0] > 0.0) return 1;
    const double h = boundary_height(q.oc.bot, xpos[1], xpos[2]);
    return (h - xpos[0] > 0.0) ? 2 : 0;
}

/* appends a reflecting ray to worklist p: surface reflections fill it
 * from the front, bottom reflections from the back, so the warps of
 * k_reflect mostly take one path */
__device__ __forceinline__ void work_append(const QueueDev& q, int p, uint8_t kind, int i) {
    if (kind == 1) {
        const uint32_t slot = atomicAdd(q.n_work[p], 1u);
        if (slot < (uint32_t)q.n) q.work[p][slot] = (uint32_t)i;
    } else {
        const uint32_t slot = atomicAdd(q.n_work_b[p], 1u);
        if (slot < (uint32_t)q.n) q.work[p][q.n - 1 - slot] = (uint32_t)i;
    }
}

/* the shadow slot of a reflecting ray: prev, curr and next states (17 doubles each), the next
 * front's attenuation and phase (nf each), the three loss tangents of the
 * step's bottom bounces, and the phases again as they are when the caustic
 * hand-off of the neighbour below shifted them by -pi/2 before the
 * reflection (nf); counts in shadow_cnt */
__device__ __forceinline__ size_t shadow_stride(const QueueDev& q) { return 54 + 3 * (size_t)q.nf; }

__device__ __forceinline__ void ray_to(double* dst, const RayS& y) {
    for (int k = 0; k < 3; ++k) {
        dst[k] = y.pos[k];
        dst[3 + k] = y.pg[k];
        dst[6 + k] = y.nd[k];
        dst[9 + k] = y.ng[k];
        dst[13 + k] = y.sg[k];
    }
    dst[12] = y.c;
    dst[16] = y.dist;
}

__device__ __forceinline__ void ray_from(const double* src, RayS& y) {
    for (int k = 0; k < 3; ++k) {
        y.pos[k] = src[k];
        y.pg[k] = src[3 + k];
        y.nd[k] = src[6 + k];
        y.ng[k] = src[9 + k];
        y.sg[k] = src[13 + k];
    }
    y.c = src[12];
    y.dist = src[16];
}

/* A ray that reflected at step s-1 keeps its post-reflection states in
 * that step's shadow slot until k_commit of step s-1, which runs on its
 * own stream behind the eigenray construction of step s-2, has written
 * them into the fronts.  At step s those are its prev state (the slot's
 * curr, at +17) and its curr state (the slot's next, at +34), with the
 * slot's counts.  Returns the slot, or null when the ray did not reflect
 * at step s-1 and the fronts hold its states. */
__device__ __forceinline__ const double* prev_step_slot(const QueueDev& q, int64_t s, int i,
                                                        const int32_t** cnt = nullptr) {
    const int p = shadow_set(s + SHADOW_SETS - 1); /* the set of step s-1 */
    if (!(__ldg(q.commit_flag[p] + i) & COMMIT_REFLECT)) return nullptr;
    const int32_t w = __ldg(q.shadow_slot[p] + i);
    WQ_CHECKED_OR(q, w >= 0 && w < q.n, return nullptr);
    if (cnt) *cnt = q.shadow_cnt[p] + 3 * (size_t)w;
    return q.shadow[p] + (size_t)w * shadow_stride(q);
}

/* the prev and curr states of ray i at step s (fronts V and C, or the
 * previous step's shadow slot) */
__device__ __forceinline__ void load_prev_curr(const QueueDev& q, int64_t s, const Roles& R, int i,
                                               RayS& v, RayS& c) {
    const double* sp = prev_step_slot(q, s, i);
    if (sp) {
        ray_from(sp + 17, v);
        ray_from(sp + 34, c);
    } else {
        load_ray_ro(*R.V, i, v);
        load_ray_ro(*R.C, i, c);
    }
}

/* rho of ray j on the curr front at step s */
__device__ __forceinline__ double curr_rho(const QueueDev& q, int64_t s, const Roles& R, int j) {
    const double* sp = prev_step_slot(q, s, j);
    return sp ? __ldg(sp + 34) : __ldg(R.C->pos[0] + j);
}

}  // namespace

namespace WQ3D_KERNEL_NS {

/* ------------------------------------------------------------------ */
/* start-up: wave_queue ctor (wave_queue.cc:83-85) for one ray         */
/* ------------------------------------------------------------------ */
__global__ void __launch_bounds__(128) k_startup(__grid_constant__ const QueueDev q) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= q.n) return;
    const int d = i / q.naz, a = i % q.naz;
    const FrontPtrs& past = q.F[0];
    const FrontPtrs& prev = q.F[1];
    const FrontPtrs& curr = q.F[2];
    const FrontPtrs& next = q.F[3];
    /* wave_front::init_wave (wave_front.cc:84-121) */
    RayS c0;
    c0.nd[0] = q.sin_de[d] / q.c_source;
    c0.nd[1] = (-q.cos_de[d] * q.cos_az[a]) / q.c_source;
    c0.nd[2] = (q.cos_de[d] * q.sin_az[a]) / q.c_source;
    c0.pos[0] = q.source[0];
    c0.pos[1] = q.source[1];
    c0.pos[2] = q.source[2];
    c0.dist = 0.0;
    update_main(q, curr, i, c0, false, nullptr);
    /* init_wavefronts (wave_queue.cc:114-150); intermediate updates of the
     * reference's _next land in registers, only final values are stored */
    const double h = -q.dt;
    RayS n1, p1, v1;
    n1.dist = 0.0;
    p1.dist = 0.0;
    v1.dist = 0.0;
    rk1(h, c0, n1);
    update1(q, n1);
    rk2(h, c0, n1, p1);
    update1(q, p1);
    rk3(h, c0, n1, p1, v1);
    update_main(q, prev, i, v1, false, nullptr);
    rk1(h, v1, n1);
    update1(q, n1);
    rk2(h, v1, n1, p1);
    update1(q, p1);
    rk3(h, v1, n1, p1, p1);
    update_main(q, past, i, p1, false, nullptr);
    RayS x;
    ab3(q.dt, p1, v1, c0, x);
    update_main(q, next, i, x, false, nullptr);
    next.plen[i] = x.dist + 0.0;
    curr.plen[i] = 0.0;
    prev.plen[i] = 0.0;
    past.plen[i] = 0.0;
    for (int f = 0; f < RING; ++f) {
        const FrontPtrs& F = q.F[f];
        F.surface[i] = 0;
        F.bottom[i] = 0;
        F.caustic[i] = 0;
        F.upper[i] = 0;
        F.lower[i] = 0;
        F.on_edge[i] = 0;
    }
    const uint8_t f = reflect_decision(q, x.pos, c0.nd);
    q.flag[0][i] = f;
    if (f) work_append(q, 0, f, i);
    (void)a;
}

/* ------------------------------------------------------------------ */
/* one step: reflections (overlapping the previous step's CPA work),   */
/* then every ray advances                                             */
/* ------------------------------------------------------------------ */

/* The shadow slot of a reflecting ray as its chain fills it (see
 * shadow_stride).  The frequencies' losses are kept per bounce and applied
 * once, at the end. */
struct SlotOut {
    const QueueDev& q;
    double* sh;
    double dl[3];
    int n;
    Loss loss[MAX_BOUNCE + 2];
    __device__ SlotOut(const QueueDev& q_, double* sh_) : q(q_), sh(sh_), dl{0.0, 0.0, 0.0}, n(0) {}
    __device__ void put(int which, const RayS& y) { ray_to(sh + 17 * which, y); }
    __device__ bool losses() const { return true; }
    __device__ void add(const Loss& l) { loss[n++] = l; }
    __device__ void tangents(const double* g) {
        for (int j = 0; j < 3; ++j) dl[j] += g[j];
    }
    __device__ void bounced(bool) {}
    __device__ bool stop(int bounces) {
        if (bounces <= MAX_BOUNCE) return false;
        set_err(q, ERR_BOUNCE_LIMIT);
        return true;
    }
    /* attenuation and phase of frequency f before the reflections */
    __device__ void apply(int f, double att, double ph) {
        double phf = ph - M_PI_2;
        for (int k = 0; k < n; ++k) {
            double a = loss[k].amp;
            if (loss[k].eckart) {
                const LossDev& Lo = loss[k].eckart == 1 ? q.oc.surf.loss : q.oc.bot.loss;
                const double x = q.freq[f] * (Lo.p[0] * Lo.p[0]) * loss[k].sin_grazing;
                a = 8.6e-9 * (x * x);
            }
            att += a;
            ph += loss[k].ph;
            phf += loss[k].ph;
        }
        sh[51 + f] = att;
        sh[51 + q.nf + f] = ph;
        sh[54 + 2 * q.nf + f] = phf;
    }
};

/* The reflection chain of ray i at the start of step s on the ray's prev,
 * curr and next states v, c, x; surface, bottom, caustic: its counts, atten
 * and phase: its next-front losses ([f][n]), all before the step's
 * reflections.  The result goes to slot w of set shadow_set(s); k_advance of
 * step s takes it from there.  (The launch that listed the ray made the
 * chain's first test on the same values, so at least one bounce fills the
 * slot.)  The caustic hand-off from the D/E neighbour below (wave_queue.cc:
 * 274-292), which the reference runs before the ray reflects, is decided by
 * k_advance of step s, when that neighbour's next front is complete; the
 * slot carries the phases both without and with its -pi/2 shift. */
__device__ __forceinline__ void reflect_chain_body(const QueueDev& q, int64_t s, int i, uint32_t w, RayC& v, RayC& c,
                                                   RayC& x, int surface, int bottom, int caustic,
                                                   const double* atten, const double* phase, double t_old) {
    Roles R;
    roles_at(q, s, R);
    const int set = shadow_set(s);
    SlotOut out(q, q.shadow[set] + (size_t)w * shadow_stride(q));
    bounce_chain(q, *R.C, i, s + 1, t_old, v, c, x, surface, bottom, out);
    for (int f = 0; f < q.nf; ++f) out.apply(f, atten[(size_t)f * q.n + i], phase[(size_t)f * q.n + i]);
    /* the next front's loss tangents take this step's bottom bounces
     * when k_commit applies the slot; the previous step's eigenray
     * construction may still be reading them */
    if (q.sens)
        for (int j = 0; j < 3; ++j) out.sh[51 + 2 * q.nf + j] = out.dl[j];
    q.shadow_cnt[set][3 * (size_t)w] = surface;
    q.shadow_cnt[set][3 * (size_t)w + 1] = bottom;
    q.shadow_cnt[set][3 * (size_t)w + 2] = caustic;
    q.shadow_slot[set][i] = (int32_t)w;
}

/* out of line for the inline schedule's advance, whose other rays need
 * none of its registers */
__device__ __noinline__ void reflect_chain(const QueueDev& q, int64_t s, int i, uint32_t w, const RayC& v,
                                           const RayC& c, const RayC& x, int surface, int bottom, int caustic,
                                           const double* atten, const double* phase, double t_old) {
    RayC a = v, b = c, d = x;
    reflect_chain_body(q, s, i, w, a, b, d, surface, bottom, caustic, atten, phase, t_old);
}

/* Reflecting rays of step s listed by the launch that produced the "next"
 * front: the reflection chain on a private copy of each ray.  The fronts
 * are only read here, so this kernel runs concurrently with k_cpa /
 * k_eigenray of step s-1.  (k_advance reflects the following step's rays
 * itself where nothing in between needs the committed fronts; this kernel
 * then finds an empty list.) */
__global__ void __launch_bounds__(64) k_reflect(__grid_constant__ const QueueDev q, int k) {
    const int64_t s = *q.d_base + k;
    const uint32_t nsurf = min(*q.n_work[s & 1], (uint32_t)q.n);
    const uint32_t nwork = nsurf + min(*q.n_work_b[s & 1], (uint32_t)q.n - nsurf);
    const uint32_t* work = q.work[s & 1];
    const double t_old = q.d_times[k];
    Roles R;
    roles_at(q, s, R);
    for (uint32_t ww = blockIdx.x * blockDim.x + threadIdx.x; ww < nwork; ww += gridDim.x * blockDim.x) {
        /* list slot: surface part at the front, bottom part at the back */
        const uint32_t w = ww < nsurf ? ww : (uint32_t)q.n - 1 - (ww - nsurf);
        const int i = (int)work[w];
        WQ_CHECKED_OR(q, i >= 0 && i < q.n, continue);
        /* the fronts are read-only here */
        RayC v, c, x;
        const double* sp = prev_step_slot(q, s, i);
        if (sp) {
            rayc_from(sp + 17, v);
            rayc_from(sp + 34, c);
        } else {
            load_rayc(*R.V, i, v);
            load_rayc(*R.C, i, c);
        }
        load_rayc(*R.X, i, x);
        reflect_chain_body(q, s, i, w, v, c, x, __ldg(R.X->surface + i), __ldg(R.X->bottom + i),
                           __ldg(R.X->caustic + i), R.X->atten, R.X->phase, t_old);
    }
    /* the last block to finish empties this step's worklist, which the
     * advance of step s+1 refills (every block has read the count by then;
     * the advance of step s fills the other list) */
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const uint32_t prev = atomicAdd(q.n_done, 1u);
        if (prev == gridDim.x - 1) {
            *q.n_work[s & 1] = 0;
            *q.n_work_b[s & 1] = 0;
            *q.n_done = 0;
        }
    }
}

/* Every ray: commit of a reflected ray's shadow slot, caustic hand-off and
 * vertices for rays that did not reflect, find_edges of the front that
 * becomes "curr" (wave_front.cc:184-216; reflecting neighbours are read
 * from their shadow slots), the rotation, AB3 and update of the new front
 * (wave_queue.cc:162-183), and the reflection decision of the next step. */
/* Five blocks per SM (96 registers, spills to L1 that cost less than the
 * lost occupancy): the advance waits for memory.  Reverberation workload
 * (651,781 rays, 32 frequencies): 322 us at five, 352 at four, 408 at three,
 * 519 at two blocks; fans that do not fill the GPU do not care. */
#define WQ_ADVANCE_BOUNDS __launch_bounds__(128, 5)
template <bool INLINE>
__device__ __forceinline__ void advance_body(const QueueDev& q, int k) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t s = *q.d_base + k;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        q.n_cand[cand_list(s + 1)] = 0;
        /* the slot count the next step's inline reflections start from */
        q.n_slot[shadow_set(s + 2)] = 0;
    }
    if (i >= q.n) return;
    Roles R;
    roles_at(q, s, R);
    const uint8_t* flag_in = q.flag[s & 1];
    uint8_t* flag_out = q.flag[(s + 1) & 1];
    const int naz = q.naz;
    const int d = i / naz;
    const size_t stride = shadow_stride(q);
    const int max_de = q.nde - 1;
    int jrow[4];
    jrow[0] = i + (max(d - 2, 0) - d) * naz;
    jrow[1] = i + (max(d - 1, 0) - d) * naz;
    jrow[2] = i + (min(d + 1, max_de) - d) * naz;
    jrow[3] = i + (min(d + 2, max_de) - d) * naz;
    const bool refl = __ldg(flag_in + i) != 0;
    bool fl[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) fl[t] = __ldg(flag_in + jrow[t]) != 0;
    /* Reads go through the read-only path: in this launch no ray reads an
     * element that another ray writes (neighbours are read only where they
     * do not reflect, and a reflecting ray's entries come from its shadow
     * slot), and a ray's own updated counters and phases stay in
     * registers, so the loads need not wait behind the stores. */
    RayS y0, y1, y2, y3;
    /* one round of loads: this ray on the three fronts, and the rows
     * d-2 .. d+2 that detect_caustics and find_edges may read (rows
     * clamped to the fan; a clamped row is never used) */
    const int set = shadow_set(s);
    if (!refl) load_prev_curr(q, s, R, i, y0, y1);
    load_ray_ro(*R.X, i, y2);
    int32_t sf = __ldg(R.X->surface + i);
    int32_t bt = __ldg(R.X->bottom + i);
    int32_t cs = __ldg(R.X->caustic + i);
    int32_t up = __ldg(R.X->upper + i);
    int32_t lo = __ldg(R.X->lower + i);
    double rr[4], nn[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        rr[t] = __ldg(R.X->pos[0] + jrow[t]);
        nn[t] = __ldg(R.X->nd[0] + jrow[t]);
    }
    const double c_below = curr_rho(q, s, R, jrow[1]);
    const int32_t sf_below = __ldg(R.X->surface + jrow[1]);
    const int32_t bt_below = __ldg(R.X->bottom + jrow[1]);
    const double x_below = rr[1];
    /* reflecting neighbours: their post-reflection entries */
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        if (fl[t]) {
            const int32_t wj = __ldg(q.shadow_slot[set] + jrow[t]);
            WQ_CHECKED_OR(q, wj >= 0 && wj < q.n, return);
            const double* shj = q.shadow[set] + (size_t)wj * stride;
            rr[t] = __ldg(shj + 34);
            nn[t] = __ldg(shj + 34 + 6);
        }
    }
    const double* sh = nullptr;
    bool fold_hit = false, vtx_up = false, vtx_lo = false;
    if (refl) {
        /* the reflected ray's states come from its shadow slot; k_commit
         * writes them into the curr and next fronts once the previous
         * step's eigenray construction no longer reads those fronts */
        const int32_t w = __ldg(q.shadow_slot[set] + i);
        WQ_CHECKED_OR(q, w >= 0 && w < q.n, return);
        sh = q.shadow[set] + (size_t)w * stride;
        ray_from(sh, y0);
        ray_from(sh + 17, y1);
        ray_from(sh + 34, y2);
        sf = __ldg(q.shadow_cnt[set] + 3 * (size_t)w);
        bt = __ldg(q.shadow_cnt[set] + 3 * (size_t)w + 1);
        cs = __ldg(q.shadow_cnt[set] + 3 * (size_t)w + 2);
        /* detect_caustics of the neighbour below on this ray's states
         * before its reflection (wave_queue.cc:274-292: the reference runs
         * it first); the fronts still hold them until k_commit */
        if (d >= 1 && !fl[1]) {
            const double A = curr_rho(q, s, R, i), B = c_below;
            const double Cc = __ldg(R.X->pos[0] + i), D = x_below;
            const bool fold = (__ldg(R.X->surface + i) == sf_below) && (__ldg(R.X->bottom + i) == bt_below);
            if ((Cc - D) * (A - B) < 0 && fold) {
                fold_hit = true;
                cs += 1;
            }
        }
    } else {
        /* detect_caustics of the neighbour below (wave_queue.cc:274-292) */
        if (d >= 1 && !fl[1]) {
            const double A = y1.pos[0], B = c_below;
            const double Cc = y2.pos[0], D = x_below;
            const bool fold = (sf == sf_below) && (bt == bt_below);
            if ((Cc - D) * (A - B) < 0 && fold) {
                fold_hit = true;
                cs += 1;
            }
        }
        /* detect_vertices (wave_queue.cc:261-269) */
        const double L = y1.nd[0];
        const double Rn = y2.nd[0];
        if (L * Rn < 0.0 && Rn < 0.0) {
            vtx_up = true;
            up += 1;
        } else if (L * Rn < 0.0 && 0.0 < Rn) {
            vtx_lo = true;
            lo += 1;
        }
    }
    /* find_edges on the post-reflection "next" front (wave_front.cc:
     * 184-216): a row is an extremum when its rho is below or above both
     * neighbour rows */
    bool edge;
    {
        auto ext = [](double r0, double rp, double rm) {
            return (r0 < rp && r0 < rm) || (r0 > rp && r0 > rm);
        };
        const double r_here = y2.pos[0], n_here = y2.nd[0];
        const bool ext_d = d >= 1 && d <= max_de - 1 && ext(r_here, rr[2], rr[1]);
        const bool ext_up = d + 1 >= 1 && d + 1 <= max_de - 1 && ext(rr[2], rr[3], r_here);
        const bool ext_dn = d - 1 >= 1 && d - 1 <= max_de - 1 && ext(rr[1], r_here, rr[0]);
        edge = (d == 0) || (d == max_de) || ext_d;
        if (!edge && ext_up) {
            const double n0 = nn[2];
            if (fabs(n0 - n_here) > fabs(n0 - nn[3])) edge = true;
        }
        if (!edge && ext_dn) {
            const double n0 = nn[1];
            if (!(fabs(n0 - nn[0]) > fabs(n0 - n_here))) edge = true;
        }
    }
    const double plen_x = __ldg(R.X->plen + i);
    /* rotate and take the AB3 step; wave_front::update of the new front
     * (the distance terms' sin(theta) is FP64 in every form) */
    ab3(q.dt, y0, y1, y2, y3);
    double st;
    if (q.precision == WQ3D_FP32) {
        update1_f32(q, y3);
        st = sin(y3.pos[1]);
    } else {
        profile_at(q, y3.pos, &y3.c, y3.sg);
        ray_derivs<!WQ3D_WITH_GRID>(y3.c, y3.sg[0], y3.sg[1], y3.sg[2], y3.pos, y3.nd, y3.pg, y3.ng, &st);
    }
    const uint8_t f_next = reflect_decision(q, y3.pos, y2.nd);
    /* the per-step finiteness check: a NaN or Inf in the environment (a
     * bad profile node, a zero sound speed) reaches the new front here */
    if (!isfinite(y3.pos[0] + y3.pos[1] + y3.pos[2] + y3.nd[0] + y3.nd[1] + y3.nd[2])) set_err(q, ERR_NONFINITE);
    /* stores: the new front, the next front's edge flag (not read by the
     * previous step's eigenray construction) and what k_commit changes on
     * the prev / curr / next fronts */
    q.commit_flag[set][i] = (uint8_t)((refl ? COMMIT_REFLECT : 0) | (fold_hit ? COMMIT_FOLD : 0) |
                                 (vtx_up ? COMMIT_UPPER : 0) | (vtx_lo ? COMMIT_LOWER : 0));
    R.X->on_edge[i] = edge ? 1 : 0;
    const FrontPtrs& P = *R.P;
    copy_ray(P, i, y3);
    P.cpa[0][i] = y3.pos[0];
    P.cpa[1][i] = y3.pos[1];
    P.cpa[2][i] = y3.pos[2];
    P.cpa[3][i] = st;
    P.plen[i] = y3.dist + plen_x;
    P.surface[i] = sf;
    P.bottom[i] = bt;
    P.upper[i] = up;
    P.lower[i] = lo;
    P.caustic[i] = cs;
    if (q.sens)
        for (int j = 0; j < 3; ++j)
            P.dA[(size_t)j * q.n + i] = __ldg(R.X->dA + (size_t)j * q.n + i) + (refl ? __ldg(sh + 51 + 2 * q.nf + j) : 0.0);
    /* attenuation (attenuation_thorp.cc:14-36 / attenuation_constant.cc:
     * 14-25) added to the next front's, phase carried over; the next
     * front's own entries take the reflection's values or the caustic's
     * phase shift first */
    const double alt = y3.pos[0] - q.R;
#pragma unroll 5
    for (int f = 0; f < q.nf; ++f) {
        const size_t o = (size_t)f * q.n + i;
        double ax, px;
        if (refl) {
            ax = __ldg(sh + 51 + f);
            px = __ldg(sh + (fold_hit ? 54 + 2 * q.nf : 51 + q.nf) + f);
        } else {
            ax = __ldg(R.X->atten + o);
            px = __ldg(R.X->phase + o);
            if (fold_hit) px -= M_PI_2;
        }
        double a;
        if (q.oc.prof.atten == WQ3D_ATTEN_CONSTANT) {
            a = q.oc.prof.atten_coef * y3.dist * q.freq[f];
        } else {
            a = y3.dist * q.alpha[f] * (1.0 + 5.88264e-6 * alt);
        }
        a += ax;
        double p = 0.0;
        p += px;
        P.atten[o] = a;
        P.phase[o] = p;
    }
    flag_out[i] = f_next;
    if (!f_next) return;
    if (!INLINE) {
        work_append(q, (int)((s + 1) & 1), f_next, i);
        return;
    }
    /* the reflections of step s+1 right here: this ray's prev and curr
     * states at step s+1 are its curr and next at step s, its next the
     * front just written (read back by this thread) */
    RayC v, c;
    if (refl) {
        rayc_from(sh + 17, v);
        rayc_from(sh + 34, c);
    } else {
        const double* sp = prev_step_slot(q, s, i);
        if (sp)
            rayc_from(sp + 34, v);
        else
            load_rayc(*R.C, i, v);
        load_rayc(*R.X, i, c);
    }
    const uint32_t w = atomicAdd(q.n_slot + shadow_set(s + 1), 1u);
    if (w >= (uint32_t)q.n) {
        set_err(q, ERR_SLOT_OVERFLOW);
        return;
    }
    reflect_chain(q, s + 1, i, w, v, c, rayc_of(y3), sf, bt, cs, P.atten, P.phase, q.d_times[k + 1]);
}

/* the side schedule: the reflecting rays of step s+1 go to the worklist
 * of k_reflect */
__global__ void WQ_ADVANCE_BOUNDS k_advance(__grid_constant__ const QueueDev q, int k) {
    advance_body<false>(q, k);
}

/* the inline schedule: each thread runs step s+1's reflection chain of
 * its ray itself */
__global__ void __launch_bounds__(128, 2) k_advance_inline(__grid_constant__ const QueueDev q, int k) {
    advance_body<true>(q, k);
}

}  // namespace WQ3D_KERNEL_NS

#if !WQ3D_STEP_KERNELS_ONLY
/* What k_advance of step s decided for the prev / curr / next fronts, done
 * after the eigenray construction of step s-1 has read them: a reflected ray's
 * states, counts and next-front losses from its shadow slot
 * (reflection_model::reflection_copy, reflection_model.cc:335-360), and for
 * the other rays the caustic hand-off (count, and phase - pi/2 on every
 * frequency, wave_queue.cc:274-292) and the vertex counts (:261-269).
 * Until it has run, step s+1 reads a reflected ray's states from the slot
 * (prev_step_slot); the eigenray construction of step s, the eigenverbs of
 * step s+1 and the commit of step s+2 (which reuses this step's slot set)
 * wait for it. */
__global__ void __launch_bounds__(128) k_commit(__grid_constant__ const QueueDev q, int k) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= q.n) return;
    const int64_t s = *q.d_base + k;
    const int set = shadow_set(s);
    const uint8_t b = q.commit_flag[set][i];
    if (!b) return;
    Roles R;
    roles_at(q, s, R);
    if (b & COMMIT_REFLECT) {
        /* the prev front is read by no later kernel (this step's AB3 took
         * the reflected prev state from the slot) but is the "past" front
         * a caller may look at after the step */
        const int32_t w = q.shadow_slot[set][i];
        WQ_CHECKED_OR(q, w >= 0 && w < q.n, return);
        const double* sh = q.shadow[set] + (size_t)w * shadow_stride(q);
        const int32_t* cnt = q.shadow_cnt[set] + 3 * (size_t)w;
        RayS y;
        ray_from(sh, y);
        copy_ray(*R.V, i, y);
        ray_from(sh + 17, y);
        copy_ray(*R.C, i, y);
        ray_from(sh + 34, y);
        copy_ray(*R.X, i, y);
        R.V->surface[i] = R.C->surface[i] = R.X->surface[i] = cnt[0];
        R.V->bottom[i] = R.C->bottom[i] = R.X->bottom[i] = cnt[1];
        /* with the caustic hand-off k_advance found before the reflection */
        const bool fold = (b & COMMIT_FOLD) != 0;
        R.X->caustic[i] = cnt[2] + (fold ? 1 : 0);
        const double* ph = sh + (fold ? 54 + 2 * q.nf : 51 + q.nf);
        for (int f = 0; f < q.nf; ++f) {
            R.X->atten[(size_t)f * q.n + i] = sh[51 + f];
            R.X->phase[(size_t)f * q.n + i] = ph[f];
        }
        if (q.sens)
            for (int j = 0; j < 3; ++j) R.X->dA[(size_t)j * q.n + i] += sh[51 + 2 * q.nf + j];
        return;
    }
    if (b & COMMIT_FOLD) {
        R.X->caustic[i] += 1;
        for (int f = 0; f < q.nf; ++f) R.X->phase[(size_t)f * q.n + i] -= M_PI_2;
    }
    if (b & COMMIT_UPPER) R.X->upper[i] += 1;
    if (b & COMMIT_LOWER) R.X->lower[i] += 1;
}

/* Volume-layer eigenverbs of the rays that do not reflect in step s
 * (wave_queue.cc:202; k_reflect handles the reflecting ones).  Launched
 * before k_advance of the same step, only when an eigenverb listener is
 * installed and the ocean has volume layers. */
__global__ void __launch_bounds__(128) k_volume(__grid_constant__ const QueueDev q, int k) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= q.n) return;
    const int64_t s = *q.d_base + k;
    if (q.flag[s & 1][i]) return;
    Roles R;
    roles_at(q, s, R);
    const double rc = R.C->pos[0][i], rx = R.X->pos[0][i];
    bool cross = false;
    for (int v = 0; v < q.oc.nvol; ++v) cross |= (q.oc.vol_rho[v] - rx) * (q.oc.vol_rho[v] - rc) < 0;
    if (!cross) return;
    RayC y0, y1, y2;
    load_rayc(*R.V, i, y0);
    load_rayc(*R.C, i, y1);
    load_rayc(*R.X, i, y2);
    int seq = 0;
    volume_scatter(q, *R.C, i, s + 1, q.d_times[k], y0, y1, y2, R.C->surface[i], R.C->bottom[i], seq);
}

/* ------------------------------------------------------------------ */
/* CPA search (wave_queue.cc:351-488)                                  */
/* ------------------------------------------------------------------ */
namespace {

struct TgtS {
    double th, ph, sn, R2, twoR;
};

__device__ __forceinline__ double d2_at(const FrontPtrs& f, int i, const TgtS& t) {
    const double rho = f.cpa[0][i];
    return target_distance2(rho, rho * rho, f.cpa[1][i], f.cpa[2][i], f.cpa[3][i],
                            t.th, t.ph, t.sn, t.R2, t.twoR);
}

/* appends (target, ray) to the candidate list of the step at s */
__device__ __forceinline__ void cand_push(const QueueDev& q, int64_t s, uint32_t t, uint32_t i) {
    const int l = cand_list(s);
    const uint32_t slot = atomicAdd(q.n_cand + l, 1u);
    if (slot < q.cap_cand) {
        uint32_t* c = q.cand + (size_t)l * 2 * q.cap_cand;
        c[2 * slot] = t;
        c[2 * slot + 1] = i;
    } else {
        set_err(q, ERR_CAND_OVERFLOW);
    }
}

__device__ __forceinline__ int wrap_az(const QueueDev& q, int az, int na) {
    int a = az + na - 1;
    if (q.az_boundary) {
        if (az + na == 0) {
            a = q.naz - 2;
        } else if (a >= q.naz - 1) {
            a = 0;
        }
    }
    return a;
}

/* is_closest_ray (wave_queue.cc:411-488).  The reference tests each
 * neighbour on the curr, next and prev fronts in turn and stops at the first
 * that fails; the order does not matter, so the curr front goes first, where
 * most pairs fail, with the loads of all eight neighbours in flight at once
 * (one after another with an early exit, 32 pairs took 12,000 cycles). */
__device__ __forceinline__ bool is_closest(const QueueDev& q, const FrontPtrs& V, const FrontPtrs& C,
                                           const FrontPtrs& X, const TgtS& t, bool de_branch, int de,
                                           int az, double center) {
    const int max_az = q.naz - 1;
    double d[9];
    unsigned compared = 0; /* neighbours that take part */
#pragma unroll
    for (int nb = 0; nb < 9; ++nb) {
        if (nb == 4) continue;
        const int a = wrap_az(q, az, nb % 3);
        const int i = (de + nb / 3 - 1) * q.naz + a;
        const bool edge = C.on_edge[i] != 0;
        d[nb] = d2_at(C, i, t);
        const bool skip = (a == 0 && !q.az_boundary) || a == max_az || ((de_branch || nb / 3 != 1) && edge);
        compared |= skip ? 0u : 1u << nb;
    }
    bool fails = false;
#pragma unroll
    for (int nb = 0; nb < 9; ++nb) {
        if (nb == 4) continue;
        const bool after = nb / 3 == 2 || nb % 3 == 2;
        const bool nearer = d[nb] < center || (after && !de_branch && d[nb] == center) || (after && de_branch && az != 0);
        fails |= nearer && ((compared >> nb) & 1u);
    }
    if (fails) return false;
    for (int nb = 0; nb < 9; ++nb) {
        if (!((compared >> nb) & 1u)) continue;
        const int i = (de + nb / 3 - 1) * q.naz + wrap_az(q, az, nb % 3);
        if (d2_at(X, i, t) <= center || d2_at(V, i, t) < center) return false;
    }
    return true;
}

}  // namespace

/* ------------------------------------------------------------------ */
/* CPA search: a warp of neighbouring rays against clusters of targets   */
/* ------------------------------------------------------------------ */
/* A pair (ray, target) is kept when the ray is nearest the target on the
 * curr front among its prev and next selves (wave_queue.cc:386-393) and its
 * neighbours (is_closest_ray).  Each comparison is the sign of a difference
 * of two distance2 values.  With coordinates relative to a reference ray (r
 * = rho - rho0, x = theta - theta0, y = phi - phi0; target Rr, X, Y
 * likewise) the reference's distance2 is, in exact arithmetic,
 *     Rr^2 + sum_k w_k(target) q_k(ray)
 *     q = (r^2, rho, rho x^2, rho x, rho s y^2, rho s y, rho s)
 *     w = (1, R X^2 - 2 Rr, R, -2 R X, R S, -2 R S Y, R S Y^2)
 * (s = sin theta, S = sin Theta), so the difference of a point (the ray on
 * another front, or a neighbour) from the ray on the curr front is sum_k
 * w_k dq_k, with seven features dq_k per ray that do not depend on the
 * target.
 *
 * One warp holds a patch of 32 neighbouring rays (QueueDev::patches) and
 * works without block barriers.  Six differences can each reject a target
 * for every ray of the patch, when an upper bound of theirs is negative:
 * the AZ neighbours' (next, prev), the next and prev fronts', and the D/E
 * neighbours'.  They are bounded
 *   per cluster  of 32 targets near one another, one lane each, from the
 *                patch's feature ranges and the cluster's centre and
 *                extents: the AZ neighbours first, which leave most patches
 *                nothing, before the other fronts are even read;
 *   per target   of a surviving cluster, one lane each.
 * The (patch, target) items that remain go to a list, and k_cpa_items
 * decides their 32 pairs by the FP64 distances, a warp an item: a few
 * patches hold nearly all of them, and one warp that worked through its own
 * took ten times as long as the rest of the launch.  The bounds only reject
 * what those comparisons reject, so they change no result; under
 * WQ3D_CHECKED the FP64 form takes every target of every patch instead.
 * A target at the source's latitude and longitude compares its neighbours
 * by other rules (de_branch); it and its cluster skip the neighbour bounds.
 *
 * Bounds.  With mid m_k and half-width h_k of dq_k over the patch's rays,
 * sum_k w_k m_k + |w_k| h_k is at least every ray's value; a cluster's
 * weights differ from its centre's by at most D_k, which adds sum_k D_k
 * (|m_k| + h_k).  Features are formed in FP32 from FP64 coordinate
 * differences; with A_k the sum of the magnitudes of dq_k's terms over the
 * patch and W_k the largest |w_k| of all targets, their rounding and the
 * weights' is below 8 u A_k W_k (u = 2^-24) and that of the 14 products and
 * sums of a bound below 17 u of 2 sum_k W_k A_k: the guards take 96 u, and
 * 192 u where a cluster's extents enter.  All add c0 = max(1 m^2, 4e-15 (rho^2 + R^2)) for
 * the rounding of the reference's FP64 expression on the two points (each
 * within 5 x 2^-53 (rho^2 + R^2), 0.05 m^2 at earth radius).  A NaN in a ray
 * makes its patch's bounds NaN, which reject nothing; targets with a NaN or
 * infinite coordinate are not searched (cpa_targets).
 *
 * Why this shape: per pair the search costs what the bounds let through.
 * On the sloped workload (1801 x 91 rays, 1024 targets, step 100) the two
 * fronts alone leave 33 targets per patch, the D/E neighbours 7.9 and the AZ
 * neighbours 1.7, in 6 % of the patches; a 16 x 8 patch with the fronts
 * alone, one thread per ray and all targets bounded one by one, left 348.
 * A launch is then bound by the latency of reading the rays and forming
 * their ranges: 29 us there and 18 us later on, where nothing survives, with
 * 4.6 us of k_cpa_items (ncu), for 94 to 103 us before; 264 -> 43 us in the
 * FP64 form (907 x 53 rays, 667 targets), 1,880 -> 170 us on the
 * reverberation workload (3601 x 181 rays, 4096 targets). */
namespace {
constexpr int CPA_K = 7; /* features */
enum { CPA_ANEXT, CPA_APREV, CPA_NEXT, CPA_PREV, CPA_DNEXT, CPA_DPREV, CPA_TESTS };

struct CpaWarp {
    float m[CPA_TESTS][8], h[CPA_TESTS][8]; /* feature mid and half-width of each difference */
    float guard[CPA_TESTS];                 /* sum_k W_k A_k; infinite where not comparable  */
};

/* the ray of a lane of a patch */
struct CpaLane {
    int de, az, i;
    bool inside, active;
};

__device__ __forceinline__ CpaLane cpa_lane(const QueueDev& q, const FrontPtrs& C, const CpaPatch& P, int lane) {
    CpaLane o;
    o.de = P.de + (lane >> P.shift);
    o.az = P.az + (lane & ((1 << P.shift) - 1));
    o.inside = o.de < q.nde && o.az < q.naz;
    o.i = o.inside ? o.de * q.naz + o.az : P.de * q.naz + P.az;
    o.active = o.inside && o.de >= 1 && o.de < q.nde - 1 && o.az >= (q.az_boundary ? 0 : 1) && o.az < q.naz - 1 &&
               !C.on_edge[o.i];
    return o;
}

/* decides the pairs of target j and the rays "rays" (lanes) of a patch by
 * the FP64 distances; called by a whole warp */
__device__ __forceinline__ void cpa_item(const QueueDev& q, int64_t s, const FrontPtrs& V, const FrontPtrs& C,
                                         const FrontPtrs& X, const CpaPatch& P, uint32_t j, unsigned rays, int lane) {
    const CpaLane L = cpa_lane(q, C, P, lane);
    const TgtS t{q.tgt[1][j], q.tgt[2][j], q.tgt_sin[j], q.tgt_R2[j], q.tgt_2R[j]};
    const bool branch = q.de_branch[j] != 0;
    const double center = d2_at(C, L.i, t), next = d2_at(X, L.i, t), prev = d2_at(V, L.i, t);
    const int pa = 1 << P.shift;
    bool hit = L.active && ((rays >> lane) & 1u) && !(next <= center) && !(prev < center);
    /* the neighbours in the patch, before is_closest loads them all */
    const double dn = __shfl_down_sync(0xffffffffu, center, pa), dp = __shfl_up_sync(0xffffffffu, center, pa);
    const unsigned ok = __ballot_sync(0xffffffffu, L.inside && !C.on_edge[L.i]);
    if (!branch && lane + pa < 32 && ((ok >> (lane + pa)) & 1u) && dn <= center) hit = false;
    if (!branch && lane >= pa && ((ok >> (lane - pa)) & 1u) && dp < center) hit = false;
    if (hit && is_closest(q, V, C, X, t, branch, L.de, L.az, center)) cand_push(q, s, j, (uint32_t)L.i);
}

/* smallest and largest of a warp's values (NaN if any is NaN) */
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm("redux.sync.min.NaN.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm("redux.sync.max.NaN.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

/* a ray on the curr front, relative to the reference */
struct CpaRay {
    double rho, th, ph, rs;
    float r, x, y;
};

/* features of point i of front f minus those of the ray; dx, dy: its
 * theta and phi differences */
__device__ __forceinline__ void feature_diff(const FrontPtrs& f, int i, const CpaRay& c, float* d, float* dx,
                                             float* dy) {
    const double rho = f.cpa[0][i];
    const double rs = rho * f.cpa[3][i];
    const float dr = (float)(rho - c.rho), ds = (float)(rs - c.rs);
    const float tx = (float)(f.cpa[1][i] - c.th), ty = (float)(f.cpa[2][i] - c.ph);
    const float R = (float)rho, S = (float)rs;
    d[0] = dr * fmaf(2.0f, c.r, dr);
    d[1] = dr;
    d[2] = fmaf(R * tx, fmaf(2.0f, c.x, tx), c.x * c.x * dr);
    d[3] = fmaf(R, tx, c.x * dr);
    d[4] = fmaf(S * ty, fmaf(2.0f, c.y, ty), c.y * c.y * ds);
    d[5] = fmaf(S, ty, c.y * ds);
    d[6] = ds;
    *dx = tx;
    *dy = ty;
}

/* a point's weights from R, R S and its offsets from the reference */
__device__ __forceinline__ void target_weights(double R, double RS, double Rr, double X, double Y, float* w) {
    w[0] = 1.0f;
    w[1] = (float)(R * X * X - 2.0 * Rr);
    w[2] = (float)R;
    w[3] = (float)(-2.0 * R * X);
    w[4] = (float)RS;
    w[5] = (float)(-2.0 * RS * Y);
    w[6] = (float)(RS * Y * Y);
}

/* the bound's two sums for weights w */
__device__ __forceinline__ float range_bound(const float* w, const float* m, const float* h) {
    float a = m[0] + h[0], b = 0.0f;
#pragma unroll
    for (int k = 1; k < CPA_K; ++k) {
        a = fmaf(w[k], m[k], a);
        b = fmaf(fabsf(w[k]), h[k], b);
    }
    return a + b;
}

/* The ranges of a difference over the lanes "mine" into the warp's slot n,
 * with its guard; xm, ym, rm: the largest |x|, |y|, |r| of the patch.  Where
 * a lane of "mine" is not "comparable" the difference rejects nothing. */
__device__ __forceinline__ void set_range(CpaWarp& S, int n, bool mine, bool comparable, const float* d, float dx,
                                          float dy, const float* W, float rm, float xm, float ym, int lane) {
    float mx[CPA_K], hx[CPA_K];
#pragma unroll
    for (int k = 0; k < CPA_K; ++k) {
        const float lo = warp_min(mine ? d[k] : INFINITY), hi = warp_max(mine ? d[k] : -INFINITY);
        mx[k] = 0.5f * (lo + hi);
        hx[k] = 1.000001f * fmaxf(hi - mx[k], mx[k] - lo);
    }
    const float dxm = warp_max(mine ? fabsf(dx) : 0.0f), dym = warp_max(mine ? fabsf(dy) : 0.0f);
    const float drm = fabsf(mx[1]) + hx[1], dsm = fabsf(mx[6]) + hx[6];
    /* A_k: W[2] and W[4] stand for rho and rho sin(theta), which are the
     * targets' R to within a factor of two */
    float g = drm * fmaf(2.0f, rm, drm);
    g = fmaf(W[1], drm, g);
    g = fmaf(W[2], 2.0f * W[2] * dxm * fmaf(2.0f, xm, dxm) + xm * xm * drm, g);
    g = fmaf(W[3], 2.0f * W[2] * dxm + xm * drm, g);
    g = fmaf(W[4], 2.0f * W[2] * dym * fmaf(2.0f, ym, dym) + ym * ym * dsm, g);
    g = fmaf(W[5], 2.0f * W[2] * dym + ym * dsm, g);
    g = fmaf(W[6], dsm, g);
    if (__any_sync(0xffffffffu, mine && !comparable)) g = INFINITY;
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < CPA_K; ++k) {
            S.m[n][k] = mx[k];
            S.h[n][k] = hx[k];
        }
        S.guard[n] = g;
    }
}

/* a cluster's centre weights and the most its targets' differ by */
struct ClusterW {
    float w[8], D[8];
    bool branch;
};

__device__ __forceinline__ void cluster_weights(const TgtCluster& cl, double rho0, double th0, double ph0,
                                                ClusterW& o) {
    const double Xo = cl.T - th0, Yo = cl.P - ph0;
    target_weights(cl.R, cl.RS, cl.R - rho0, Xo, Yo, o.w);
    const float ax = fabsf((float)Xo), ay = fabsf((float)Yo);
    const float Rt = o.w[2] + cl.dR, St = fabsf(o.w[4]) + cl.dRS;
    o.D[1] = fmaf(2.0f, cl.dR, fmaf(Rt * cl.dT, fmaf(2.0f, ax, cl.dT), ax * ax * cl.dR));
    o.D[2] = cl.dR;
    o.D[3] = 2.0f * fmaf(Rt, cl.dT, ax * cl.dR);
    o.D[4] = cl.dRS;
    o.D[5] = 2.0f * fmaf(St, cl.dP, ay * cl.dRS);
    o.D[6] = fmaf(St * cl.dP, fmaf(2.0f, ay, cl.dP), ay * ay * cl.dRS);
    o.branch = cl.branch != 0;
}

constexpr float CPA_U = 5.9604645e-8f; /* 2^-24 */

/* whether difference n may be non-negative for some ray and some target of
 * the cluster */
__device__ __forceinline__ bool cluster_keeps(const CpaWarp& S, int n, const ClusterW& c, float c0) {
    float b = 0.0f;
#pragma unroll
    for (int k = 1; k < CPA_K; ++k) b = fmaf(c.D[k], fabsf(S.m[n][k]) + S.h[n][k], b);
    b = fmaf(1.001f, b, range_bound(c.w, S.m[n], S.h[n]));
    return !(b + fmaf(192.0f * CPA_U, S.guard[n], 1.001f * c0) < 0.0f);
}

__device__ __forceinline__ bool target_keeps(const CpaWarp& S, int n, const float* w, float c0) {
    return !(range_bound(w, S.m[n], S.h[n]) + fmaf(96.0f * CPA_U, S.guard[n], 1.001f * c0) < 0.0f);
}
}  // namespace

/* four blocks per SM (128 registers) */
__global__ void __launch_bounds__(32 * CPA_WARPS, 4) k_cpa(__grid_constant__ const QueueDev q, int k) {
    __shared__ CpaWarp shared[CPA_WARPS];
    const int64_t s = *q.d_base + k + 1;
    const FrontPtrs& V = q.F[ring_slot(s + 1)];
    const FrontPtrs& C = q.F[ring_slot(s + 2)];
    const FrontPtrs& X = q.F[ring_slot(s + 3)];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wid = blockIdx.x * CPA_WARPS + warp;
    if (wid >= q.n_patch) return; /* a whole warp: no block barrier follows */
    CpaWarp& S = shared[warp];
    const CpaPatch P = q.patches[wid];
    const int pa = 1 << P.shift;
    const CpaLane L = cpa_lane(q, C, P, lane);
    const int az = L.az, i = L.i;
    const bool inside = L.inside, active = L.active;
    if (!__any_sync(0xffffffffu, active)) return;

    /* local coordinates about the patch's middle ray */
    const int i_ref = min(P.de + (16 >> P.shift), q.nde - 1) * q.naz + min(P.az + pa / 2, q.naz - 1);
    const double rho0 = C.cpa[0][i_ref], th0 = C.cpa[1][i_ref], ph0 = C.cpa[2][i_ref];
    CpaRay ray;
    ray.rho = C.cpa[0][i];
    ray.th = C.cpa[1][i];
    ray.ph = C.cpa[2][i];
    ray.rs = ray.rho * C.cpa[3][i];
    ray.r = (float)(ray.rho - rho0);
    ray.x = (float)(ray.th - th0);
    ray.y = (float)(ray.ph - ph0);
    const float rm = warp_max(active ? fabsf(ray.r) : 0.0f);
    const float xm = warp_max(active ? fabsf(ray.x) : 0.0f);
    const float ym = warp_max(active ? fabsf(ray.y) : 0.0f);
    /* largest weights of all targets */
    float W[8];
    {
        const float Xm = (float)fmax(fabs(q.tgt_box[2] - th0), fabs(q.tgt_box[3] - th0));
        const float Ym = (float)fmax(fabs(q.tgt_box[4] - ph0), fabs(q.tgt_box[5] - ph0));
        const float Rm = (float)fmax(fabs(q.tgt_box[0] - rho0), fabs(q.tgt_box[1] - rho0));
        const float R = 1.0001f * fmaxf((float)q.tgt_box[1], (float)rho0);
        W[1] = 1.0001f * (R * Xm * Xm + 2.0f * Rm);
        W[2] = W[4] = R;
        W[3] = 2.0f * R * Xm;
        W[5] = 2.0f * R * Ym;
        W[6] = 1.0001f * R * Ym * Ym;
    }
    const float c0 = fmaxf(1.0f, 4.0e-15f * ((float)rho0 * (float)rho0 + W[2] * W[2]));

    /* The AZ neighbours that is_closest compares the ray with: all but the
     * first and last ray of a fan that does not wrap. */
    {
        float d[8], dx, dy;
        const int an = active ? wrap_az(q, az, 2) : az, ap = active ? wrap_az(q, az, 0) : az;
        const int row = i - (inside ? az : P.az);
        feature_diff(C, inside ? row + an : i, ray, d, &dx, &dy);
        set_range(S, CPA_ANEXT, active, an != q.naz - 1 && (an != 0 || q.az_boundary), d, dx, dy, W, rm, xm, ym, lane);
        feature_diff(C, inside ? row + ap : i, ray, d, &dx, &dy);
        set_range(S, CPA_APREV, active, ap != q.naz - 1 && (ap != 0 || q.az_boundary), d, dx, dy, W, rm, xm, ym, lane);
    }
    __syncwarp();
    /* this warp's share of the clusters; nothing more to do for most warps */
    const int ncl = (q.n_cpa_tgt + 31) >> 5;
    const int per = (ncl + P.parts - 1) / P.parts;
    const int c_begin = P.part * per, c_end = min(ncl, c_begin + per);
    {
        bool keep = false;
        for (int c = c_begin + lane; c < c_end && !keep; c += 32) {
            ClusterW cw;
            cluster_weights(q.clusters[c], rho0, th0, ph0, cw);
            keep = cw.branch || (cluster_keeps(S, CPA_ANEXT, cw, c0) && cluster_keeps(S, CPA_APREV, cw, c0));
        }
#if WQ3D_CHECKED
        keep = keep || q.precision == WQ3D_FP64;
#endif
        if (!__any_sync(0xffffffffu, keep)) return;
    }

    /* the ray on the next and prev fronts, and its D/E neighbours (those on
     * an edge are not compared) */
    float dx[8], dv[8], dn[8], dp[8], tx[4], ty[4];
    feature_diff(X, i, ray, dx, &tx[0], &ty[0]);
    feature_diff(V, i, ray, dv, &tx[1], &ty[1]);
    const int in = active ? i + q.naz : i, ip = active ? i - q.naz : i;
    feature_diff(C, in, ray, dn, &tx[2], &ty[2]);
    feature_diff(C, ip, ray, dp, &tx[3], &ty[3]);
    const bool edge_n = C.on_edge[in] != 0, edge_p = C.on_edge[ip] != 0;

    /* appends the items of this patch's rays "rays" and the lanes' targets
     * to the step's list; one that finds no room is decided here */
    const int list = (int)(s & 1);
    const unsigned lt = (1u << lane) - 1u;
    auto append = [&](bool want, uint32_t t, unsigned rays) {
        unsigned mask = __ballot_sync(0xffffffffu, want);
        if (!mask) return;
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(q.n_item + list, (uint32_t)__popc(mask));
        base = __shfl_sync(0xffffffffu, base, 0);
        const uint32_t slot = base + (uint32_t)__popc(mask & lt);
        const bool fits = slot < q.cap_item;
        if (want && fits) q.items[slot] = make_uint4((uint32_t)wid, t, rays, 0u);
        mask = __ballot_sync(0xffffffffu, want && !fits);
        while (mask) {
            const uint32_t tl = __shfl_sync(0xffffffffu, t, __ffs(mask) - 1);
            mask &= mask - 1;
            cpa_item(q, s, V, C, X, P, tl, rays, lane);
        }
    };
#if WQ3D_CHECKED
    if (q.precision == WQ3D_FP64) {
        for (int j0 = c_begin * 32; j0 < min(q.n_cpa_tgt, c_end * 32); j0 += 32) {
            const int j = j0 + lane;
            append(j < q.n_cpa_tgt, j < q.n_cpa_tgt ? q.cpa_index[j] : 0u, 0xffffffffu);
        }
        return;
    }
#endif

    /* Rays that have just met a boundary move unlike their neighbours, and
     * one range over both would let most targets through: where the radial
     * parts of a patch's steps differ by more than 0.3 of its longest step,
     * the rays on either side of the middle are searched on their own. */
    int key = 0;
    {
        const float len = warp_max(active ? fmaxf(fabsf(dx[1]), fmaxf(fabsf(dx[3]), fabsf(dx[5]))) : 0.0f);
        const float lx = warp_min(active ? dx[1] : INFINITY), hx = warp_max(active ? dx[1] : -INFINITY);
        const float lv = warp_min(active ? dv[1] : INFINITY), hv = warp_max(active ? dv[1] : -INFINITY);
        if (hx - lx > 0.3f * len && dx[1] > 0.5f * (lx + hx)) key |= 1;
        if (hv - lv > 0.3f * len && dv[1] > 0.5f * (lv + hv)) key |= 2;
    }

    unsigned left = __ballot_sync(0xffffffffu, active);
    while (left) {
        const int lead = __shfl_sync(0xffffffffu, key, __ffs(left) - 1); /* every lane takes part */
        const bool mine = active && key == lead;
        const unsigned group = __ballot_sync(0xffffffffu, mine);
        left &= ~group;
        __syncwarp();
        set_range(S, CPA_NEXT, mine, true, dx, tx[0], ty[0], W, rm, xm, ym, lane);
        set_range(S, CPA_PREV, mine, true, dv, tx[1], ty[1], W, rm, xm, ym, lane);
        set_range(S, CPA_DNEXT, mine, !edge_n, dn, tx[2], ty[2], W, rm, xm, ym, lane);
        set_range(S, CPA_DPREV, mine, !edge_p, dp, tx[3], ty[3], W, rm, xm, ym, lane);
        __syncwarp();
        for (int cb = c_begin; cb < c_end; cb += 32) {
            bool keep = false;
            if (cb + lane < c_end) {
                ClusterW cw;
                cluster_weights(q.clusters[cb + lane], rho0, th0, ph0, cw);
                keep = cluster_keeps(S, CPA_NEXT, cw, c0) && cluster_keeps(S, CPA_PREV, cw, c0);
                if (keep && !cw.branch)
                    keep = cluster_keeps(S, CPA_ANEXT, cw, c0) && cluster_keeps(S, CPA_APREV, cw, c0) &&
                           cluster_keeps(S, CPA_DNEXT, cw, c0) && cluster_keeps(S, CPA_DPREV, cw, c0);
            }
            unsigned cmask = __ballot_sync(0xffffffffu, keep);
            while (cmask) {
                const int j = ((cb + __ffs(cmask) - 1) << 5) + lane;
                cmask &= cmask - 1;
                bool want = false;
                uint32_t t = 0;
                if (j < q.n_cpa_tgt) {
                    const double2 a = __ldg(reinterpret_cast<const double2*>(q.cpa_tgt) + 2 * (size_t)j);
                    const double2 b = __ldg(reinterpret_cast<const double2*>(q.cpa_tgt) + 2 * (size_t)j + 1);
                    t = __ldg(q.cpa_index + j);
                    float w[8];
                    target_weights(a.x, a.x * b.y, a.x - rho0, a.y - th0, b.x - ph0, w);
                    want = target_keeps(S, CPA_NEXT, w, c0) && target_keeps(S, CPA_PREV, w, c0);
                    if (want && q.de_branch[t] == 0)
                        want = target_keeps(S, CPA_ANEXT, w, c0) && target_keeps(S, CPA_APREV, w, c0) &&
                               target_keeps(S, CPA_DNEXT, w, c0) && target_keeps(S, CPA_DPREV, w, c0);
                }
                append(want, t, group);
            }
        }
    }
}

/* the items that k_cpa left, a warp each */
__global__ void __launch_bounds__(128) k_cpa_items(__grid_constant__ const QueueDev q, int k) {
    const int64_t s = *q.d_base + k + 1;
    const FrontPtrs& V = q.F[ring_slot(s + 1)];
    const FrontPtrs& C = q.F[ring_slot(s + 2)];
    const FrontPtrs& X = q.F[ring_slot(s + 3)];
    const int lane = threadIdx.x & 31;
    const uint32_t n = min(q.n_item[s & 1], q.cap_item);
    for (uint32_t e = blockIdx.x * 4 + (threadIdx.x >> 5); e < n; e += gridDim.x * 4) {
        const uint4 it = q.items[e];
        WQ_CHECKED_OR(q, it.x < (uint32_t)q.n_patch && it.y < (uint32_t)q.nt, continue);
        cpa_item(q, s, V, C, X, q.patches[it.x], it.y, it.z, lane);
    }
    /* the next step's count (its k_cpa follows this launch on the stream;
     * the step before last used it) */
    if (blockIdx.x == 0 && threadIdx.x == 0) q.n_item[(s + 1) & 1] = 0;
}

/* ------------------------------------------------------------------ */
/* eigenray construction (wave_queue.cc:495-977 + spreading models)    */
/* ------------------------------------------------------------------ */
namespace {

/* One warp builds one eigenray (with a second warp for the AZ walks of
 * hybrid Gaussian spreading).  Lanes share the parallel parts (the 27
 * distance2 values, the 54 direction angles, the cell widths and Gaussian
 * terms of the beam walks, the per-frequency sums); every value that feeds
 * a rounding-sensitive recurrence (cell distances, the running intensity
 * and its threshold test) is formed in the reference's sequential order,
 * so results equal the one-thread-per-eigenray evaluation.
 *
 * A step has few candidates, and the next step's commit waits for them, so
 * what counts is one candidate's latency.  A cell's width is up to four
 * distances of four sines each, 200 cycles a sine: one pass forms the widths
 * of the cells on either side of the ray, lanes sharing the sines of their
 * common ray, where most walks end (three passes of 32 before).  The
 * recurrences run on every lane from widths and terms in shared memory, two
 * additions a cell, instead of five shuffles; the terms that the threshold
 * test needs are those that the lowest frequency adds; and divisions are
 * branch-free.  Per launch, with the event timing's overhead: 29.7 -> 24.3 us
 * (Munk workload, one or two candidates a step), 65 -> 46 us (sloped
 * workload, 907 x 53 rays); with more than EIG_FG frequencies, whose sums
 * dominate, as before (first_cells), and with more candidates than the GPU
 * holds 209 -> 227 us (49 x 32 rays, 1,660 eigenrays a step). */
constexpr int EIG_FG = 8;    /* frequencies per pass of a walk chunk's Gaussian terms */
constexpr int EIG_SIDE = 16; /* cells on a side whose widths the first pass forms     */

struct WarpBuild {
    const QueueDev* q;
    const FrontPtrs* pV;
    const FrontPtrs* pC;
    const FrontPtrs* pX;
    const double* spread2;   /* [nf] for this target */
    int lane;
    double Ilo, Ihi;         /* running intensity of frequencies lane, lane+32 */
    double (*sg)[EIG_FG + 1]; /* this warp's [cell][frequency] Gaussian terms */
    double* sw;               /* this warp's cell widths: [32], of the first pass the lower side's */
    double* su;               /* [16] and the upper side's                    */
    double u, v;              /* the walk's offset in time and across, in spacings */
    const FrontPtrs* p2;      /* the front that the time offset leads to      */

    static __device__ __forceinline__ double sine(double x) {
        double s, c;
        sin_cos(x, &s, &c);
        return s;
    }
    /* wvector1::distance of two rays whose sines of theta are known */
    static __device__ __forceinline__ double dist(double r1, double t1, double p1, double s1, double r2, double t2,
                                                  double p2, double s2) {
        const double st = sine(0.5 * (t1 - t2));
        const double sp = sine(0.5 * (p1 - p2));
        const double dn = 1.0 - 2.0 * (st * st + s1 * s2 * sp * sp);
        const double dot = r1 * r2 * dn;
        return sqrt(fabs(r1 * r1 + r2 * r2 - 2.0 * dot));
    }
    __device__ double fdist(const FrontPtrs& f, int d1, int a1, int d2, int a2) const {
        const int i = d1 * q->naz + a1, j = d2 * q->naz + a2;
        const double t1 = f.pos[1][i], t2 = f.pos[1][j];
        return dist(f.pos[0][i], t1, f.pos[2][i], sine(t1), f.pos[0][j], t2, f.pos[2][j], sine(t2));
    }
    /* the same for rays (d, a) and (d + 1, a), where lane "next" has d + 1;
     * called by a whole warp */
    __device__ double fdist_de(const FrontPtrs& f, int d, int a, int next) const {
        const int i = d * q->naz + a, j = min(d + 1, q->nde - 1) * q->naz + a;
        const double t1 = f.pos[1][i];
        const double s1 = sine(t1);
        const double s2 = __shfl_sync(0xffffffffu, s1, next);
        return dist(f.pos[0][i], t1, f.pos[2][i], s1, f.pos[0][j], f.pos[1][j], f.pos[2][j], s2);
    }
    __device__ double de_inc(int d) const { return q->de_inc[min(max(d, 0), q->nde - 1)]; }
    __device__ double az_inc(int a) const { return q->az_inc[min(max(a, 0), q->naz - 1)]; }

    /* spreading_hybrid_gaussian.h:148-153 for one frequency */
    __device__ double gauss(double d, double w, double A, int f) const {
        const double bw = spread2[f] + 2.0 * 2.0 * w * w;
        const double e = -0.5 * d * d, s = sqrt(bw);
        if (divisor_ok(bw) && divisor_ok(s) && dividend_ok(e)) {
            const double g = exp(quot(e, recip(bw)));
            return (dividend_ok(g) ? quot(g, recip(s)) : g / s) * A;
        }
        return exp(e / bw) / s * A;
    }
    /* running intensity += gaussian, frequencies spread over the lanes */
    __device__ void acc(double d, double w, double A, bool first) {
        const int nf = q->nf;
        if (lane < nf) {
            const double g = gauss(d, w, A, lane);
            Ilo = first ? g : Ilo + g;
        }
        if (lane + 32 < nf) {
            const double g = gauss(d, w, A, lane + 32);
            Ihi = first ? g : Ihi + g;
        }
    }
    __device__ double I0() const { return __shfl_sync(0xffffffffu, Ilo, 0); }

    /* Cells 0..nend-1 of a walk, whose distance, width and normalisation
     * lane k holds for cell k: the reference's threshold test on the lowest
     * frequency's running intensity after each cell (new / old <
     * 1.002305238), then every frequency's sum over the cells up to the first
     * that passes, or all; both in cell order.  The sums are sequential; the
     * divisions of the tests are not, so they run on all lanes at once.
     * Returns the first cell that passes the test, or -1. */
    __device__ int add_cells(int nend, double cd, double cw, double nm) {
        const int nf = q->nf;
        int last = nend - 1, hit_cell = -1;
        for (int f0 = 0; f0 < nf; f0 += EIG_FG) {
            const int nfg = min(EIG_FG, nf - f0);
            if (lane <= last)
                for (int j = 0; j < nfg; ++j) sg[lane][j] = gauss(cd, cw, nm, f0 + j);
            __syncwarp();
            if (f0 == 0) {
                double i0 = I0(), my_new = 1.0, my_old = 1.0;
#pragma unroll 4
                for (int k = 0; k < nend; ++k) {
                    const double old = i0;
                    i0 += sg[k][0];
                    if (lane == k) {
                        my_new = i0;
                        my_old = old;
                    }
                }
                const unsigned hit = __ballot_sync(0xffffffffu, lane < nend && my_new / my_old < 1.002305238);
                if (hit) last = hit_cell = __ffs(hit) - 1;
            }
            if (lane >= f0 && lane < f0 + nfg) {
                double I = Ilo;
#pragma unroll 4
                for (int k = 0; k <= last; ++k) I = I + sg[k][lane - f0];
                Ilo = I;
            }
            if (lane + 32 >= f0 && lane + 32 < f0 + nfg) {
                double I = Ihi;
#pragma unroll 4
                for (int k = 0; k <= last; ++k) I = I + sg[k][lane + 32 - f0];
                Ihi = I;
            }
            __syncwarp();
        }
        return hit_cell;
    }

    /* u, v and p2 of a walk: |offset in time| over the step, |offset across|
     * over its spacing */
    __device__ void set_offsets(double dtime, double across, double spacing) {
        u = fabs(dtime) / q->dt;
        v = fabs(across) / spacing;
        p2 = (dtime < 0.0) ? pV : pX;
    }

    /* the blend of the four distances (spreading_hybrid_gaussian.cc:430-571) */
    template <class F>
    __device__ double width(bool cross, F column) const {
        double L1 = column(*pC, 0);
        const double length1 = cross ? (1.0 - v) * L1 + v * column(*pC, 1) : L1;
        if (u < 1e-10) return 0.5 * length1;
        L1 = column(*p2, 0);
        const double length2 = cross ? (1.0 - v) * L1 + v * column(*p2, 2) : L1;
        return 0.5 * ((1.0 - u) * length1 + u * length2);
    }

    /* spreading_hybrid_gaussian.cc:430-495; "next": the lane with ray d + 1
     * (a whole warp then calls it), or -1 */
    __device__ double width_de(int d, int a, int next) const {
        const int max_az = q->naz - 1;
        const int az_wrap = (a + 1 >= max_az) ? 0 : a + 1;
        return width(!(v < 1e-10), [&](const FrontPtrs& f, int side) {
            const int col = side == 0 ? a : side == 1 ? az_wrap : az_wrap + 1;
            return next < 0 ? fdist(f, d, col, d + 1, col) : fdist_de(f, d, col, next);
        });
    }

    /* spreading_hybrid_gaussian.cc:500-571 */
    __device__ double width_az(int d, int a) const {
        const int max_az = q->naz - 1;
        const int max_de = q->nde - 1;
        const int de_upper = (d + 1 >= max_de) ? max_de - 2 : d;
        const int az_wrap = (a + 1 > max_az) ? 0 : a + 1;
        return width(!(v < 1e-10 || fabs(v - 1.0) < 1e-10), [&](const FrontPtrs& f, int side) {
            const int row = side == 0 ? d : de_upper + 1;
            return fdist(f, row, a, row, az_wrap);
        });
    }

    /* Processes up to 32 cells of one walk, whose widths are w[0..ncell-1] in
     * shared memory.  Lane k holds whether cell k is a virtual ray (virt_k,
     * where the walk ends) and its two normalisation candidates.  sign = +1
     * for a walk away from the lower side, -1 for the upper.  Returns true
     * when the walk ends; *stop: the cell it passed the threshold on, if so. */
    __device__ bool run_cells(int ncell, const double* w, bool virt_k, double norm_k, double norm_virt_k,
                              double sign, double& cell_dist, double& cell_width, int* stop) {
        const unsigned virt = __ballot_sync(0xffffffffu, lane < ncell && virt_k);
        const int nend = virt ? __ffs(virt) : ncell; /* cells used; the last may be virtual */
        double my_cd = 0.0, my_cw = 0.0;
        double cd = cell_dist, cw = cell_width;
#pragma unroll 4
        for (int k = 0; k < nend; ++k) {
            const double wk = w[k];
            const bool keep = virt && k == nend - 1; /* a virtual ray keeps the width */
            cd = sign > 0.0 ? cd + cw : cd - cw;
            if (!keep) cw = wk;
            cd = sign > 0.0 ? cd + cw : cd - cw;
            if (lane == k) {
                my_cd = cd;
                my_cw = cw;
            }
        }
        cell_dist = cd;
        cell_width = cw;
        const int hit = add_cells(nend, my_cd, my_cw, virt && lane == nend - 1 ? norm_virt_k : norm_k);
        if (hit >= 0) *stop = hit;
        return hit >= 0 || virt != 0;
    }

    /* How many cells of a side the walk takes first: those whose widths the
     * first pass made, or all 32 where a cell's terms (one a frequency) cost
     * more than a second pass of widths, since most walks then go on beyond
     * 15 cells.  Per launch, 15 against 32 cells: 203 and 181 us with 64
     * frequencies on 383 x 7 rays, 197 and 189 with 32 on the reverberation
     * workload; 140 and 147 with 64 on 83 x 17 rays, whose walks are short.
     * With 8 or fewer (one group of EIG_FG) the shorter start is the faster. */
    __device__ int first_cells(int made) const { return q->nf > EIG_FG ? 32 : made; }

    /* widths of cells 0..ncell-1, lane k's by width(), but for the first
     * "have" that are at "made" */
    template <class F>
    __device__ const double* cell_widths(int have, const double* made, int ncell, bool skip, F width) {
        if (ncell <= have) return made;
        const double x = lane < have ? made[lane] : lane < ncell && !skip ? width() : 0.0;
        __syncwarp();
        sw[lane] = x;
        __syncwarp();
        return sw;
    }

    /* spreading_hybrid_gaussian.cc:124-258 */
    __device__ void intensity_de(int de0, int a, const double* offset, const double* distance) {
        const QueueDev& Q = *q;
        const FrontPtrs& C = *pC;
        set_offsets(offset[0], offset[2], az_inc(a));
        /* lanes 0-15: cells de0-1, de0-2, ...; lanes 16-30: cells de0, de0+1, ... */
        {
            const bool lower = lane < EIG_SIDE;
            const int d = lower ? max(de0 - 1 - lane, 0) : min(de0 + lane - EIG_SIDE, Q.nde - 1);
            const double w = width_de(d, a, lower ? (lane == 0 ? EIG_SIDE : lane - 1) : min(lane + 1, 31));
            if (lower)
                sw[lane] = w;
            else
                su[lane - EIG_SIDE] = w;
        }
        __syncwarp();
        const double wl = sw[0], wc = su[0];
        const double L = distance[1];
        acc(L - wc, wc, Q.norm_de[de0], true);
        acc(L + wl, wl, Q.norm_de[de0 - 1], false);
        if (I0() < 1e-10) return;
        int stop;
        /* lower D/E cells: de0-2 down to 0; "at" 1 while the first pass's
         * widths serve */
        double cell_width = wl, cell_dist = L + wl;
        for (int d0 = de0 - 2, at = 1; d0 >= 0; at = 0) {
            const int d = d0 - lane;
            const int ncell = min(at ? first_cells(EIG_SIDE - 1) : 32, d0 + 1);
            bool virt = false;
            double nm = 0.0, nmv = 0.0;
            if (lane < ncell) {
                virt = C.on_edge[(d + 1) * Q.naz + a] && C.on_edge[d * Q.naz + a];
                nm = Q.norm_de[d];
                nmv = Q.norm_de[d + 1];
            }
            const double* w = cell_widths(at ? EIG_SIDE - 1 : 0, sw + 1, ncell, virt, [&] { return width_de(d, a, -1); });
            if (run_cells(ncell, w, virt, nm, nmv, 1.0, cell_dist, cell_width, &stop)) break;
            d0 -= ncell;
        }
        /* upper D/E cells: de0+1 up to num_de-2 */
        cell_width = wc;
        cell_dist = L - wc;
        const int size = Q.nde - 1;
        for (int d0 = de0 + 1, at = 1; d0 < size; at = 0) {
            const int d = d0 + lane;
            const int ncell = min(at ? first_cells(EIG_SIDE - 2) : 32, size - d0);
            bool virt = false;
            double nm = 0.0, nmv = 0.0;
            if (lane < ncell) {
                virt = C.on_edge[(d + 1) * Q.naz + a] && C.on_edge[d * Q.naz + a];
                nm = Q.norm_de[d];
                nmv = Q.norm_de[d - 1];
            }
            const double* w = cell_widths(at ? EIG_SIDE - 2 : 0, su + 1, ncell, virt, [&] { return width_de(d, a, -1); });
            if (run_cells(ncell, w, virt, nm, nmv, -1.0, cell_dist, cell_width, &stop)) break;
            d0 += ncell;
        }
    }

    /* spreading_hybrid_gaussian.cc:264-425.  The duplicate mask of the
     * reference is a cyclic range: the lower walk marks a contiguous run of
     * AZ indices below the centre, so membership is a range test. */
    __device__ void intensity_az(int d, int az0, const double* offset, const double* distance) {
        const QueueDev& Q = *q;
        const FrontPtrs& C = *pC;
        const int max_de = Q.nde - 2;
        const int max_az = Q.naz - 1;
        const int az_lower = Q.az_boundary ? az0 : 0;
        const int az_upper = Q.az_boundary ? az0 : max_az - 1;
        auto norm = [&](int aa) { return (d >= max_de) ? Q.norm_az[1 * Q.naz + aa] : Q.norm_az[d * Q.naz + aa]; };
        const int a1 = (az0 < 1) ? max_az - 1 : az0 - 1;
        const int start = (a1 < 1) ? max_az - 1 : a1 - 1;
        set_offsets(offset[0], offset[1], de_inc(d));
        /* lanes 0-15: cells a1, then start, start-1, ... (cyclic); lanes
         * 16-31: cells az0, az0+1, ... (cyclic) */
        if (lane < EIG_SIDE)
            sw[lane] = width_az(d, lane == 0 ? a1 : (((start - (lane - 1)) % max_az) + max_az) % max_az);
        else
            su[lane - EIG_SIDE] = width_az(d, lane == EIG_SIDE ? az0 : (az0 + lane - EIG_SIDE) % max_az);
        __syncwarp();
        const double wl = sw[0], wc = su[0];
        const double L = distance[2];
        acc(L - wc, wc, norm(az0), true);
        acc(L + wl, wl, norm(a1), false);
        if (I0() < 1e-10) return;
        /* lower walk: a1-1, a1-2, ... (cyclic) until az_lower */
        double cell_width = wl, cell_dist = L + wl;
        int marked = -1; /* index (in walk order) of the last cell marked */
        bool done = false;
        for (int k0 = 0, at = 1; !done && k0 < max_az; at = 0) {
            const int len = at ? first_cells(EIG_SIDE - 1) : 32;
            const int k = k0 + lane;
            int a = start - k;
            a = ((a % max_az) + max_az) % max_az;
            /* per-cell stop tests, in the reference's order */
            int kind = 0; /* 0 process, 1 loop end (not marked), 2 marked stop */
            if (k >= max_az || a == az_lower) {
                kind = 1;
            } else if (a == az0 || a == a1) {
                kind = 1;
            } else if (C.on_edge[d * Q.naz + a]) {
                kind = 2;
            }
            const unsigned stopmask = __ballot_sync(0xffffffffu, kind != 0 && lane < len);
            int ncell = len, fk = 0;
            if (stopmask) {
                ncell = __ffs(stopmask) - 1;
                fk = __shfl_sync(0xffffffffu, kind, ncell);
            }
            const double nm = (lane < ncell) ? norm(a) : 0.0;
            const double* w = cell_widths(at ? EIG_SIDE - 1 : 0, sw + 1, ncell, false, [&] { return width_az(d, a); });
            int kst = -1;
            const bool brk = (ncell > 0) && run_cells(ncell, w, false, nm, nm, 1.0, cell_dist, cell_width, &kst);
            if (brk) {
                marked = k0 + kst; /* the threshold stop happens on a marked cell */
                done = true;
            } else {
                if (ncell > 0) marked = k0 + ncell - 1;
                if (stopmask) {
                    done = true;
                    if (fk == 2) marked = k0 + ncell; /* on_edge cells are marked, not used */
                }
            }
            k0 += len;
        }
        /* upper walk: az0+1, az0+2, ... (cyclic) until az_upper */
        cell_width = wc;
        cell_dist = L - wc;
        done = false;
        for (int k0 = 0, at = 1; !done && k0 < max_az; at = 0) {
            const int len = at ? first_cells(EIG_SIDE - 1) : 32;
            const int k = k0 + lane;
            const int a = (az0 + 1 + k) % max_az;
            int kind = 0;
            /* membership of the lower walk's marked cells: start-j, j <= marked */
            const int off = ((start - a) % max_az + max_az) % max_az;
            const bool dup = (a == az0) || (a == a1) || (marked >= 0 && off <= marked);
            if (k >= max_az || a == az_upper) {
                kind = 1;
            } else if (dup) {
                kind = 1;
            } else if (C.on_edge[d * Q.naz + a]) {
                kind = 1;
            }
            const unsigned stopmask = __ballot_sync(0xffffffffu, kind != 0 && lane < len);
            int ncell = len;
            if (stopmask) {
                ncell = __ffs(stopmask) - 1;
                done = true;
            }
            const double nm = (lane < ncell) ? norm(a) : 0.0;
            const double* w = cell_widths(at ? EIG_SIDE - 1 : 0, su + 1, ncell, false, [&] { return width_az(d, a); });
            int kst = -1;
            if (ncell > 0 && run_cells(ncell, w, false, nm, nm, -1.0, cell_dist, cell_width, &kst))
                done = true;
            k0 += len;
        }
    }

    /* wvector1::area on four points (types/wvector1.cc) */
    __device__ double area4(const FrontPtrs& f, int d, int a) const {
        double aa = fdist(f, d, a, d + 1, a);
        const double b = fdist(f, d, a, d + 1, a + 1);
        double c = fdist(f, d + 1, a, d + 1, a + 1);
        const double area1 = 0.25 * sqrt((aa + b + c) * (b + c - aa) * (c + aa - b) * (aa + b - c));
        aa = fdist(f, d, a, d, a + 1);
        c = fdist(f, d, a + 1, d + 1, a + 1);
        const double area2 = 0.25 * sqrt((aa + b + c) * (b + c - aa) * (c + aa - b) * (aa + b - c));
        return area1 + area2;
    }
};

/* the spacings that a candidate's Taylor fits divide by, and whether quot()
 * may divide by all of them; the dividends are differences of distance2 (m^2)
 * or of degrees, and quotients of those */
struct TaylorDiv {
    Recip d[3];   /* delta             */
    Recip two[3]; /* 2 delta           */
    Recip sq[3];  /* delta^2           */
    bool ok;
    __device__ explicit TaylorDiv(const double* delta) : ok(true) {
        for (int k = 0; k < 3; ++k) {
            d[k] = recip(delta[k]);
            two[k] = recip(2.0 * delta[k]);
            sq[k] = recip(delta[k] * delta[k]);
            ok = ok && divisor_ok(delta[k]) && divisor_ok(2.0 * delta[k]) && divisor_ok(delta[k] * delta[k]);
        }
    }
};

template <bool FAST>
__device__ __forceinline__ double divide(double a, Recip r) {
    return FAST ? quot(a, r) : a / r.b;
}

template <bool FAST>
__device__ __forceinline__ void taylor_coeff(const double v[3][3][3], const TaylorDiv& D, double& center, double* g,
                                             double h[3][3]) {
    center = v[1][1][1];
    h[0][0] = divide<FAST>(v[2][1][1] + v[0][1][1] - 2.0 * center, D.sq[0]);
    h[1][1] = divide<FAST>(v[1][2][1] + v[1][0][1] - 2.0 * center, D.sq[1]);
    h[2][2] = divide<FAST>(v[1][1][2] + v[1][1][0] - 2.0 * center, D.sq[2]);
    g[0] = divide<FAST>(v[2][0][1] - v[0][0][1], D.two[0]);
    g[2] = divide<FAST>(v[2][2][1] - v[0][2][1], D.two[0]);
    h[0][1] = divide<FAST>(g[2] - g[0], D.two[1]);
    h[1][0] = h[0][1];
    g[0] = divide<FAST>(v[2][1][0] - v[0][1][0], D.two[0]);
    g[2] = divide<FAST>(v[2][1][2] - v[0][1][2], D.two[0]);
    h[0][2] = divide<FAST>(g[2] - g[0], D.two[2]);
    h[2][0] = h[0][2];
    g[0] = divide<FAST>(v[1][2][0] - v[1][0][0], D.two[1]);
    g[2] = divide<FAST>(v[1][2][2] - v[1][0][2], D.two[1]);
    h[1][2] = divide<FAST>(g[2] - g[0], D.two[2]);
    h[2][1] = h[1][2];
    g[0] = divide<FAST>(v[2][1][1] - v[0][1][1], D.two[0]);
    g[1] = divide<FAST>(v[1][2][1] - v[1][0][1], D.two[1]);
    g[2] = divide<FAST>(v[1][1][2] - v[1][1][0], D.two[2]);
}

__device__ __forceinline__ void make_taylor_coeff(const double v[3][3][3], const TaylorDiv& D, double& center,
                                                  double* g, double h[3][3]) {
    if (D.ok)
        taylor_coeff<true>(v, D, center, g, h);
    else
        taylor_coeff<false>(v, D, center, g, h);
}

/* m /= x */
__device__ __forceinline__ void divide_all(double m[3][3], double x) {
    const Recip r = recip(x);
    const bool ok = divisor_ok(x);
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) m[i][j] = ok ? quot(m[i][j], r) : m[i][j] / x;
}

__device__ __forceinline__ double dot3(const double* a, const double* b) {
    double t = 0.0;
    t += a[0] * b[0];
    t += a[1] * b[1];
    t += a[2] * b[2];
    return t;
}
__device__ __forceinline__ void matvec(const double m[3][3], const double* x, double* y) {
    for (int r = 0; r < 3; ++r) {
        double t = 0.0;
        t += m[r][0] * x[0];
        t += m[r][1] * x[1];
        t += m[r][2] * x[2];
        y[r] = t;
    }
}
__device__ __forceinline__ double norm2(const double* g) {
    double t = 0.0;
    t += fabs(g[0]) * fabs(g[0]);
    t += fabs(g[1]) * fabs(g[1]);
    t += fabs(g[2]) * fabs(g[2]);
    return sqrt(t);
}

/* wave_queue::compute_offsets (wave_queue.cc:708-924).  Called by a whole
 * warp: lanes 0-8 test the 3x3 neighbours' stability at once. */
__device__ void compute_offsets(const QueueDev& q, const FrontPtrs& V, const FrontPtrs& C,
                                const FrontPtrs& X, int t, int de0, int az0,
                                const double cube[3][3][3], const double* delta, const TaylorDiv& D,
                                double* offset, double* distance) {
    const int ic = de0 * q.naz + az0;
    bool bad = false;
    {
        const int lane = threadIdx.x & 31;
        if (lane < 9) {
            const int surface = C.surface[ic], bottom = C.bottom[ic], caustic = C.caustic[ic];
            const int i = (de0 + lane / 3 - 1) * q.naz + wrap_az(q, az0, lane % 3);
            bad = V.surface[i] != surface || C.surface[i] != surface || X.surface[i] != surface ||
                  V.bottom[i] != bottom || C.bottom[i] != bottom || X.bottom[i] != bottom ||
                  V.caustic[i] != caustic || C.caustic[i] != caustic || X.caustic[i] != caustic ||
                  V.on_edge[i];
        }
    }
    bool unstable = __any_sync(0xffffffffu, bad);
    double center, g[3], h[3][3], inv[3][3];
    make_taylor_coeff(cube, D, center, g, h);
    /* kept: hessian(2,1)*hessian(2,0) in the last cofactor (wave_queue.cc:762-763) */
    double determinant = fmax(1e-6, h[0][0] * (h[1][1] * h[2][2] - h[1][2] * h[2][1]) +
                                        h[0][1] * (h[1][2] * h[2][0] - h[1][0] * h[2][2]) +
                                        h[0][2] * (h[1][0] * h[2][1] - h[2][1] * h[2][0]));
    unstable = unstable || determinant < norm2(g);
    const double hh[3] = {fmax(1e-10, h[0][0]), fmax(1e-10, h[1][1]), fmax(1e-10, h[2][2])};
    const bool fast = D.ok && divisor_ok(hh[0]) && divisor_ok(hh[1]) && divisor_ok(hh[2]);
    double ratio[3];
    for (int k = 0; k < 3; ++k) {
        offset[k] = fast ? quot(-g[k], recip(hh[k])) : -g[k] / hh[k];
        ratio[k] = fast ? quot(offset[k], D.d[k]) : offset[k] / delta[k];
    }
    for (int k = 0; k < 3; ++k) {
        if (fabs(ratio[k]) > 0.5) {
            unstable = true;
            offset[k] = (offset[k] < 0.0) ? -(0.5 * delta[k]) : 0.5 * delta[k];
        }
    }
    if (!unstable) {
        inv[0][0] = h[1][1] * h[2][2] - h[1][2] * h[2][1];
        inv[1][0] = h[1][2] * h[2][0] - h[1][0] * h[2][2];
        inv[2][0] = h[1][0] * h[2][1] - h[1][1] * h[2][0];
        inv[0][1] = inv[1][0];
        inv[1][1] = h[0][0] * h[2][2] - h[0][2] * h[2][0];
        inv[2][1] = h[2][0] * h[0][1] - h[0][0] * h[2][1];
        inv[0][2] = inv[2][0];
        inv[1][2] = inv[2][1];
        inv[2][2] = h[0][0] * h[1][1] - h[0][1] * h[1][0];
        divide_all(inv, determinant);
        const double ng[3] = {-g[0], -g[1], -g[2]};
        matvec(inv, ng, offset);
        unstable = unstable || fabs(offset[1]) >= 0.5 * fabs(delta[1]);
    } else {
        const double save_offset = offset[1];
        g[1] = 0.0;
        determinant = h[0][0] * h[2][2] - h[0][2] * h[2][0];
        if (determinant >= norm2(g)) {
            for (int r = 0; r < 3; ++r)
                for (int c = 0; c < 3; ++c) inv[r][c] = 0.0;
            inv[0][0] = h[2][2];
            inv[0][2] = -h[0][2];
            inv[1][1] = 1.0;
            inv[2][0] = -h[2][0];
            inv[2][2] = h[0][0];
            divide_all(inv, determinant);
            const double ng[3] = {-g[0], -g[1], -g[2]};
            matvec(inv, ng, offset);
            offset[1] = save_offset;
        }
    }
    for (int k = 0; k < 3; ++k) {
        distance[k] = -g[k] * offset[k] - 0.5 * h[k][k] * offset[k] * offset[k];
        distance[k] = sqrt(fmax(0.0, distance[k]));
        if (offset[k] < 0.0) distance[k] *= -1.0;
    }
    if (unstable) {
        distance[1] = center - distance[0] * distance[0] - distance[2] * distance[2];
        if (distance[1] <= 0.0) {
            distance[1] = 0.0;
            offset[1] = 0.0;
        } else {
            distance[1] = sqrt(distance[1]);
            offset[1] = fabs(offset[1]);
            double cpa[3], nxt[3], prv[3], dir[3], speed;
            collision_location(q, V, C, X, ic, offset[0], cpa, dir, &speed);
            collision_location(q, V, C, X, ic + q.naz, offset[0], nxt, dir, &speed);
            collision_location(q, V, C, X, ic - q.naz, offset[0], prv, dir, &speed);
            double nxt_dir[3], tgt_dir[3];
            nxt_dir[0] = nxt[0] - cpa[0];
            nxt_dir[1] = (nxt[1] - prv[1]) * cpa[0];
            nxt_dir[2] = (nxt[2] - prv[2]) * cpa[0] * sin(cpa[1]);
            if (fabs(nxt_dir[0]) < 0.01) nxt_dir[0] = 0.0;
            tgt_dir[0] = q.tgt[0][t] - cpa[0];
            tgt_dir[1] = (q.tgt[1][t] - cpa[1]) * cpa[0];
            tgt_dir[2] = (q.tgt[2][t] - cpa[2]) * cpa[0] * sin(cpa[1]);
            if (dot3(nxt_dir, tgt_dir) < 0.0) {
                distance[1] *= -1.0;
                offset[1] *= -1.0;
            }
        }
    }
}

}  // namespace

constexpr int EIG_WARPS = 4;

/* the two warps of pair p (warps 2p, 2p+1 of the block) meet here */
__device__ __forceinline__ void pair_sync(int pair) {
    static_assert(EIG_WARPS == 4, "two warp pairs per block: named barriers 1 and 2");
    if (pair == 0)
        asm volatile("bar.sync 1, 64;" ::: "memory");
    else
        asm volatile("bar.sync 2, 64;" ::: "memory");
}

__global__ void __launch_bounds__(32 * EIG_WARPS) k_eigenray(__grid_constant__ const QueueDev q, int k) {
    __shared__ double s_cube[EIG_WARPS][27];
    __shared__ double s_ang[EIG_WARPS][2][27];
    __shared__ double s_g[EIG_WARPS][32][EIG_FG + 1];
    __shared__ double s_az[EIG_WARPS / 2][64];
    __shared__ double s_w[EIG_WARPS][32 + EIG_SIDE];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    /* a warp pair per candidate: with hybrid Gaussian spreading the even
     * warp runs the D/E walks and the odd warp the AZ walks, which are
     * independent sums; the odd warp hands its sums over and moves on */
    const int pair = warp >> 1, half = warp & 1;
    const int64_t s = *q.d_base + k + 1;
    const double time = q.d_times[k + 1];
    const int list = cand_list(s);
    const uint32_t ncand = min(q.n_cand[list], q.cap_cand);
    const uint32_t* cand = q.cand + (size_t)list * 2 * q.cap_cand;
    WarpBuild B;
    B.q = &q;
    B.pV = &q.F[ring_slot(s + 1)];
    B.pC = &q.F[ring_slot(s + 2)];
    B.pX = &q.F[ring_slot(s + 3)];
    B.lane = lane;
    B.sg = s_g[warp];
    B.sw = s_w[warp];
    B.su = s_w[warp] + 32;
    const FrontPtrs& V = *B.pV;
    const FrontPtrs& C = *B.pC;
    const FrontPtrs& X = *B.pX;
    double (*cube)[3][3] = reinterpret_cast<double (*)[3][3]>(s_cube[warp]);
    const uint32_t npairs = gridDim.x * (EIG_WARPS / 2);
    for (uint32_t c = blockIdx.x * (EIG_WARPS / 2) + pair; c < ncand; c += npairs) {
        __syncwarp();
        const uint32_t tu = cand[2 * c], iu = cand[2 * c + 1];
        /* the CPA kernels only queue interior rays and real targets */
        if (tu >= (uint32_t)q.nt || iu >= (uint32_t)q.n || iu / q.naz < 1 || iu / q.naz > (uint32_t)q.nde - 2) {
            if (lane == 0) set_err(q, ERR_BAD_CANDIDATE);
            continue;
        }
        const int t = (int)tu;
        const int i = (int)iu;
        const int de0 = i / q.naz, az0 = i % q.naz;
        /* above_bounce_threshold (wave_thresholds.h:192-199) */
        if (C.bottom[i] > q.max_bottom || C.surface[i] > q.max_surface ||
            C.caustic[i] > q.max_caustic || C.upper[i] > q.max_upper || C.lower[i] > q.max_lower)
            continue;
        const TgtS tg{q.tgt[1][t], q.tgt[2][t], q.tgt_sin[t], q.tgt_R2[t], q.tgt_2R[t]};
        /* the 27 distance2 values, one per lane */
        if (lane < 27) {
            const int m = lane / 9, nd_ = (lane / 3) % 3, na = lane % 3;
            const int j = (de0 + nd_ - 1) * q.naz + wrap_az(q, az0, na);
            const FrontPtrs& F = (m == 0) ? V : (m == 1) ? C : X;
            s_cube[warp][lane] = d2_at(F, j, tg);
        }
        __syncwarp();
        double delta[3] = {q.dt, q.de_inc[de0], q.az_inc[az0]};
        double offset[3], distance[3];
        const TaylorDiv D(delta);
        compute_offsets(q, V, C, X, t, de0, az0, cube, delta, D, offset, distance);

        /* spreading: lane f holds frequency f (and f + 32) */
        double si_lo = 0.0, si_hi = 0.0;
        B.spread2 = q.tgt_spread2 + (size_t)t * q.nf;
        if (q.spreading == WQ3D_HYBRID_GAUSSIAN) {
            /* spreading_hybrid_gaussian.cc:65-119 */
            int a = az0;
            double no[3] = {offset[0], offset[1], offset[2]};
            if (offset[2] < 0.0) {
                if (az0 > 0) {
                    a = az0 - 1;
                } else if (q.az_boundary) {
                    a = q.naz - 2;
                }
                no[2] = offset[2] + B.az_inc(a);
            }
            double de_lo = 0.0, de_hi = 0.0;
            if (half == 0) {
                B.Ilo = B.Ihi = 0.0;
                B.intensity_de(de0, a, no, distance);
                de_lo = B.Ilo;
                de_hi = B.Ihi;
            } else {
                no[2] = offset[2];
                int d = de0;
                if (offset[1] < 0.0 && !C.on_edge[i - q.naz]) {
                    d = de0 - 1;
                    no[1] = offset[1] + B.de_inc(d);
                }
                B.Ilo = B.Ihi = 0.0;
                B.intensity_az(d, az0, no, distance);
                s_az[pair][lane] = B.Ilo;
                s_az[pair][32 + lane] = B.Ihi;
            }
            /* both warps pass both barriers once per candidate */
            pair_sync(pair);
            if (half == 1) {
                pair_sync(pair);
                continue;
            }
            const double az_lo = s_az[pair][lane], az_hi = s_az[pair][32 + lane];
            pair_sync(pair);
            si_lo = de_lo * az_lo;
            si_hi = de_hi * az_hi;
        } else {
            if (half == 1) continue;
            /* spreading_ray.cc:47-133; an AZ wrap below index 0 is wrapped */
            int d = de0, a = az0;
            if (offset[1] < 0.0) --d;
            if (offset[2] < 0.0) a = (a == 0) ? q.naz - 2 : a - 1;
            const double area1 = B.area4(C, d, a);
            const double area2 = (offset[0] < 0.0) ? B.area4(V, d, a) : B.area4(X, d, a);
            double u = fabs(offset[0]) / q.dt;
            const double area = (1.0 - u) * area1 + u * area2;
            const double loss = q.init_area[d * q.naz + a] * q.tgt_c[t] / (area * q.init_sound_speed);
            bool zero = false;
            u = fabs(offset[1]) / B.de_inc(d) - 1.0;
            if (u > 4.0) zero = true;
            u = fabs(offset[2]) / B.az_inc(a) - 1.0;
            if (u > 4.0) zero = true;
            si_lo = si_hi = zero ? loss * 0.0 : loss;
        }
        const bool has_lo = lane < q.nf, has_hi = lane + 32 < q.nf;
        const bool bad = (has_lo && isnan(si_lo)) || (has_hi && isnan(si_hi));
        if (__any_sync(0xffffffffu, bad)) continue;
        double tl_lo = -10.0 * log10(fmax(si_lo, 1e-30));
        double tl_hi = -10.0 * log10(fmax(si_hi, 1e-30));
        double ddt = offset[0] / q.dt;
        const FrontPtrs& A0 = (ddt >= 0.0) ? C : V;
        const FrontPtrs& A1 = (ddt >= 0.0) ? X : C;
        if (ddt < 0.0) ddt = 1.0 + ddt;
        if (has_lo)
            tl_lo = tl_lo + A0.atten[(size_t)lane * q.n + i] * (1.0 - ddt) +
                    A1.atten[(size_t)lane * q.n + i] * ddt;
        if (has_hi)
            tl_hi = tl_hi + A0.atten[(size_t)(lane + 32) * q.n + i] * (1.0 - ddt) +
                    A1.atten[(size_t)(lane + 32) * q.n + i] * ddt;
        const bool above = (has_lo && tl_lo < q.intensity_threshold) ||
                           (has_hi && tl_hi < q.intensity_threshold);
        if (!__any_sync(0xffffffffu, above)) continue;

        /* direction angles of the 27 neighbours on three fronts
         * (wvector1::direction, types/wvector1.cc) */
        if (lane < 27) {
            const int m = lane / 9, nd_ = (lane / 3) % 3, na = lane % 3;
            const int j = (de0 + nd_ - 1) * q.naz + wrap_az(q, az0, na);
            const FrontPtrs& F = (m == 0) ? V : (m == 1) ? C : X;
            const double n0 = F.nd[0][j], n1 = F.nd[1][j], n2 = F.nd[2][j];
            s_ang[warp][0][lane] = atan2(n0, sqrt(n1 * n1 + n2 * n2)) * (180.0 / M_PI);
            s_ang[warp][1][lane] = atan2(n2, -n1) * (180.0 / M_PI);
        }
        __syncwarp();
        double tang[2];
        for (int which = 0; which < 2; ++which) {
            double center, g[3], h[3][3], hv[3];
            make_taylor_coeff(reinterpret_cast<double (*)[3][3]>(s_ang[warp][which]), D, center, g, h);
            matvec(h, offset, hv);
            tang[which] = center + dot3(g, offset) + 0.5 * dot3(offset, hv);
        }
        uint32_t slot = 0;
        if (lane == 0) slot = atomicAdd(q.n_rec, 1u);
        slot = __shfl_sync(0xffffffffu, slot, 0);
        if (slot >= q.cap_rec) {
            if (lane == 0) set_err(q, ERR_REC_OVERFLOW);
            __syncwarp();
            continue;
        }
        if (lane == 0) {
            wq3d_eigenray r;
            r.time = time + offset[0];
            r.source_de = q.de[de0] + offset[1];
            r.source_az = q.az[az0] + offset[2];
            r.target_de = tang[0];
            r.target_az = tang[1];
            r.surface = C.surface[i];
            r.bottom = C.bottom[i];
            r.caustic = C.caustic[i];
            r.upper = C.upper[i];
            r.lower = C.lower[i];
            r.t1 = t / q.nt2;
            r.t2 = t % q.nt2;
            r.de = de0;
            r.az = az0;
            r.pad = 0;
            r.step = s;
            q.rec[slot] = r;
        }
        if (q.sens && lane < 3)
            q.rec_sens[(size_t)slot * 3 + lane] = A0.dA[(size_t)lane * q.n + i] * (1.0 - ddt) +
                                                  A1.dA[(size_t)lane * q.n + i] * ddt;
        if (has_lo) {
            q.rec_inten[(size_t)slot * q.nf + lane] = tl_lo;
            q.rec_phase[(size_t)slot * q.nf + lane] = C.phase[(size_t)lane * q.n + i];
        }
        if (has_hi) {
            q.rec_inten[(size_t)slot * q.nf + lane + 32] = tl_hi;
            q.rec_phase[(size_t)slot * q.nf + lane + 32] = C.phase[(size_t)(lane + 32) * q.n + i];
        }
        __syncwarp();
    }
}

/* ------------------------------------------------------------------ */
/* single-point model evaluations (ocean parity tests)                 */
/* ------------------------------------------------------------------ */
__global__ void k_sound_speed(OceanDev oc, double R, int n, const double* rho,
                              const double* theta, const double* phi, double* c,
                              double* g) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double cc, gg[3];
    sound_speed(oc.prof, R, rho[i], theta[i], phi[i], &cc, gg);
    c[i] = cc;
    if (g) {
        g[i] = gg[0];
        g[n + i] = gg[1];
        g[2 * n + i] = gg[2];
    }
}

__global__ void k_height(BoundaryDev b, int n, const double* theta, const double* phi,
                         double* h, double* nrm) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double nn[3];
    h[i] = boundary_height_normal(b, theta[i], phi[i], nn);
    if (nrm) {
        nrm[i] = nn[0];
        nrm[n + i] = nn[1];
        nrm[2 * n + i] = nn[2];
    }
}

/* attenuation_thorp.cc:29-35 with the per-frequency alpha precomputed on
 * the host, or attenuation_constant.cc:14-25 */
__global__ void k_attenuation(ProfileDev pr, double R, int n, const double* rho,
                              const double* dist, int nf, const double* freq,
                              const double* alpha, double* atten) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double alt = rho[i] - R;
    for (int f = 0; f < nf; ++f) {
        atten[(size_t)i * nf + f] = (pr.atten == WQ3D_ATTEN_CONSTANT)
                                        ? pr.atten_coef * dist[i] * freq[f]
                                        : dist[i] * alpha[f] * (1.0 + 5.88264e-6 * alt);
    }
}

__global__ void k_reflect_loss(BoundaryDev b, int n, const double* grazing, int nf,
                               const double* freq, double* amp, double* ph) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const LossDev& L = b.loss;
    double a0 = 0.0, p0 = 0.0;
    if (L.kind != WQ3D_LOSS_ECKART) reflect_loss_scalar(L, grazing[i], &a0, &p0);
    const double w2 = L.p[0] * L.p[0];
    const double sg = sin(grazing[i]);
    for (int f = 0; f < nf; ++f) {
        double a = a0, p = p0;
        if (L.kind == WQ3D_LOSS_ECKART) {
            const double x = freq[f] * w2 * sg;
            a = 8.6e-9 * (x * x);
            p = M_PI;
        }
        amp[(size_t)i * nf + f] = a;
        if (ph) ph[(size_t)i * nf + f] = p;
    }
}

#endif  // !WQ3D_STEP_KERNELS_ONLY

}  // namespace wq3d

#if WQ3D_WITH_GRID && !WQ3D_STEP_KERNELS_ONLY
/* the adjoint's kernels reuse the step functions above */
#define WQ3D_ADJOINT_IMPL 1
#include "wq3d_adjoint.cuh"
#endif
