/*
 * LOQUAT-B200 integrator of one material slot, shared by the stand-alone
 * predictor and corrector kernels (integrate.cu) and by the native driver's
 * pair kernel, which integrates each target as soon as its sums are done
 * (sph.cu): the target's rates then never leave the registers, and the
 * state's traffic overlaps other targets' pair sums.
 */
#pragma once

#include "lq_device.cuh"

namespace lqb {

/* The rates of one slot: acceleration and density rate, spin, strain rate. */
struct SlotRates {
    float4 a, w;
    tensor2d de;
};

__device__ __forceinline__ SlotRates load_rates(const Rates& rt, int i)
{
    return SlotRates{__ldg(rt.accad + i), __ldg(rt.spin + i), load_t2(rt.acestn, i)};
}

/* FP64 position (pressure p in the float word's w) and velocity into the
 * float high words x, v and, with `lo`, the low words of `out` at slot i. */
__device__ __forceinline__ void split_words(const State& out, int i, const double4& xd, const double4& vd, float p,
                                            float4& x, float4& v, bool lo = true)
{
    float4 xl, vl;
    split4(make_double4(xd.x, xd.y, xd.z, 0.0), x, xl);
    split4(vd, v, vl);
    x.w = p;
    if (lo) {
        out.xlo[i] = xl;
        out.vlo[i] = vl;
    }
}

/* A material slot's entry of the pair kernel's packed neighbour arrays from
 * the position, velocity and stress just stored (what k_pack_neighbors
 * would write from them), when nb is set.  kPk (the mixed form) packs the
 * velocity into two words. */
template <bool kPk>
__device__ __forceinline__ void pack_slot(const NbrArrays& nb, int i, const float4& x, const float4& v,
                                          const tensor2d& s)
{
    if (!nb.xs) return;
    nb.xs[2 * (size_t)i] = make_float4(x.x, x.y, x.z, v.w);
    store_packed<kPk>(nb, i, v, s);
}

/* When the corrector raises the neighbour lists' flag (launch_correct_into). */
struct VerletCheck {
    const float4* xbuild;
    int* rebuild;
    float half_skin;
    float dt_bound;   /* the largest step the next one can take */
    const float4* xwide;   /* two-level lists: positions at the wide build */
    float half_margin;     /* (wide - skin) / 2 */
};

/* A dynamic step never exceeds the fixed one, cfl h / cs (ph->dt). */
inline VerletCheck verlet_of(const Parameters* ph, const ListCheck& l)
{
    return VerletCheck{l.xbuild, l.flag, 0.5f * l.skin, ph->dt, l.xwide, 0.5f * (l.wide - l.skin)};
}

/* The list checks of one material particle at its new position x. */
__device__ __forceinline__ void verlet_check(const VerletCheck& vc, int i, const float4& x, const float4& v,
                                             const float4& a)
{
    const float4 xb = __ldg(vc.xbuild + i);
    const float dx = x.x - xb.x, dy = x.y - xb.y, dz = x.z - xb.z;
    const float moved = sqrtf(dx * dx + dy * dy + dz * dz);
    const float speed = sqrtf(v.x * v.x + v.y * v.y + v.z * v.z);
    const float accel = sqrtf(a.x * a.x + a.y * a.y + a.z * a.z);
    /* next step: the predictor half step and the corrector full step
     * move a particle by at most dt |v| + dt^2 |a| each; 2x covers both */
    const float dtb = vc.dt_bound;
    const float ahead = 2.0f * dtb * (speed + dtb * accel);
    if (!(moved + ahead < vc.half_skin)) atomicOr(vc.rebuild, 1);
    if (vc.xwide) {
        /* lists renewed at x from the wide ones hold every pair within
         * 2h + skin while no particle is (wide - skin) / 2 from xwide */
        const float4 xw = __ldg(vc.xwide + i);
        const float ex = x.x - xw.x, ey = x.y - xw.y, ez = x.z - xw.z;
        if (!(sqrtf(ex * ex + ey * ey + ez * ez) < vc.half_margin)) atomicOr(vc.rebuild, 2);
    }
}

__device__ __forceinline__ bool finite_kinematics(const float4& x, const float4& v)
{
    return isfinite(x.x) && isfinite(x.y) && isfinite(x.z) && isfinite(v.x) && isfinite(v.y) && isfinite(v.z) &&
           isfinite(v.w);
}

__device__ __forceinline__ bool finite_stress(const tensor2d& s)
{
    return isfinite(s.xx) && isfinite(s.yy) && isfinite(s.zz) && isfinite(s.xy) && isfinite(s.xz) && isfinite(s.yz);
}

/* Half step of material slot i (reference src/predictor_corrector.cu:169-218):
 * v += dt/2 a; rho += dt/2 drho; x += dt/2 v_new; eps += dt/2 deps;
 * stress and plastic strain from the model at dt/2, from `in` into `out`.
 * With `stage` the output is a stage buffer that only the neighbour kernels
 * and the corrector read: the position and velocity high words (with the
 * pressure) and the stress; the corrector restarts everything else from its
 * snapshot, so the strain (neither read nor written), the low words and the
 * object word are left out.  Model 3's stress is k_vw_trial's: its slots
 * get their kinematics and a packed entry with the old stress here. */
template <bool kMixed>
__device__ __forceinline__ void predict_slot(const Parameters* __restrict__ P, int i, const State& in,
                                             const State& out, const SlotRates& r, const MaterialTable& mt,
                                             const NbrArrays& nb, bool stage, const float4& x0, const float4& v0,
                                             const float4& id, const tensor2d& s0, const tensor2d& e0)
{
    const float dt = __ldg(&P->dt);
    const Material M = particle_material(load_material(P), mt, id.x);
    float4 x, v;
    tensor2d s = s0, e = e0;
    float ep = id.y;
    if (kMixed) {
        /* FP64 accumulation of velocity, density and position; FP64 stress update */
        const double hdt = 0.5 * (double)dt;
        double4 vd = join4(v0, in.vlo[i]), xd = join4(x0, in.xlo[i]);
        vd.x += hdt * r.a.x; vd.y += hdt * r.a.y; vd.z += hdt * r.a.z; vd.w += hdt * r.a.w;
        xd.x += hdt * vd.x; xd.y += hdt * vd.y; xd.z += hdt * vd.z;
        T6d ed = widen6(e0), dd = widen6(r.de);
        ed.xx += dd.xx * hdt; ed.yy += dd.yy * hdt; ed.zz += dd.zz * hdt;
        ed.xy += dd.xy * hdt; ed.xz += dd.xz * hdt; ed.yz += dd.yz * hdt;
        double p = x0.w, epd = id.y;
        if (M.model != 3) {
            T6d sd = widen6(s0);
            if (M.model == 1)
                dp_update_d(M, hdt, r.w, dd, p, epd, sd);
            else
                hypo_update_d(M, hdt, dd, r.w, sd);
            s = narrow6(sd);
        }
        if (M.model != 1 && !stage) epd = sqrt(2.0 / 3.0 * contract6(ed, ed));
        ep = (float)epd;
        split_words(out, i, xd, vd, (float)p, x, v, !stage);
        e = narrow6(ed);
    } else {
        v = v0;
        v.x += 0.5f * dt * r.a.x;
        v.y += 0.5f * dt * r.a.y;
        v.z += 0.5f * dt * r.a.z;
        v.w += 0.5f * dt * r.a.w;
        x = x0;
        x.x += 0.5f * dt * v.x;
        x.y += 0.5f * dt * v.y;
        x.z += 0.5f * dt * v.z;
        e = e0 + r.de * (0.5f * dt);
        float p = x0.w;
        if (M.model == 1)
            dp_update(M, 0.5f * dt, r.w, r.de, p, ep, s);
        else if (M.model != 3)
            hypo_update(M, 0.5f * dt, r.de, r.w, s);
        if (M.model != 1 && !stage) ep = sqrtf(2.0f / 3.0f * J2(e));
        x.w = p;
    }
    out.pos[i] = x;
    out.vel[i] = v;
    if (M.model != 3) store_t2(out.str, i, s);
    if (!stage) {
        out.idep[i] = make_float4(id.x, ep, id.z, id.w);
        store_t2(out.stn, i, e);
    }
    pack_slot<kMixed>(nb, i, x, v, s);
}

/* Full step of material slot i from the snapshot `ini`
 * (reference src/predictor_corrector.cu:256-307): v = v0 + dt a;
 * x = x0 + dt/2 (v + v0); eps = eps0 + dt deps; the model restarts from the
 * snapshot's stress and plastic strain; the pressure passed in, p_now, is
 * the current one.  Writes `out` (which may be ini), counts non-finite
 * results in health, and with `verlet` checks the lists.  Model 3's stress
 * and void ratio are k_vw_trial's, as above. */
template <bool kMixed>
__device__ __forceinline__ void correct_slot(const Parameters* __restrict__ P, int i, float p_now,
                                             const float4& id, const State& ini, const State& out,
                                             const SlotRates& r, const MaterialTable& mt, const NbrArrays& nb,
                                             int* __restrict__ health, const VerletCheck& verlet)
{
    const float dt = __ldg(&P->dt);
    const float4 x0 = ini.pos[i];
    const float4 v0 = ini.vel[i];
    const float ep0 = ini.idep[i].y;
    const tensor2d s0 = load_t2_rw(ini.str, i);
    const tensor2d e0 = load_t2_rw(ini.stn, i);
    const Material M = particle_material(load_material(P), mt, id.x);
    float4 v, x;
    tensor2d s = s0, e;
    float ep;
    if (kMixed) {
        const double ddt = dt;
        const double4 v0d = join4(v0, ini.vlo[i]), x0d = join4(x0, ini.xlo[i]);
        double4 vd, xd;
        vd.x = v0d.x + ddt * r.a.x; vd.y = v0d.y + ddt * r.a.y; vd.z = v0d.z + ddt * r.a.z; vd.w = v0d.w + ddt * r.a.w;
        xd.x = 0.5 * (vd.x + v0d.x) * ddt + x0d.x;
        xd.y = 0.5 * (vd.y + v0d.y) * ddt + x0d.y;
        xd.z = 0.5 * (vd.z + v0d.z) * ddt + x0d.z;
        xd.w = 0.0;
        T6d ed = widen6(e0), dd = widen6(r.de);
        ed.xx += dd.xx * ddt; ed.yy += dd.yy * ddt; ed.zz += dd.zz * ddt;
        ed.xy += dd.xy * ddt; ed.xz += dd.xz * ddt; ed.yz += dd.yz * ddt;
        double pd = p_now, epd = ep0;
        if (M.model != 3) {
            T6d sd = widen6(s0);
            if (M.model == 1)
                dp_update_d(M, ddt, r.w, dd, pd, epd, sd);
            else
                hypo_update_d(M, ddt, dd, r.w, sd);
            s = narrow6(sd);
        }
        if (M.model != 1) epd = sqrt(2.0 / 3.0 * contract6(ed, ed));
        split_words(out, i, xd, vd, (float)pd, x, v);
        e = narrow6(ed);
        ep = (float)epd;
    } else {
        v.x = v0.x + dt * r.a.x;
        v.y = v0.y + dt * r.a.y;
        v.z = v0.z + dt * r.a.z;
        v.w = v0.w + dt * r.a.w;
        x.x = 0.5f * (v.x + v0.x) * dt + x0.x;
        x.y = 0.5f * (v.y + v0.y) * dt + x0.y;
        x.z = 0.5f * (v.z + v0.z) * dt + x0.z;
        e = e0 + r.de * dt;
        float p = p_now;
        ep = ep0;
        if (M.model == 1)
            dp_update(M, dt, r.w, r.de, p, ep, s);
        else if (M.model != 3)
            hypo_update(M, dt, r.de, r.w, s);
        if (M.model != 1) ep = sqrtf(2.0f / 3.0f * J2(e));
        x.w = p;
    }
    out.pos[i] = x;
    out.vel[i] = v;
    out.idep[i] = make_float4(id.x, ep, id.z, id.w);
    if (M.model != 3) store_t2(out.str, i, s);
    store_t2(out.stn, i, e);
    pack_slot<kMixed>(nb, i, x, v, s);
    if (health && !(finite_kinematics(x, v) && (M.model == 3 || finite_stress(s))))
        atomicAdd(health + HEALTH_NONFINITE, 1);
    if (verlet.xbuild) verlet_check(verlet, i, x, v, r.a);
}

}  // namespace lqb
