/*
 * LOQUAT-B200 predictor-corrector integrator with the Drucker-Prager and
 * hypoplastic stress updates (reference src/predictor_corrector.cu:169-336),
 * its C ABI entry points and the C++ drop-in functions.
 *
 * The reference issues five device-to-device snapshot copies and then the
 * predictor kernel; here the snapshot is written by the same kernel that
 * reads the state, so the state is read once.  The native driver skips the
 * snapshot entirely: the predictor step writes into a second buffer and the
 * corrector step restarts from the untouched first one, in place.  Its
 * thread-per-target pair kernels take both steps themselves (sph.cu); the
 * kernels here serve the drop-in calls, the warp-cooperative pair shapes and,
 * for every shape, model 3's stresses.
 */
#include <cstdio>
#include <cstdlib>

#include "lq_internal.cuh"
#include "lq_device.cuh"
#include "lq_integrate.cuh"
#include <predictor_corrector.h>

namespace lqb {

namespace {

constexpr int kBlock = 128;
/* resident blocks per SM asked of the model-3 kernels: 4 caps them at 128
 * registers; on the 2.85 M-particle slope in flow the two integrations take
 * 1299 us a step with 4, 1332 with 5 (96 registers, spills), 1348 with 6 */
#ifndef LQ_VW_MIN_BLOCKS
#define LQ_VW_MIN_BLOCKS 4
#endif
/* resident blocks per SM asked of k_predict and k_correct: 6 caps them at 80
 * registers (the mixed form's FP64 return map spills), 24 warps per SM instead
 * of 16 uncapped (117 to 120); when the native driver still integrated by
 * them in every shape, the 256-scenario ensemble's mixed integrations took
 * 2.19 ms a step against 2.25 (5), 2.22 (7), 2.36 (8) and 2.49 uncapped; the
 * plain ones (78 registers) are unaffected */
#ifndef LQ_INT_MIN_BLOCKS
#define LQ_INT_MIN_BLOCKS 6
#endif

inline int blocks_for(long long n, int b) { return (int)((n + b - 1) / b); }

/* What the model-3 kernels store of a finished stress: the stress, the void
 * ratio (`full`: not in a stage buffer), the packed entry's stress words,
 * and a non-finite stress in health unless the slot's kinematics already
 * counted. */
__device__ __forceinline__ void store_vw(const State& out, int i, const T6d& sd, double e, bool full,
                                         const NbrArrays& nb, int* __restrict__ health)
{
    const tensor2d s = narrow6(sd);
    store_t2(out.str, i, s);
    if (full) reinterpret_cast<float*>(out.idep + i)[2] = (float)e;
    const float4 v = out.vel[i];
    if (nb.xs) store_packed_stress(nb, i, v.w, s);
    if (health && !finite_stress(s) && finite_kinematics(out.pos[i], v)) atomicAdd(health + HEALTH_NONFINITE, 1);
}

/* Model 3: the stress and void ratio of the material slots over part x dt,
 * by the first trial sub-step, which spans the whole interval.  Nine in ten
 * particles of a half step and two in three of a full step need no more
 * (the slope in flow); the others are queued with the step of their next
 * trial, for k_vw_finish.  A kernel of its own, after the kinematics, keeps
 * the trial's state in as few registers as its two rate evaluations allow:
 * it is bound by FP64 latency, so by the warps in flight (the FP64 pipe is
 * busy 46 % of the time at 15 warps per SM).  On the 2.85 M-particle slope
 * a half step's trials take 258 us and its queue 138, a full step's 271 and
 * 330; one kernel that ran each particle to its end took 660 and 740 with
 * the kinematics (106 and 177) in it. */
__global__ void __launch_bounds__(kBlock, LQ_VW_MIN_BLOCKS) k_vw_trial(const Parameters* __restrict__ P, double part,
                                                                       int npb, int np, const float4* idep,
                                                                       const tensor2d* src_str, State out, bool full,
                                                                       Rates rt, MaterialTable vw, NbrArrays nb,
                                                                       int* __restrict__ health, SubstepQueue q)
{
    const int i = npb + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    const double dt = part * (double)__ldg(&P->dt);
    const float4 id = idep[i];
    const tensor2d s0 = load_t2_rw(src_str, i);
    if (!(dt > 0.0)) {
        store_vw(out, i, widen6(s0), id.z, full, nb, health);
        return;
    }
    const VWConst& c = *vw_row(vw, id.x);
    VWTrial g;
    const float4 w = __ldg(rt.spin + i);
    const tensor2d de = load_t2(rt.acestn, i);
    if (g.run(c, dt, s0, id.z, de, w)) {
        store_vw(out, i, g.s, g.e, full, nb, health);
        return;
    }
    const bool hard = !(g.h > 0.2 * dt);    /* the largest cut of a step: the longest runs */
    const unsigned act = __activemask();
    const unsigned hards = __ballot_sync(act, hard);
    const unsigned peers = hard ? hards : act & ~hards;
    const int lane = threadIdx.x & 31, leader = __ffs((int)peers) - 1;
    int at = 0;
    if (lane == leader) at = atomicAdd(q.counts + (hard ? 0 : 1), __popc(peers));
    at = __shfl_sync(peers, at, leader) + __popc(peers & ((1u << lane) - 1u));
    if (!hard) at = q.cap - 1 - at;
    if (!lq_in_range(at, q.cap)) return;
    q.item[at] = i;
    q.h[at] = g.h;
}

/* Model 3: the queued particles' remaining sub-steps from the start of
 * their interval (src_str, and the void ratio in idep).  The numbers of sub-steps
 * differ widely between neighbours (a warp of the slope's full steps needs
 * ten for its slowest lane, two on average), so a lane that has finished
 * takes the next particle of the queue while the others go on: every lane
 * evaluates a rate in every turn.  The particles whose step was cut most
 * come first, since the longest chain of evaluations ends the launch.
 * Bound by FP64 latency, and in small cases by the longest chain: 64
 * trials of two evaluations take 150 us where a warp has its part of the SM to
 * itself.  A short queue is therefore left to as many blocks as it fills, which
 * lie on different SMs; whichever warps came first took it otherwise, on a few
 * SMs (5 k particles with up to 64 sub-steps each: 840 us a step, so 564). */
__global__ void __launch_bounds__(kBlock, LQ_VW_MIN_BLOCKS) k_vw_finish(const Parameters* __restrict__ P, double part,
                                                                        const float4* idep,
                                                                        const tensor2d* src_str, State out,
                                                                        bool full, Rates rt, MaterialTable vw,
                                                                        NbrArrays nb, int* __restrict__ health,
                                                                        SubstepQueue q)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int nhard = q.counts[0], n = nhard + q.counts[1];
    if ((long long)blockIdx.x * kBlock >= n) return;
    const double dt = part * (double)__ldg(&P->dt);
    int i = -1;
    bool drained = false;
    VWIntegration g{};
    const VWConst* c = nullptr;
    tensor2d de{};
    float4 w{};
    for (;;) {
        const unsigned idle = __ballot_sync(FULL, i < 0 && !drained);
        if (idle) {
            int at = 0;
            if (lane == __ffs((int)idle) - 1) at = atomicAdd(q.counts + 2, __popc(idle));
            at = __shfl_sync(FULL, at, __ffs((int)idle) - 1) + __popc(idle & ((1u << lane) - 1u));
            if (idle >> lane & 1u) {
                if (at < n) {
                    if (at >= nhard) at = q.cap - 1 - (at - nhard);
                    if (lq_in_range(at, q.cap)) i = q.item[at];
                    if (lq_in_range(i, __ldg(&P->np))) {
                        const float4 id = idep[i];
                        c = vw_row(vw, id.x);
                        w = __ldg(rt.spin + i);
                        de = load_t2(rt.acestn, i);
                        g.start(widen6(load_t2_rw(src_str, i)), id.z, de, q.h[at], 1);
                    } else {
                        i = -1;
                    }
                } else {
                    drained = true;
                }
            }
        }
        if (__all_sync(FULL, i < 0)) break;
        if (i >= 0 && !g.advance(*c, dt, de, w)) {
            store_vw(out, i, g.s, g.e, full, nb, health);
            i = -1;
        }
    }
}

__global__ void k_vw_rows(int n, const float* __restrict__ rows, VWConst* __restrict__ derived)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) derived[k] = vw_const(rows + 10 * (size_t)k);
}

/* Predictor of the slots, into `out` (or in place); with do_snap each
 * slot's state is copied to `snap` first. */
template <bool kMixed>
__global__ void __launch_bounds__(kBlock, LQ_INT_MIN_BLOCKS) k_predict(const Parameters* __restrict__ P, int np,
                                                                       int npb, State in, State out, State snap,
                                                                       bool do_snap, Rates rt, MaterialTable mt,
                                                                       NbrArrays nb, bool stage)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    /* boundary slots change only by Adami, which writes both state buffers
     * of the native driver; without a snapshot there is nothing to do */
    if (i < npb && !do_snap) return;
    const float4 x0 = in.pos[i];
    const float4 v0 = in.vel[i];
    const float4 id = in.idep[i];
    const tensor2d s0 = load_t2_rw(in.str, i);
    const tensor2d e0 = stage ? make_tensor2d(0.0f) : load_t2_rw(in.stn, i);
    if (do_snap) {
        snap.pos[i] = x0;
        snap.vel[i] = v0;
        snap.idep[i] = id;
        store_t2(snap.str, i, s0);
        store_t2(snap.stn, i, e0);
    }
    if (i < npb) {
        /* a boundary slot of another output buffer takes the stress (the
         * Adami extrapolation); the rest never changes */
        if (out.pos != in.pos) store_t2(out.str, i, s0);
        return;
    }
    predict_slot<kMixed>(P, i, in, out, load_rates(rt, i), mt, nb, stage, x0, v0, id, s0, e0);
}

/* Corrector of the material slots from the snapshot `ini` and the current
 * state `cur` into `out` (which may be either); boundary slots are Adami's. */
template <bool kMixed>
__global__ void __launch_bounds__(kBlock, LQ_INT_MIN_BLOCKS) k_correct(const Parameters* __restrict__ P, int np,
                                                                       int npb, State cur, State ini, State out,
                                                                       Rates rt, int* __restrict__ health,
                                                                       VerletCheck verlet, MaterialTable mt,
                                                                       NbrArrays nb)
{
    const int i = npb + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    correct_slot<kMixed>(P, i, cur.pos[i].w, cur.idep[i], ini, out, load_rates(rt, i), mt, nb, health, verlet);
}

}  // namespace

/* This translation unit's count of bounds violations (always 0 without
 * LQ_CHECKED). */
int bounds_count_integrate(unsigned long long* v)
{
#ifdef LQ_CHECKED
    LQ_TRY_CUDA(cudaMemcpyFromSymbol(v, lq_bounds_count, sizeof(*v)), "bounds counter");
#else
    *v = 0;
#endif
    return LQ_OK;
}

size_t vw_row_bytes() { return sizeof(VWConst); }

int launch_vw_rows(const MaterialTable& vw, void* derived, cudaStream_t s)
{
    if (vw.n <= 0) return LQ_OK;
    k_vw_rows<<<blocks_for(vw.n, kBlock), kBlock, 0, s>>>(vw.n, vw.p, static_cast<VWConst*>(derived));
    LQ_TRY_CUDA(cudaGetLastError(), "k_vw_rows");
    return LQ_OK;
}

namespace {

/* The stresses of the material slots over part x dt: every slot's first
 * trial, then the queued ones by as many blocks as the device holds. */
int enqueue_substeps(const Parameters* ph, const Parameters* pd, double part, const float4* idep,
                     const tensor2d* src_str, const State& out, bool full, const Rates& r, const MaterialTable& vw,
                     const NbrArrays& nb, int* health, const SubstepQueue& q, cudaStream_t s)
{
    int dev = 0, sms = 0;
    LQ_TRY_CUDA(cudaGetDevice(&dev), "sub-steps");
    LQ_TRY_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "sub-steps");
    LQ_TRY_CUDA(cudaMemsetAsync(q.counts, 0, 3 * sizeof(int), s), "sub-step queue");
    k_vw_trial<<<blocks_for(ph->npm, kBlock), kBlock, 0, s>>>(pd, part, ph->npb, ph->np, idep, src_str, out, full, r,
                                                              vw, nb, health, q);
    LQ_TRY_CUDA(cudaGetLastError(), "k_vw_trial");
    k_vw_finish<<<sms * LQ_VW_MIN_BLOCKS, kBlock, 0, s>>>(pd, part, idep, src_str, out, full, r, vw, nb, health, q);
    LQ_TRY_CUDA(cudaGetLastError(), "k_vw_finish");
    return LQ_OK;
}

}  // namespace

int check_substeps(const Parameters* ph, const char* who, const MaterialTable& vw, const SubstepQueue& q)
{
    if (ph->constitutive_model != 3) return LQ_OK;
    if (!vw.p || vw.n <= 0 || !vw.derived)
        return set_error(LQ_ERR_ARG, "%s: constitutive model 3 needs a von Wolffersdorff table", who);
    if (!q.item || !q.h || !q.counts || q.cap < ph->npm)
        return set_error(LQ_ERR_ARG, "%s: constitutive model 3 needs a sub-step queue", who);
    return LQ_OK;
}

int launch_predict_substeps(const Parameters* ph, const Parameters* pd, const State& in, const State& out,
                            const Rates& r, cudaStream_t s, const MaterialTable& vw, float* rec,
                            const SubstepQueue& q)
{
    if (ph->constitutive_model != 3 || ph->npm <= 0) return LQ_OK;
    const NbrArrays nb = rec ? nbr_arrays(rec, ph->np) : NbrArrays{nullptr, nullptr, nullptr};
    return enqueue_substeps(ph, pd, 0.5, in.idep, in.str, out, false, r, vw, nb, nullptr, q, s);
}

int launch_correct_substeps(const Parameters* ph, const Parameters* pd, const State& st, const Rates& r, int* health,
                            cudaStream_t s, const MaterialTable& vw, float* rec, const SubstepQueue& q)
{
    if (ph->constitutive_model != 3 || ph->npm <= 0) return LQ_OK;
    const NbrArrays nb = rec ? nbr_arrays(rec, ph->np) : NbrArrays{nullptr, nullptr, nullptr};
    return enqueue_substeps(ph, pd, 1.0, st.idep, st.str, st, true, r, vw, nb, health, q, s);
}

int launch_predict(const Parameters* ph, const Parameters* pd, const State& in, const State& out, const State* snap,
                   const Rates& r, cudaStream_t s, const MaterialTable& mt, const MaterialTable& vw, float* rec,
                   bool stage, const SubstepQueue& q)
{
    if (ph->np <= 0) return LQ_OK;
    LQ_TRY(check_substeps(ph, "predictor", vw, q));
    const bool do_snap = snap && snap->pos;
    if (stage && (do_snap || out.pos == in.pos))
        return set_error(LQ_ERR_ARG, "predictor: a stage buffer needs its own output and no snapshot");
    if (ph->constitutive_model == 3 && !stage)
        return set_error(LQ_ERR_ARG, "predictor: constitutive model 3 runs in stage buffers only");
    State sn = do_snap ? *snap : State{nullptr, nullptr, nullptr, nullptr, nullptr};
    const int nb = blocks_for(ph->np, kBlock);
    const NbrArrays pk = rec ? nbr_arrays(rec, ph->np) : NbrArrays{nullptr, nullptr, nullptr};
    if (in.xlo && out.xlo)
        k_predict<true><<<nb, kBlock, 0, s>>>(pd, ph->np, ph->npb, in, out, sn, do_snap, r, mt, pk, stage);
    else
        k_predict<false><<<nb, kBlock, 0, s>>>(pd, ph->np, ph->npb, in, out, sn, do_snap, r, mt, pk, stage);
    LQ_TRY_CUDA(cudaGetLastError(), "k_predict");
    return launch_predict_substeps(ph, pd, in, out, r, s, vw, rec, q);
}

int launch_correct(const Parameters* ph, const Parameters* pd, const State& cur, const State& ini, const Rates& r,
                   cudaStream_t s)
{
    if (ph->npm <= 0) return LQ_OK;
    if (ph->constitutive_model == 3)
        return set_error(LQ_ERR_ARG, "corrector: constitutive model 3 needs a von Wolffersdorff table");
    k_correct<false><<<blocks_for(ph->npm, kBlock), kBlock, 0, s>>>(
        pd, ph->np, ph->npb, cur, ini, cur, r, nullptr, VerletCheck{nullptr, nullptr, 0.0f, 0.0f, nullptr, 0.0f},
        MaterialTable(), NbrArrays{nullptr, nullptr, nullptr});
    LQ_TRY_CUDA(cudaGetLastError(), "k_correct");
    return LQ_OK;
}

int launch_correct_into(const Parameters* ph, const Parameters* pd, const State& cur, const State& ini,
                        const Rates& r, int* health, const ListCheck& lists, cudaStream_t s, const MaterialTable& mt,
                        const MaterialTable& vw, float* rec, const SubstepQueue& q)
{
    if (ph->npm <= 0) return LQ_OK;
    LQ_TRY(check_substeps(ph, "corrector", vw, q));
    if (lists.xwide && !(lists.wide > lists.skin))
        return set_error(LQ_ERR_ARG, "corrector: the wide cut-off must exceed the skin");
    const VerletCheck vc = verlet_of(ph, lists);
    const int nb = blocks_for(ph->npm, kBlock);
    const NbrArrays pk = rec ? nbr_arrays(rec, ph->np) : NbrArrays{nullptr, nullptr, nullptr};
    if (ini.xlo)
        k_correct<true><<<nb, kBlock, 0, s>>>(pd, ph->np, ph->npb, cur, ini, ini, r, health, vc, mt, pk);
    else
        k_correct<false><<<nb, kBlock, 0, s>>>(pd, ph->np, ph->npb, cur, ini, ini, r, health, vc, mt, pk);
    LQ_TRY_CUDA(cudaGetLastError(), "k_correct");
    return launch_correct_substeps(ph, pd, ini, r, health, s, vw, rec, q);
}

}  // namespace lqb

/* ------------------------------------------------------------------ C ABI */

extern "C" int lq_predictor(const void* par_host, const void* par_device, float* pospres, float* velrhop,
                            float* idep, float* str, float* stn, float* pospres_ini, float* velrhop_ini,
                            float* idep_ini, float* str_ini, float* stn_ini, const float* accad, const float* spin,
                            const float* acestn, void* stream)
{
    if (!par_host || !par_device) return lqb::set_error(LQ_ERR_ARG, "lq_predictor: null Parameters");
    const Parameters* ph = static_cast<const Parameters*>(par_host);
    if (ph->npm == 0) return LQ_OK; /* reference returns before the snapshot too */
    if (!pospres || !velrhop || !idep || !str || !stn || !pospres_ini || !velrhop_ini || !idep_ini || !str_ini ||
        !stn_ini || !accad || !spin || !acestn)
        return lqb::set_error(LQ_ERR_ARG, "lq_predictor: null array");
    lqb::State st{(float4*)pospres, (float4*)velrhop, (float4*)idep, (tensor2d*)str, (tensor2d*)stn};
    lqb::State sn{(float4*)pospres_ini, (float4*)velrhop_ini, (float4*)idep_ini, (tensor2d*)str_ini,
                  (tensor2d*)stn_ini};
    lqb::Rates r{(float4*)accad, (float4*)spin, (tensor2d*)acestn};
    return lqb::launch_predict(ph, static_cast<const Parameters*>(par_device), st, st, &sn, r,
                               static_cast<cudaStream_t>(stream));
}

extern "C" int lq_corrector(const void* par_host, const void* par_device, float* pospres, float* velrhop,
                            float* idep, float* str, float* stn, const float* pospres_ini, const float* velrhop_ini,
                            const float* idep_ini, const float* str_ini, const float* stn_ini, const float* accad,
                            const float* spin, const float* acestn, void* stream)
{
    if (!par_host || !par_device) return lqb::set_error(LQ_ERR_ARG, "lq_corrector: null Parameters");
    const Parameters* ph = static_cast<const Parameters*>(par_host);
    if (ph->npm == 0) return LQ_OK;
    if (!pospres || !velrhop || !idep || !str || !stn || !pospres_ini || !velrhop_ini || !idep_ini || !str_ini ||
        !stn_ini || !accad || !spin || !acestn)
        return lqb::set_error(LQ_ERR_ARG, "lq_corrector: null array");
    lqb::State st{(float4*)pospres, (float4*)velrhop, (float4*)idep, (tensor2d*)str, (tensor2d*)stn};
    lqb::State in{(float4*)pospres_ini, (float4*)velrhop_ini, (float4*)idep_ini, (tensor2d*)str_ini,
                  (tensor2d*)stn_ini};
    lqb::Rates r{(float4*)accad, (float4*)spin, (tensor2d*)acestn};
    return lqb::launch_correct(ph, static_cast<const Parameters*>(par_device), st, in, r,
                               static_cast<cudaStream_t>(stream));
}

/* ------------------------------------------- C++ drop-in functions */

namespace {

void check_or_die(int st, const char* what)
{
    if (st != LQ_OK) {
        fprintf(stderr, "%s failed: %s\n", what, lq_last_error());
        exit(EXIT_FAILURE);
    }
}

}  // namespace

void Predictor(Parameters* par_host, Parameters* par_device, float4* pospres, float4* velrhop, float4* idep,
               tensor2d* str, tensor2d* stn, float4* pospres_ini, float4* velrhop_ini, float4* idep_ini,
               tensor2d* str_ini, tensor2d* stn_ini, float4* accad, float4* spin, tensor2d* acestn)
{
    check_or_die(lq_predictor(par_host, par_device, (float*)pospres, (float*)velrhop, (float*)idep, (float*)str,
                              (float*)stn, (float*)pospres_ini, (float*)velrhop_ini, (float*)idep_ini,
                              (float*)str_ini, (float*)stn_ini, (const float*)accad, (const float*)spin,
                              (const float*)acestn, nullptr),
                 "Predictor");
}

void Corrector(Parameters* par_host, Parameters* par_device, float4* pospres, float4* velrhop, float4* idep,
               tensor2d* str, tensor2d* stn, float4* pospres_ini, float4* velrhop_ini, float4* idep_ini,
               tensor2d* str_ini, tensor2d* stn_ini, float4* accad, float4* spin, tensor2d* acestn)
{
    check_or_die(lq_corrector(par_host, par_device, (float*)pospres, (float*)velrhop, (float*)idep, (float*)str,
                              (float*)stn, (const float*)pospres_ini, (const float*)velrhop_ini,
                              (const float*)idep_ini, (const float*)str_ini, (const float*)stn_ini,
                              (const float*)accad, (const float*)spin, (const float*)acestn, nullptr),
                 "Corrector");
}
