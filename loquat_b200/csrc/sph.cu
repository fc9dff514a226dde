/*
 * LOQUAT-B200 neighbour-loop kernels: particle interaction, Adami boundary
 * and Shepard stress filter, with their C ABI entry points and the C++
 * drop-in functions of the reference interface.
 *
 * Layout: the state is cell-sorted AoS as the reference stores it
 * (float4 position/velocity, 24-byte tensor2d).  Because cell keys are
 * z-fastest, the particles of three z-adjacent cells of one (x, y) column
 * are one contiguous slot range, so a 27-cell stencil is 9 contiguous runs
 * per layer; neighbouring threads (consecutive sorted particles) walk the
 * same runs and their loads hit L1.
 */
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <utility>
#include <vector>

#include <cub/device/device_scan.cuh>
#include <cub/device/device_select.cuh>
#include <thrust/iterator/counting_iterator.h>

#include "lq_internal.cuh"
#include "lq_lanes.h"
#include "lq_tile.h"
#include "lq_device.cuh"
#include "lq_integrate.cuh"
#include <adami_boundary.h>
#include <field_smoothing.h>
#include <particle_interaction.h>

namespace lqb {

namespace {

constexpr int kBlock = 128;

inline int blocks_for(long long n, int b) { return (int)((n + b - 1) / b); }

/* -------------------------------------------------------- interaction */
/* Formulation (weakly compressible SPH, Wendland C2, tension-positive
 * stress); the reference's implementation of this pass is closed
 * (src/particle_interaction.h:27-40):
 *   g      = C' (2 - q)^3 x_ij                    grad_i W_ij, q = r/h < 2
 *   drho  += m v_ij . g
 *   a     += m (sig_i/rho_i^2 + sig_j/rho_j^2) g  - m Pi_ij g  [+ m (R_i+R_j) f^4 g]
 *   L     -= (m/rho_j) v_ij (x) g
 * over both layers, j != i.  Pi_ij is Monaghan's viscosity with
 * mu = h v_ij.x_ij / (r^2 + eta) for approaching pairs; R is the diagonal
 * artificial stress -eps sig_aa / rho^2 of tensile components, f = W/W(dr).
 *
 * Neighbours are visited through lists: k_neighbor_list holds the candidates
 * of a warp's targets in its lanes, tests them against one target after the
 * other and writes each target's hits to its column of a global list; the
 * pair kernels then evaluate each particle's pairs from its list with every
 * lane busy.  The native driver
 * keeps the lists across steps (Verlet lists with a skin); the drop-in
 * ParticleInteraction builds them at each call in the caller's grid.  A
 * particle whose list overflowed walks its stencil directly (walk_stencil),
 * in the same order. */

struct PairConst {
    float ih, eta, mCg, Cw, avh, eps, iwdr, cut2;
    bool artp;
};

__device__ __forceinline__ PairConst load_pair_const(const Parameters* __restrict__ P)
{
    PairConst K;
    const float h = __ldg(&P->h);
    K.ih = __ldg(&P->i_h);
    K.eta = __ldg(&P->eta);
    /* every sum takes the factor m C' of its terms once, in rates_of */
    K.mCg = __ldg(&P->m) * __ldg(&P->kernel_gradient_normalization_par);
    K.Cw = __ldg(&P->kernel_normalization_par);
    /* -2 alpha cs h; zero without viscosity, so the pair body can evaluate
     * the term unconditionally (it then adds exact zeros) */
    K.avh = __ldg(&P->viscosity_type) == 1
                ? -2.0f * __ldg(&P->artificial_viscosity_alpha) * __ldg(&P->cs) * h
                : 0.0f;
    K.artp = __ldg(&P->artificial_pressure) == 1;
    K.eps = __ldg(&P->artificial_pressure_coefficient);
    K.iwdr = 1.0f / __ldg(&P->kernel_dr);
    K.cut2 = 4.0f * h * h * 1.0001f; /* candidate test; the pair body applies q < 2 exactly */
    return K;
}

/* The particle whose rates are being summed, and its running sums. */
struct Target {
    float4 x, v;
    float Sxx, Syy, Szz, Sxy, Sxz, Syz; /* sigma_i / rho_i^2 */
    float Rx, Ry, Rz;                   /* artificial stress of i */
    float drho, ax, ay, az;
    float cdrho, cax, cay, caz;         /* compensation terms (mixed form) */
    float l00, l01, l02, l10, l11, l12, l20, l21, l22;
};

/* Compensated (Kahan) accumulation: sum + y with the lost low-order part
 * carried in c. */
__device__ __forceinline__ void kahan_add(float& sum, float& c, float y)
{
    const float yy = y - c;
    const float t = sum + yy;
    c = (t - sum) - yy;
    sum = t;
}

__device__ __forceinline__ void load_target(const PairConst& K, const State& st, int i, bool active, Target& T)
{
    T.x = make_float4(0.f, 0.f, 0.f, 0.f);
    T.v = make_float4(0.f, 0.f, 0.f, 1.f);
    tensor2d si = make_tensor2d(0.0f);
    if (active) {
        T.x = __ldg(st.pos + i);
        T.v = __ldg(st.vel + i);
        si = load_t2(st.str, i);
    }
    const float ri2 = 1.0f / (T.v.w * T.v.w);
    T.Sxx = __fmul_rn(si.xx, ri2); T.Syy = __fmul_rn(si.yy, ri2); T.Szz = __fmul_rn(si.zz, ri2);
    T.Sxy = __fmul_rn(si.xy, ri2); T.Sxz = __fmul_rn(si.xz, ri2); T.Syz = __fmul_rn(si.yz, ri2);
    T.Rx = T.Ry = T.Rz = 0.f;
    if (K.artp) {
        T.Rx = si.xx > 0.f ? -K.eps * T.Sxx : 0.f;
        T.Ry = si.yy > 0.f ? -K.eps * T.Syy : 0.f;
        T.Rz = si.zz > 0.f ? -K.eps * T.Szz : 0.f;
    }
    T.drho = T.ax = T.ay = T.az = 0.f;
    T.cdrho = T.cax = T.cay = T.caz = 0.f;
    T.l00 = T.l01 = T.l02 = T.l10 = T.l11 = T.l12 = T.l20 = T.l21 = T.l22 = 0.f;
}

__device__ __forceinline__ float sqrt_approx(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

/* The factors of one pair's terms, without branches and without the common
 * factor m C' (rates_of applies it): the density rate is t3 vr, the
 * momentum t3 p and the velocity gradient -w (x) d.  (x_j, rho_j), v_j and
 * s_j = sigma_j / rho_j^2 are the neighbour's.  The kernel gradient is
 * t^3 x_ij with t = max(2 - q, 0), so a pair at q >= 2 adds zero to every
 * sum, and a pair of a particle with itself (the filler of a list's last
 * group) adds exact zeros: d = 0.
 *
 * The pair sums are bound by issue slots and the L1 data pipe, so the terms
 * are factored to the fewest operations: t^3 multiplies v_ij . x_ij (shared
 * by the density rate and the viscosity) and the contracted stress instead
 * of forming the gradient's three components, the viscosity enters as a
 * pressure on the diagonal of the stress sum, and each quotient is one
 * reciprocal: 57 arithmetic operations a pair and three of the special
 * function unit (about 70 and as many before; with the sums' other work
 * 115 -> 98 instructions an entry, 758 -> 703 us a launch on the 1.97 M
 * cylinder, 640 x 1, mixed form).  The viscosity is always evaluated (K.avh
 * is zero without it); kArtp adds the artificial stress.  Every product and
 * sum is contracted as written, so that all kernels that sum these terms in
 * one order give one result. */
struct PairFactors {
    float t3, vr, px, py, pz, wx, wy, wz, dx, dy, dz;
};

template <bool kArtp>
__device__ __forceinline__ PairFactors pair_factors(const PairConst& K, const Target& T, const float4& xj,
                                                    const float3& vj, const tensor2d& sj)
{
    PairFactors f;
    f.dx = T.x.x - xj.x;
    f.dy = T.x.y - xj.y;
    f.dz = T.x.z - xj.z;
    const float r2 = fmaf(f.dx, f.dx, fmaf(f.dy, f.dy, f.dz * f.dz));
    const float t = fmaxf(fmaf(-sqrt_approx(r2), K.ih, 2.0f), 0.0f);
    f.t3 = t * t * t;
    const float vx = T.v.x - vj.x, vy = T.v.y - vj.y, vz = T.v.z - vj.z;
    f.vr = fmaf(vx, f.dx, fmaf(vy, f.dy, vz * f.dz));
    /* Pi = -alpha cs h vr / ((r^2 + eta) rhobar) for vr < 0, rhobar = (rho_i + rho_j) / 2 */
    const float pi = __fmul_rn(K.avh * fminf(f.vr, 0.0f), rcp_approx((r2 + K.eta) * (T.v.w + xj.w)));
    float Txx = T.Sxx + sj.xx - pi, Tyy = T.Syy + sj.yy - pi, Tzz = T.Szz + sj.zz - pi;
    const float Txy = T.Sxy + sj.xy, Txz = T.Sxz + sj.xz, Tyz = T.Syz + sj.yz;
    if (kArtp) {
        /* W = Cw t^4 (q + 1/2), q = 2 - t where W is not zero */
        const float w = K.Cw * (t * f.t3) * (2.5f - t) * K.iwdr;
        const float w4 = (w * w) * (w * w);
        Txx = fmaf(fmaf(-K.eps, fmaxf(sj.xx, 0.0f), T.Rx), w4, Txx);
        Tyy = fmaf(fmaf(-K.eps, fmaxf(sj.yy, 0.0f), T.Ry), w4, Tyy);
        Tzz = fmaf(fmaf(-K.eps, fmaxf(sj.zz, 0.0f), T.Rz), w4, Tzz);
    }
    f.px = fmaf(Txx, f.dx, fmaf(Txy, f.dy, Txz * f.dz));
    f.py = fmaf(Txy, f.dx, fmaf(Tyy, f.dy, Tyz * f.dz));
    f.pz = fmaf(Txz, f.dx, fmaf(Tyz, f.dy, Tzz * f.dz));
    const float u = f.t3 * rcp_approx(xj.w);
    f.wx = u * vx;
    f.wy = u * vy;
    f.wz = u * vz;
    return f;
}

/* A pair's density-rate and momentum terms added to (drho, ax, ay, az), its
 * velocity-gradient terms to T. */
__device__ __forceinline__ void add_pair(const PairFactors& f, Target& T, float& drho, float& ax, float& ay, float& az)
{
    drho = fmaf(f.t3, f.vr, drho);
    ax = fmaf(f.t3, f.px, ax);
    ay = fmaf(f.t3, f.py, ay);
    az = fmaf(f.t3, f.pz, az);
    T.l00 = fmaf(-f.wx, f.dx, T.l00); T.l01 = fmaf(-f.wx, f.dy, T.l01); T.l02 = fmaf(-f.wx, f.dz, T.l02);
    T.l10 = fmaf(-f.wy, f.dx, T.l10); T.l11 = fmaf(-f.wy, f.dy, T.l11); T.l12 = fmaf(-f.wy, f.dz, T.l12);
    T.l20 = fmaf(-f.wz, f.dx, T.l20); T.l21 = fmaf(-f.wz, f.dy, T.l21); T.l22 = fmaf(-f.wz, f.dz, T.l22);
}

/* A neighbour's packed record as it is gathered. */
template <bool kPk>
struct PackedRecord {
    float4 xr, sa, sb;
    float vz;
};

template <bool kPk>
__device__ __forceinline__ void load_record(const NbrArrays& nb, int j, PackedRecord<kPk>& r)
{
    load_xs(nb, j, r.xr, r.sa);
    r.sb = __ldg(nb.sb + j);
    if (!kPk) r.vz = __ldg(nb.vz + j);
}

/* One pair from a gathered record. */
template <bool kArtp, bool kPk>
__device__ __forceinline__ void pair_terms(const PairConst& K, const PackedRecord<kPk>& r, Target& T, float& drho,
                                           float& ax, float& ay, float& az)
{
    const float3 vj = kPk ? unpack_velocity(r.sb.z, r.sb.w) : make_float3(r.sb.z, r.sb.w, r.vz);
    add_pair(pair_factors<kArtp>(K, T, r.xr, vj,
                                 make_tensor2d(r.sa.x, r.sa.y, r.sa.z, r.sa.w, r.sb.x, r.sb.y)),
             T, drho, ax, ay, az);
}

/* One pair from the state arrays (the walk of a target whose list
 * overflowed), every sum compensated pair by pair with kKahan. */
template <bool kKahan = false>
__device__ __forceinline__ void pair_body(const PairConst& K, const State& st, Target& T, int j)
{
    const float4 x = __ldg(st.pos + j);
    const float4 v = __ldg(st.vel + j);
    const float rinv = rcp_approx(v.w);
    const tensor2d s = load_t2(st.str, j) * (rinv * rinv);
    const float4 xj = make_float4(x.x, x.y, x.z, v.w);
    const float3 vj = make_float3(v.x, v.y, v.z);
    float d = 0.f, ax = 0.f, ay = 0.f, az = 0.f;
    add_pair(K.artp ? pair_factors<true>(K, T, xj, vj, s) : pair_factors<false>(K, T, xj, vj, s), T, d, ax, ay, az);
    if (kKahan) {
        kahan_add(T.drho, T.cdrho, d);
        kahan_add(T.ax, T.cax, ax);
        kahan_add(T.ay, T.cay, ay);
        kahan_add(T.az, T.caz, az);
    } else {
        T.drho += d;
        T.ax += ax;
        T.ay += ay;
        T.az += az;
    }
}

/* One pair into T's sums.  kKahan selects the mixed form: the density
 * and momentum sums compensated pair by pair, and the neighbour's velocity
 * gathered in the packed record. */
template <bool kKahan = false>
__device__ __forceinline__ void pair_body_rec(const PairConst& K, const NbrArrays& nb, Target& T, int j)
{
    PackedRecord<kKahan> r;
    load_record(nb, j, r);
    float d = 0.f, x = 0.f, y = 0.f, z = 0.f;
    if (K.artp)
        pair_terms<true>(K, r, T, d, x, y, z);
    else
        pair_terms<false>(K, r, T, d, x, y, z);
    if (kKahan) {
        kahan_add(T.drho, T.cdrho, d);
        kahan_add(T.ax, T.cax, x);
        kahan_add(T.ay, T.cay, y);
        kahan_add(T.az, T.caz, z);
    } else {
        T.drho += d;
        T.ax += x;
        T.ay += y;
        T.az += z;
    }
}

/* The target's rates from its sums; products rounded as such, whatever the
 * kernel goes on to do with them. */
__device__ __forceinline__ SlotRates rates_of(const Parameters* __restrict__ P, const PairConst& K, const Target& T)
{
    const float c = K.mCg, hc = 0.5f * K.mCg;
    SlotRates r;
    r.a = make_float4(fmaf(c, T.ax, __ldg(&P->acc_x)), fmaf(c, T.ay, __ldg(&P->acc_y)), fmaf(c, T.az, __ldg(&P->acc_z)),
                      __fmul_rn(c, T.drho));
    r.w = make_float4(__fmul_rn(hc, T.l10 - T.l01), __fmul_rn(hc, T.l20 - T.l02), __fmul_rn(hc, T.l21 - T.l12), 0.0f);
    r.de = make_tensor2d(__fmul_rn(c, T.l00), __fmul_rn(c, T.l11), __fmul_rn(c, T.l22),
                         __fmul_rn(hc, T.l01 + T.l10), __fmul_rn(hc, T.l02 + T.l20), __fmul_rn(hc, T.l12 + T.l21));
    return r;
}

__device__ __forceinline__ void store_rates(const Parameters* __restrict__ P, const PairConst& K, const Rates& rt,
                                            int i, const Target& T)
{
    const SlotRates r = rates_of(P, K, T);
    rt.accad[i] = r.a;
    rt.spin[i] = r.w;
    store_t2(rt.acestn, i, r.de);
}

/* The 27-cell walk of one particle (both layers), calling f(j) for every
 * candidate that passes the distance test, in the order shared by every
 * neighbour visit of this file: layer, then column (dy outer, dx inner),
 * then slot. */
template <class F>
__device__ __forceinline__ void walk_stencil(const Parameters* __restrict__ P, const PairConst& K, const State& st,
                                             const Cells& cells, int i, const float4& xi, F&& f,
                                             const Frames& fr = Frames())
{
    const int nx = __ldg(&P->cell_num_x), ny = __ldg(&P->cell_num_y), nz = __ldg(&P->cell_num_z);
    const int L = __ldg(&P->ncell_one_layer);
    const int cx = stencil_axis(xi.x, K.ih), cz = stencil_axis(xi.z, K.ih);
    int cy = stencil_axis(xi.y, K.ih);
    if (fr.rows) cy = frame_stencil_row(fr, __ldg(&st.idep[i].x), cy);
    const int zlo = max(cz - 1, 0), zhi = min(cz + 1, nz - 1);
    if (zlo > zhi) return;
    for (int layer = 0; layer < 2; ++layer) {
        const int off = layer ? L : 0;
        for (int col = 0; col < 9; ++col) {
            const int X = cx + (col % 3) - 1, Y = cy + (col / 3) - 1;
            if (X < 0 || X >= nx || Y < 0 || Y >= ny) continue;
            int s, e;
            if (!zrun_range(cells, off + (X * ny + Y) * nz, zlo, zhi, s, e)) continue;
            for (int j = s; j < e; ++j) {
                const float4 xj = __ldg(st.pos + j);
                const float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
                if (dx * dx + dy * dy + dz * dz < K.cut2 && j != i) f(j);
            }
        }
    }
}

#ifndef LQ_PAIR_MIN_BLOCKS
#define LQ_PAIR_MIN_BLOCKS 6   /* 128-thread blocks per SM: 80 registers */
#endif

constexpr int kListWarps = kBlock / 32;
constexpr int kListChunk = 128;     /* candidates a warp holds at once, four a lane */

/* Neighbour lists: list[k * stride + t] is the k-th neighbour slot of target
 * slot first + t, count[t] their number (entries past LQ_NBR_CAP are not
 * stored).  Candidates come from grid layers layer_lo..1 (0: both layers,
 * 1: material only) and are kept when r^2 < cut2, the cut-off (2h) plus any
 * skin, in the order of the walk: layer, column (dy outer, dx inner), slot.
 * A lane's own slot passes the test too: its pair adds exactly zero.  Along
 * z the walk covers every cell the target's cut-off sphere reaches (two
 * cells down or up when the particle lies within the skin of a cell face),
 * so a list holds all its particle's pairs within the cut-off in those
 * columns; across columns it covers the 3 x 3 around the particle's own,
 * which holds every pair within 2h.  A pair within 2h + skin that lies two
 * columns apart is left out: it is more than 2h apart when the list is
 * built, so until the next build its distance stays above 2h - skin
 * (q > 2 - skin/h), where the kernel factor (2 - q)^3 stays below
 * (skin/h)^3.
 *
 * A warp's targets are grouped by grid column; for each group the warp
 * walks the union of their stencils, one contiguous slot range per column
 * and layer, joined to one sequence of about 700 candidates.  The lanes
 * hold 128 of them at once from coalesced loads and test them against one
 * target after the other (broadcast from shared memory, each coordinate
 * twice, for the paired FP32 instructions that take two candidates); votes
 * give the target's hits as bit masks, from which its own lane then writes
 * its list.  Bound by issue slots.  With a lane per target and a broadcast
 * load per candidate, each candidate took four passes of the L1 data pipe
 * to reach the lanes (79 % busy) and eight instructions a lane instead of
 * six.  At 786 k
 * targets 377 us against 496, and in small cases, where the loads' latency
 * was the time, 107 us for all lists of the 5 k column against 204.
 *
 * With `shell` (the wide build of two-level lists) the hits are split: those
 * with r^2 < inner2 go to `list` (count_out[t] of them) and the rest to
 * shell (shell_count[t]), each list in hit order; each part stores at most
 * LQ_NBR_CAP entries. */
template <bool kSplit>
__global__ void __launch_bounds__(kBlock) k_neighbor_list(const Parameters* __restrict__ P, int first, int ntarget,
                                                          int layer_lo, float cut2, const float4* __restrict__ pos,
                                                          Cells cells, int* __restrict__ list,
                                                          int* __restrict__ count_out, int stride,
                                                          int* __restrict__ health, const float4* __restrict__ idep,
                                                          Frames fr, int* __restrict__ shell,
                                                          int* __restrict__ shell_count, float inner2,
                                                          const int* __restrict__ gate)
{
    if (gate && *gate == 0) return;     /* the whole grid leaves: no collective is split */
    __shared__ float4 target_xy[kListWarps][32];    /* x, x, y, y */
    __shared__ float2 target_z[kListWarps][32];     /* z, z */
    __shared__ int slot[kListWarps][kListChunk];
    __shared__ uint4 hits[kListWarps][32], ins[kListWarps][kSplit ? 32 : 1];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = first + t;
    const bool active = t < ntarget;
    const float ih = __ldg(&P->i_h);
    const int nx = __ldg(&P->cell_num_x), ny = __ldg(&P->cell_num_y), nz = __ldg(&P->cell_num_z);
    const int L = __ldg(&P->ncell_one_layer);
    const int np_all = __ldg(&P->np);
    const float4 xi = active ? __ldg(pos + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    target_xy[w][lane] = make_float4(xi.x, xi.x, xi.y, xi.y);
    target_z[w][lane] = make_float2(xi.z, xi.z);

    /* the z cells the particle's cut-off sphere reaches (a run walks the
     * group's union of them), so a lane's list never depends on which
     * other lanes share its group */
    const float cut = sqrtf(cut2);
    int cx = 0, cy = 0, czl = 0, czh = 0;
    if (active) {
        cx = stencil_axis(xi.x, ih);
        cy = stencil_axis(xi.y, ih);
        czl = stencil_axis(xi.z - cut, ih);
        czh = stencil_axis(xi.z + cut, ih);
        if (fr.rows) cy = frame_stencil_row(fr, __ldg(&idep[i].x), cy);
    }
    int ni = 0, ns = 0;
    unsigned todo = __ballot_sync(FULL, active);
    __syncwarp();
    while (todo) {
        const int leader = __ffs(todo) - 1;
        const int gx = __shfl_sync(FULL, cx, leader), gy = __shfl_sync(FULL, cy, leader);
        const bool mine = active && cx == gx && cy == gy;
        const unsigned group = __ballot_sync(FULL, mine);
        const int lo = __ffs(group) - 1, hi = 31 - __clz(group);
        todo &= ~group;
        const int zmin = __reduce_min_sync(FULL, mine ? czl : INT_MAX);
        const int zmax = __reduce_max_sync(FULL, mine ? czh : INT_MIN);
        const int zlo = max(zmin, 0), zhi = min(zmax, nz - 1);
        if (zlo > zhi) continue;
        /* lane r < 9 per layer: the slot range [s, s + len) of run r, which
         * begins at place `at` of the joined sequence */
        int s = 0, len = 0;
        {
            const int layer = layer_lo + lane / 9, col = lane % 9;
            const int X = gx + (col % 3) - 1, Y = gy + (col / 3) - 1;
            int e;
            if (layer < 2 && X >= 0 && X < nx && Y >= 0 && Y < ny &&
                zrun_range(cells, (layer ? L : 0) + (X * ny + Y) * nz, zlo, zhi, s, e) && lq_in_range(s, np_all) &&
                lq_in_range(e - 1, np_all))
                len = e - s;
        }
        int end = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL, end, o);
            if (lane >= o) end += v;
        }
        const int at = end - len, total = __shfl_sync(FULL, end, 31);
        unsigned runs = __ballot_sync(FULL, len > 0);       /* from the one that holds `base` on */
        for (int base = 0; base < total; base += kListChunk) {
            /* lane l holds places base + 32 c + l: their slots and, negated,
             * their positions, far beyond any cut-off past the end */
            int j[4] = {-1, -1, -1, -1};
            int last = 0;
            for (unsigned m = runs; m; m &= m - 1) {
                const int r = __ffs(m) - 1;
                const int ra = __shfl_sync(FULL, at, r), rs = __shfl_sync(FULL, s, r);
                if (ra >= base + kListChunk) break;
                last = r;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int q = base + 32 * c + lane;
                    if (q >= ra && q < total) j[c] = rs + (q - ra);
                }
            }
            runs &= ~0u << last;
            float4 x[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                x[c] = j[c] >= 0 && lq_in_range(j[c], np_all) ? __ldg(pos + j[c])
                                                              : make_float4(3.0e18f, 3.0e18f, 3.0e18f, 0.0f);
                slot[w][32 * c + lane] = j[c];
            }
            float2 mx[2], my[2], mz[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                mx[c] = make_float2(-x[2 * c].x, -x[2 * c + 1].x);
                my[c] = make_float2(-x[2 * c].y, -x[2 * c + 1].y);
                mz[c] = make_float2(-x[2 * c].z, -x[2 * c + 1].z);
            }
            /* the group's lanes are neighbours (slots of one column follow
             * one another); a lane between them that is not of the group
             * leaves its masks unread */
#pragma unroll 2
            for (int tt = lo; tt <= hi; ++tt) {
                const float4 xy = target_xy[w][tt];
                const float2 tx = make_float2(xy.x, xy.y), ty = make_float2(xy.z, xy.w), tz = target_z[w][tt];
                unsigned h[4], b[4];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const float2 dx = __fadd2_rn(tx, mx[c]), dy = __fadd2_rn(ty, my[c]), dz = __fadd2_rn(tz, mz[c]);
                    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                    h[2 * c] = __ballot_sync(FULL, r2.x < cut2);
                    h[2 * c + 1] = __ballot_sync(FULL, r2.y < cut2);
                    if (kSplit) {
                        b[2 * c] = __ballot_sync(FULL, r2.x < inner2);
                        b[2 * c + 1] = __ballot_sync(FULL, r2.y < inner2);
                    }
                }
                if (lane == 0) {
                    hits[w][tt] = make_uint4(h[0], h[1], h[2], h[3]);
                    if (kSplit) ins[w][tt] = make_uint4(b[0], b[1], b[2], b[3]);
                }
            }
            /* each lane's hits, in the sequence's order */
            __syncwarp();
            const uint4 none = make_uint4(0u, 0u, 0u, 0u);
            const uint4 h4 = mine ? hits[w][lane] : none, b4 = mine && kSplit ? ins[w][kSplit ? lane : 0] : none;
            const unsigned hit[4] = {h4.x, h4.y, h4.z, h4.w}, in[4] = {b4.x, b4.y, b4.z, b4.w};
            int c = 0;
            unsigned h = hit[0], b = in[0];
            for (;;) {
#pragma unroll
                for (int k = 1; k < 4; ++k)
                    if (h == 0 && c < k) {
                        c = k;
                        h = hit[k];
                        b = in[k];
                    }
                if (h == 0) break;
                const int bit = __ffs(h) - 1;
                h &= h - 1;
                const int hj = slot[w][32 * c + bit];
                if (kSplit && !(b >> bit & 1u)) {
                    if (ns < LQ_NBR_CAP) shell[(size_t)ns * stride + t] = hj;
                    ++ns;
                } else {
                    if (ni < LQ_NBR_CAP) list[(size_t)ni * stride + t] = hj;
                    ++ni;
                }
            }
            __syncwarp();
        }
    }
    if (active) {
        /* the list's last group of four filled up with the target itself
         * (the split build's lists are filled up by their renewal) */
        if (!kSplit)
            for (int k = ni; k < LQ_NBR_CAP && (k & 3); ++k) list[(size_t)k * stride + t] = i;
        count_out[t] = ni;
        if (kSplit) shell_count[t] = ns;
        if ((ni > LQ_NBR_CAP || ns > LQ_NBR_CAP) && health) atomicAdd(health + HEALTH_NBR_OVERFLOW, 1);
    }
}

/* Slot i's packed record; the slots below n2 also into nb2. */
template <bool kPk>
__global__ void __launch_bounds__(kBlock) k_pack_neighbors(int first, int np, State st, NbrArrays nb,
                                                           NbrArrays nb2, int n2)
{
    const int i = first + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    const float4 x = __ldg(st.pos + i);
    const float4 v = __ldg(st.vel + i);
    const tensor2d s = load_t2(st.str, i);
    pack_slot<kPk>(nb, i, x, v, s);
    if (i < n2) pack_slot<kPk>(nb2, i, x, v, s);
}

/* A list entry: each 128-byte row of a list is read once per launch, so it
 * bypasses L1 (no allocation) and leaves L1 to the neighbour data that the
 * targets of a block share. */
__device__ __forceinline__ int ld_list(const int* p)
{
    int v;
    asm("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

/* Two-level lists: the lists the stages read (cut-off 2h + skin) renewed
 * at the current positions without a search.  The wide build (cut-off
 * 2h + wide) wrote each target's pairs closer than inner = 2h + 2 skin -
 * wide into rows [0, ni) of the stages' list and the rest into its shell
 * list.  While no particle has moved (wide - skin) / 2 from its position at
 * that build (the corrector's check), a pair's distance has changed by less
 * than wide - skin, so every inner pair is still within 2h + skin and every
 * pair now within 2h + skin was within 2h + wide: the renewal keeps rows
 * [0, ni) as they are and appends, in their order, the shell entries now
 * within the cut-off.  Entries are fetched a group ahead so the position
 * gathers overlap.  Overflows keep LQ_NBR_CAP valid rows and a count above
 * it (the pair kernel then walks that target's stencil): a truncated shell
 * list fills the rows after the inner part with its stored entries. */
__global__ void __launch_bounds__(kBlock) k_list_refresh(int first, int ntarget, int np, float cut2,
                                                         const float4* __restrict__ pos,
                                                         const int* __restrict__ inner_count,
                                                         const int* __restrict__ shell,
                                                         const int* __restrict__ shell_count, int* __restrict__ list,
                                                         int* __restrict__ count, int stride,
                                                         int* __restrict__ health)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntarget) return;
    const int ni = __ldg(inner_count + t), ns = __ldg(shell_count + t);
    const int* p = shell + t;
    if (ni > LQ_NBR_CAP) {
        count[t] = ni;          /* rows [0, LQ_NBR_CAP) hold inner entries */
        return;
    }
    if (ns > LQ_NBR_CAP) {
        for (int k = 0; ni + k < LQ_NBR_CAP; ++k) list[(size_t)(ni + k) * stride + t] = ld_list(p + (size_t)k * stride);
        count[t] = ni + ns;
        return;
    }
    const int i = first + t;
    const float4 xi = __ldg(pos + i);
    /* groups of kG entries; the last group is filled up with the target's
     * own slot (a valid address; never kept) */
    constexpr int kG = 8;
    int nxt[kG];
#pragma unroll
    for (int u = 0; u < kG; ++u) nxt[u] = u < ns ? ld_list(p + (size_t)u * stride) : i;
    int n = ni;
    for (int k = 0; k < ns; k += kG) {
        int j[kG];
        float4 xj[kG];
#pragma unroll
        for (int u = 0; u < kG; ++u) {
            j[u] = nxt[u];
            nxt[u] = k + kG + u < ns ? ld_list(p + (size_t)(k + kG + u) * stride) : i;
        }
#pragma unroll
        for (int u = 0; u < kG; ++u) xj[u] = lq_in_range(j[u], np) ? __ldg(pos + j[u]) : xi;
#pragma unroll
        for (int u = 0; u < kG; ++u) {
            const float dx = xi.x - xj[u].x, dy = xi.y - xj[u].y, dz = xi.z - xj[u].z;
            if (k + u < ns && lq_in_range(j[u], np) && dx * dx + dy * dy + dz * dz < cut2) {
                if (n < LQ_NBR_CAP) list[(size_t)n * stride + t] = j[u];
                ++n;
            }
        }
    }
    for (int k = n; k < LQ_NBR_CAP && (k & 3); ++k) list[(size_t)k * stride + t] = i;
    count[t] = n;
    if (n > LQ_NBR_CAP && health) atomicAdd(health + HEALTH_NBR_OVERFLOW, 1);
}

/* Each target's list put into an order in which the lanes of a warp gather
 * from different banks.  The pair kernel's lanes take consecutive targets,
 * and row k of their lists is one gather per lane: eight lanes form one
 * pass over the banks when their records' slots differ modulo 8 (eight
 * 16-byte words per 128 bytes), and as many passes as the fullest residue
 * holds otherwise.  In the order of the cell walk the residues are as good
 * as random: about 26 passes for the two gathers of a warp's row, 12 being
 * the least.  Target t takes an entry of residue (t + k) mod 8 in row k
 * while it has one, else of the next residue that it has: about 16 (counted
 * on the cylinder's lists; with the gathers in separate 16-byte words the
 * launch went from 703 to 646 us at 1.97 M targets).  It pays where lists
 * last: a build costs 1.8 ms there and this pass 0.5, the two pair launches
 * of each of the 20 to 80 steps between builds gain 0.1 ms.
 *
 * One thread per target.  Its entries (kArrangeRows at a time) stand in
 * shared memory as one chain per residue (hd: the chain's first row, nxt:
 * the row after each), then leave in the rows' order.  Bound by the two
 * passes over the list rows and the chains' shared-memory latency.  A list
 * that overflowed is left as it is. */
constexpr int kArrangeRows = 96;    /* an ordinary list (about 80 entries) in one piece; 7 blocks per SM */
constexpr int kArrangeBlock = 64;
__global__ void __launch_bounds__(kArrangeBlock) k_list_arrange(int ntarget, const int* __restrict__ count, int* list,
                                                                int stride)
{
    __shared__ int ent[kArrangeRows][kArrangeBlock];
    __shared__ unsigned char nxt[kArrangeRows][kArrangeBlock], hd[8][kArrangeBlock];
    const int t = blockIdx.x * kArrangeBlock + threadIdx.x, x = threadIdx.x;
    if (t >= ntarget) return;
    const int n = __ldg(count + t);
    if (n > LQ_NBR_CAP) return;
    for (int base = 0; base < n; base += kArrangeRows) {
        const int m = min(n - base, kArrangeRows);
        int* p = list + (size_t)base * stride + t;
        unsigned have = 0;      /* bit r: residue r's chain has entries */
#pragma unroll 8
        for (int k = 0; k < m; ++k) {
            const int j = p[(size_t)k * stride], r = j & 7;
            ent[k][x] = j;
            nxt[k][x] = (have >> r & 1u) ? hd[r][x] : (unsigned char)255;
            hd[r][x] = (unsigned char)k;
            have |= 1u << r;
        }
        int k = 0;
        /* while every chain has an entry: eight rows at a time, one from each */
        for (const int w = t + base; k + 8 <= m && have == 255u; k += 8) {
            int row[8];
#pragma unroll
            for (int o = 0; o < 8; ++o) row[o] = hd[(w + o) & 7][x];
#pragma unroll
            for (int o = 0; o < 8; ++o) {
                if (!lq_in_range(row[o], m)) continue;
                const unsigned char next = nxt[row[o]][x];
                p[(size_t)(k + o) * stride] = ent[row[o]][x];
                hd[(w + o) & 7][x] = next;
                if (next == 255) have &= ~(1u << ((w + o) & 7));
            }
        }
        for (; k < m; ++k) {
            const int w = (t + base + k) & 7;
            const int r = (w + __ffs((int)((have | have << 8) >> w)) - 1) & 7;
            const int row = hd[r][x];
            if (!lq_in_range(row, m)) break;
            const unsigned char next = nxt[row][x];
            p[(size_t)k * stride] = ent[row][x];
            hd[r][x] = next;
            if (next == 255) have &= ~(1u << r);
        }
    }
}

/* The sums over one target's list (entry k at p[k * stride]), in groups of
 * four entries; the list's builder has filled the last group up with the
 * target itself (exact zeros), so a group has no branch and no test.  A
 * group's four records are gathered together and the next group's entries
 * are fetched a group ahead, so the dependent gathers do not wait on the
 * list stream.  The compensated (mixed) form adds each group's plain sum of
 * four pairs to the compensated sums and reads the packed velocity. */
template <bool kKahan, bool kArtp>
__device__ __forceinline__ void list_sums(const PairConst& K, const NbrArrays& nb, Target& T, const int* p, int n,
                                          int stride, int i, int np)
{
    const size_t step4 = 4 * (size_t)stride;
    auto entry = [&](int u) {
        const int j = ld_list(p + (size_t)u * stride);
        return lq_in_range(j, np) ? j : i;
    };
    if (n <= 0) return;
    int cur[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) cur[u] = entry(u);
    for (int k = 0; k < n; k += 4) {
        if (k + 4 < n) p += step4;      /* the last group fetches its own entries again */
        int nxt[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) nxt[u] = entry(u);
        PackedRecord<kKahan> r[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) load_record(nb, cur[u], r[u]);
        if (kKahan) {
            float d = 0.f, x = 0.f, y = 0.f, z = 0.f;
#pragma unroll
            for (int u = 0; u < 4; ++u) pair_terms<kArtp>(K, r[u], T, d, x, y, z);
            kahan_add(T.drho, T.cdrho, d);
            kahan_add(T.ax, T.cax, x);
            kahan_add(T.ay, T.cay, y);
            kahan_add(T.az, T.caz, z);
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) pair_terms<kArtp>(K, r[u], T, T.drho, T.ax, T.ay, T.az);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) cur[u] = nxt[u];
    }
}

/* What a stage's pair kernel does with a target's rates (StageOps): kStage 0
 * stores them, 1 and 2 take the target's predictor or corrector step at
 * once. */
struct StageTail {
    State in, out;          /* 1: state to stage buffer; 2: the snapshot, updated in place (out unused) */
    MaterialTable mt;
    NbrArrays nbw;          /* the records of the stage that follows */
    int* health;
    VerletCheck verlet;
    bool keep_rates;        /* also store what later kernels of the stage read */
};

/* A target's step from its finished sums. */
template <bool kKahan, int kStage>
__device__ __forceinline__ void integrate_target(const Parameters* __restrict__ P, const PairConst& K, const Target& T,
                                                 const State& st, const Rates& rt, int i, const StageTail& tail)
{
    const SlotRates r = rates_of(P, K, T);
    if (tail.keep_rates) {
        rt.accad[i] = r.a;
        rt.spin[i] = r.w;
        store_t2(rt.acestn, i, r.de);
    }
    if (kStage == 1)
        predict_slot<kKahan>(P, i, tail.in, tail.out, r, tail.mt, tail.nbw, true, tail.in.pos[i], tail.in.vel[i],
                             tail.in.idep[i], load_t2_rw(tail.in.str, i), make_tensor2d(0.0f));
    else
        correct_slot<kKahan>(P, i, __ldg(&st.pos[i].w), tail.in.idep[i], tail.in, tail.in, r, tail.mt, tail.nbw,
                             tail.health, tail.verlet);
}

/* Pair sums over the lists from the packed neighbour arrays; a particle
 * whose list overflowed walks its stencil over the state arrays instead.
 * kThreads x kMinBlocks sets the register cap (kPairShapes).
 *
 * With kStage 1 or 2 the target is integrated where its sums end: the
 * 56 bytes of rates are neither written nor read back, and the integrator's
 * traffic, which as a kernel of its own runs at the memory's pace with the
 * SMs' arithmetic idle, overlaps the other warps' pair sums: a step of
 * the 1.97 M cylinder takes 1401 us so and 1501 with the integrators as
 * kernels of their own (131 us each after pair launches of 605), the
 * 5 k column 69 and 75.  The
 * step writes the records that the next stage gathers, so the two stages'
 * records are separate arrays: this one's are still being read.  At 80
 * registers the mixed form spills 76 bytes (stage 1) and 156 (stage 2), all
 * in the FP64 integration after the sums; at 96 24 and 88, at 72 160 and 244.
 * The plain form spills none. */
template <bool kKahan, int kThreads, int kMinBlocks, int kStage>
__global__ void __launch_bounds__(kThreads, kMinBlocks) k_interaction_rec(
    const Parameters* __restrict__ P, int np, int npb, State st, Rates rt, Cells cells, const int* __restrict__ list,
    const int* __restrict__ count, int stride, Frames fr, NbrArrays nb, const int* __restrict__ order,
    const int* __restrict__ rows, StageTail tail)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= np - npb) return;
    /* thread g takes target order[g] (tile order) or target g (slot order) */
    const int t = order ? __ldg(order + g) : g;
    if (!lq_in_range(t, np - npb)) return;
    const int i = npb + t;
    const PairConst K = load_pair_const(P);
    Target T;
    load_target(K, st, i, true, T);
    /* with rows: target t's list is row rows[t] (-1: none), whose entries
     * index records packed in that other slot order, the target's own at
     * npb + row (the filler of the last group) */
    int row = t, self = i;
    if (kStage == 0 && rows) {
        row = __ldg(rows + t);
        if (!lq_in_range(row + 1, np - npb + 1)) row = -1;
        self = npb + row;
    }
    const int n = row >= 0 ? __ldg(count + row) : LQ_NBR_CAP + 1;
    if (n <= LQ_NBR_CAP) {
        if (K.artp)
            list_sums<kKahan, true>(K, nb, T, list + row, n, stride, self, np);
        else
            list_sums<kKahan, false>(K, nb, T, list + row, n, stride, self, np);
    } else {
        walk_stencil(P, K, st, cells, i, T.x, [&](int j) { pair_body<kKahan>(K, st, T, j); }, fr);
    }
    if (kStage == 0) {
        store_rates(P, K, rt, i, T);
        return;
    }
    integrate_target<kKahan, kStage>(P, K, T, st, rt, i, tail);
}

/* The pair kernel for few targets: a team of 16 lanes per target, with the
 * sums of the thread-per-target form bit for bit.  A thread's list of about
 * 80 entries is a chain of 20 groups of dependent gathers and about 8000
 * instructions; below some 30 k targets there are too few warps to hide it
 * and the launch takes 23 us however few there are.  Here each lane forms the
 * factors of one entry in 16 (the bulk of the work, in any order) and puts
 * them into shared memory; then the lanes each own one of the target's 13
 * sums and add the 16 terms in the list's order, in the groups of four of
 * list_sums.  One warp of the block then integrates its targets.  A launch of
 * 5 k targets takes 15 us instead of 23, one of 12 k 29 instead of 24: three
 * times the work per target. */
constexpr int kTeam = 16;
constexpr int kTeamBlock = 128;
template <bool kKahan, int kStage>
__global__ void __launch_bounds__(kTeamBlock) k_interaction_team(
    const Parameters* __restrict__ P, int np, int npb, State st, Rates rt, Cells cells, const int* __restrict__ list,
    const int* __restrict__ count, int stride, Frames fr, NbrArrays nb, StageTail tail)
{
    __shared__ __align__(16) float val[kTeamBlock / kTeam][11][kTeam + 4];   /* rows on different banks */
    __shared__ float sums[13][kTeamBlock / kTeam];
    const int team = threadIdx.x / kTeam, c = threadIdx.x % kTeam;
    const unsigned mates = 0xffffu << (threadIdx.x & 16);
    const int first = npb + blockIdx.x * (kTeamBlock / kTeam);
    const int i = first + team;
    const PairConst K = load_pair_const(P);
    Target T;
    load_target(K, st, i < np ? i : first, true, T);
    const int n = i < np ? __ldg(count + i - npb) : 0;
    if (n <= LQ_NBR_CAP) {
        /* the rows of val that lane c's sum multiplies: t3 and one of
         * (vr, p), or one of -w and one of d; lanes 13 to 15 shadow 12 */
        const int s = min(c, 12);
        const int ra = s < 4 ? 0 : 5 + (s - 4) / 3, rb = s < 4 ? 1 + s : 8 + (s - 4) % 3;
        const bool compensated = kKahan && s < 4;
        const int n4 = (n + 3) & ~3;    /* the rows that the list's builder filled */
        const int* p = list + (i - npb);
        float sum = 0.0f, comp = 0.0f;
        int j = c < n4 ? ld_list(p + (size_t)c * stride) : i;
        for (int base = 0; base < n4; base += kTeam) {
            PackedRecord<kKahan> r;
            load_record(nb, lq_in_range(j, np) ? j : i, r);
            const int k = base + kTeam + c;
            j = k < n4 ? ld_list(p + (size_t)k * stride) : i;
            const float3 vj = kKahan ? unpack_velocity(r.sb.z, r.sb.w) : make_float3(r.sb.z, r.sb.w, r.vz);
            const tensor2d sj = make_tensor2d(r.sa.x, r.sa.y, r.sa.z, r.sa.w, r.sb.x, r.sb.y);
            const PairFactors f = K.artp ? pair_factors<true>(K, T, r.xr, vj, sj) : pair_factors<false>(K, T, r.xr, vj, sj);
            float(&v)[11][kTeam + 4] = val[team];
            v[0][c] = f.t3;
            v[1][c] = f.vr;
            v[2][c] = f.px;
            v[3][c] = f.py;
            v[4][c] = f.pz;
            v[5][c] = -f.wx;
            v[6][c] = -f.wy;
            v[7][c] = -f.wz;
            v[8][c] = f.dx;
            v[9][c] = f.dy;
            v[10][c] = f.dz;
            __syncwarp(mates);
#pragma unroll
            for (int m = 0; m < kTeam / 4; ++m)
                if (base + 4 * m < n4) {
                    const float4 a = *reinterpret_cast<const float4*>(&v[ra][4 * m]);
                    const float4 b = *reinterpret_cast<const float4*>(&v[rb][4 * m]);
                    float d = compensated ? 0.0f : sum;
                    d = fmaf(a.x, b.x, d);
                    d = fmaf(a.y, b.y, d);
                    d = fmaf(a.z, b.z, d);
                    d = fmaf(a.w, b.w, d);
                    if (compensated)
                        kahan_add(sum, comp, d);
                    else
                        sum = d;
                }
            __syncwarp(mates);
        }
        if (c < 13) sums[c][team] = sum;
    } else if (c == 0) {
        walk_stencil(P, K, st, cells, i, T.x, [&](int j) { pair_body<kKahan>(K, st, T, j); }, fr);
        const float of[13] = {T.drho, T.ax, T.ay, T.az, T.l00, T.l01, T.l02, T.l10, T.l11, T.l12, T.l20, T.l21, T.l22};
#pragma unroll
        for (int k = 0; k < 13; ++k) sums[k][team] = of[k];
    }
    __syncthreads();
    const int x = threadIdx.x;
    if (x >= kTeamBlock / kTeam || first + x >= np) return;
    T.drho = sums[0][x];
    T.ax = sums[1][x]; T.ay = sums[2][x]; T.az = sums[3][x];
    T.l00 = sums[4][x]; T.l01 = sums[5][x]; T.l02 = sums[6][x];
    T.l10 = sums[7][x]; T.l11 = sums[8][x]; T.l12 = sums[9][x];
    T.l20 = sums[10][x]; T.l21 = sums[11][x]; T.l22 = sums[12][x];
    integrate_target<kKahan, kStage>(P, K, T, st, rt, first + x, tail);
}

/* ------------------------------------------------- tile order of targets */
/* The pair kernel's targets in tile order (lq_tile.h has the index
 * arithmetic): tiles of 3 x 3 columns by tz cells, each tile column one run
 * of consecutive slots.  A block of the pair kernel then holds a compact
 * box of targets whose neighbourhood fits in L1, instead of a thin z-run of
 * one column whose neighbours the next block on the SM does not share. */
__global__ void __launch_bounds__(kBlock) k_tile_segments(const int* __restrict__ start, TileGrid tg, int npb,
                                                          int np, int* __restrict__ seg_beg,
                                                          int* __restrict__ seg_len)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= tg.nseg) return;
    int b, len;
    tile_segment(tg, start, npb, np, s, &b, &len);
    seg_beg[s] = b;
    seg_len[s] = len;
}

/* One warp per segment writes its targets (slot - npb) at the segment's
 * offset. */
__global__ void __launch_bounds__(kBlock) k_tile_fill(int nseg, int npb, int npm, const int* __restrict__ seg_beg,
                                                      const int* __restrict__ seg_len,
                                                      const int* __restrict__ seg_off, int* __restrict__ order)
{
    const int w = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (w >= nseg) return;
    const int b = __ldg(seg_beg + w), n = __ldg(seg_len + w), o = __ldg(seg_off + w);
    for (int k = lane; k < n; k += 32)
        if (o + k < npm) order[o + k] = b + k - npb;
}

/* Warp-cooperative form: a group of G lanes (G = 8 or 32) shares one
 * target, lane g taking list entries g, g + G, ...; the group's partial sums
 * are combined with shuffle reductions.  With few targets (a small case) a
 * thread per target leaves most of the GPU idle and each thread's chain of
 * dependent gathers long; groups give G times the parallelism.  In the
 * compensated form each lane keeps its Kahan pair and the reduction adds
 * sum - compensation. */
template <int G>
__device__ __forceinline__ float group_sum(float v)
{
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, G);
    return v;
}

template <bool kKahan, int G>
__global__ void __launch_bounds__(128) k_interaction_group(const Parameters* __restrict__ P, int np, int npb,
                                                           State st, Rates rt, Cells cells,
                                                           const int* __restrict__ list,
                                                           const int* __restrict__ count, int stride, Frames fr,
                                                           NbrArrays nb)
{
    const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
    const int g = threadIdx.x % G;
    const int t = gid;
    const int i = npb + t;
    const bool active = i < np;      /* whole groups leave together: no early return before the shuffles */
    const PairConst K = load_pair_const(P);
    Target T;
    load_target(K, st, active ? i : npb, active, T);
    const int n = active ? __ldg(count + t) : 0;
    if (n <= LQ_NBR_CAP) {
        for (int k = g; k < n; k += G) {
            const int j = __ldg(list + (size_t)k * stride + t);
            if (lq_in_range(j, np)) pair_body_rec<kKahan>(K, nb, T, j);
        }
    } else if (g == 0) {
        walk_stencil(P, K, st, cells, i, T.x, [&](int j) { pair_body<kKahan>(K, st, T, j); }, fr);
    }
    if (kKahan) {
        T.drho -= T.cdrho;
        T.ax -= T.cax;
        T.ay -= T.cay;
        T.az -= T.caz;
    }
    T.drho = group_sum<G>(T.drho);
    T.ax = group_sum<G>(T.ax);
    T.ay = group_sum<G>(T.ay);
    T.az = group_sum<G>(T.az);
    T.l00 = group_sum<G>(T.l00); T.l01 = group_sum<G>(T.l01); T.l02 = group_sum<G>(T.l02);
    T.l10 = group_sum<G>(T.l10); T.l11 = group_sum<G>(T.l11); T.l12 = group_sum<G>(T.l12);
    T.l20 = group_sum<G>(T.l20); T.l21 = group_sum<G>(T.l21); T.l22 = group_sum<G>(T.l22);
    if (active && g == 0) store_rates(P, K, rt, i, T);
}

/* ------------------------------------- drop-in Adami and Shepard filter */
/* The sums of the reference's two kernels that walk the material layer
 * (src/adami_boundary.cu:27-123, src/field_smoothing.cu:65-121): sigma_j
 * V_j W in S, x_ij V_j W and V_j W in acc, over the 27 cells around a
 * target.  Eight lanes share a target: they test its candidates eight (two
 * times eight) at a time, queue those within 2h in shared memory and then
 * form the terms of eight queued ones at once, so the square root, the
 * quotient and the loads of a term are done by full groups; one thread per
 * target ran them for the one candidate in six that passed, with the other
 * lanes waiting, as a chain of dependent loads (8 warps per SM in the wall's
 * case).  Bound by issue slots (78 %), so a term's distance is a plain square
 * root of the squared sum (norm3df, which guards against overflow of the
 * squares, cost 18 us of 400) and its two factors are multiplied once.  The
 * wall of 116 k particles takes 20.6 us instead of 84, the filter over 402 k
 * soil particles 376 instead of 674; groups that voted and looped each by
 * themselves ran one after another (754).
 *
 * Where every target of a warp has at most kCellFew candidates, testing them
 * column by column leaves most lanes idle: they are queued untested, and a
 * warp without any ends there.  A sheet of 1 M particles in one layer with 1.4,
 * 2.6 and 4 a cell: filter 147, 167 and 202 us so, 225, 240 and 242 column by
 * column; up to 32 or 64 candidates instead of 40 it is slower for 36, or for
 * 61.  One thread per target is still faster there (119, 142 and 190 us),
 * where latency is hidden by many targets, but by far the slower one with
 * fewer targets or more candidates. */
constexpr int kCellLanes = 8;
constexpr int kCellQueue = 64;
constexpr int kCellFew = 40;

struct CellSums {
    tensor2d S;
    float4 acc;     /* x_ij V_j W, and V_j W in w */
};

/* Cell c's slots; false when it is empty. */
__device__ __forceinline__ bool cell_range(const Cells& c, int cell, int& s, int& e)
{
    s = __ldg(c.beg + cell);
    if (s == -1) return false;
    e = __ldg(c.end + cell);
    return true;
}

/* The whole warp calls it, its four groups in step (votes and loops are the
 * warp's, so the groups never run one after another); a group with active
 * false adds nothing. */
__device__ __forceinline__ CellSums sum_material_cells(const Parameters* __restrict__ P, const State& st,
                                                       const Cells& cells, bool active, const float4& xi, int* queue)
{
    const unsigned FULL = 0xffffffffu;
    const int g = threadIdx.x % kCellLanes;
    const unsigned shift = threadIdx.x & 31 & ~(kCellLanes - 1), below = (1u << g) - 1u;
    const float ih = __ldg(&P->i_h), m = __ldg(&P->m), Cw = __ldg(&P->kernel_normalization_par);
    const float h = __ldg(&P->h), cut2 = 4.0f * h * h * 1.0001f;    /* q < 2 is tested exactly below */
    const int nx = __ldg(&P->cell_num_x), ny = __ldg(&P->cell_num_y), nz = __ldg(&P->cell_num_z);
    const int L = __ldg(&P->ncell_one_layer);
    const int cx = stencil_axis(xi.x, ih), cy = stencil_axis(xi.y, ih), cz = stencil_axis(xi.z, ih);
    const int zlo = max(cz - 1, 0), zhi = active ? min(cz + 1, nz - 1) : -1;
    CellSums r{make_tensor2d(0.0f), make_float4(0.f, 0.f, 0.f, 0.f)};
    int n = 0;
    auto drain = [&]() {
        __syncwarp();
        for (int k = g; __any_sync(FULL, k < n); k += kCellLanes) {
            if (k >= n) continue;
            const int j = queue[k];
            const float4 xj = __ldg(st.pos + j);
            const float3 d = make_float3(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z);
            const float q = sqrtf(fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z))) * ih;
            if (q < 2.0f) {
                const float ker = Cw * (2.0f - q) * (2.0f - q) * (2.0f - q) * (2.0f - q) * (q + 0.5f);
                const float vol = m / __ldg(&st.vel[j].w);
                const tensor2d sj = load_t2(st.str, j);
                const float kv = ker * vol;
                r.S.xx += sj.xx * kv;
                r.S.yy += sj.yy * kv;
                r.S.zz += sj.zz * kv;
                r.S.xy += sj.xy * kv;
                r.S.xz += sj.xz * kv;
                r.S.yz += sj.yz * kv;
                r.acc.x += d.x * kv;
                r.acc.y += d.y * kv;
                r.acc.z += d.z * kv;
                r.acc.w += kv;
            }
        }
        __syncwarp();
        n = 0;
    };
    /* the candidates of each group's slots [s, e) */
    auto test = [&](int s, int e) {
        for (int base = s; __any_sync(FULL, base < e); base += 2 * kCellLanes) {
            const int j0 = base + g, j1 = j0 + kCellLanes;
            float4 x0 = xi, x1 = xi;
            if (j0 < e) x0 = __ldg(st.pos + j0);
            if (j1 < e) x1 = __ldg(st.pos + j1);
            const float ax = xi.x - x0.x, ay = xi.y - x0.y, az = xi.z - x0.z;
            const float bx = xi.x - x1.x, by = xi.y - x1.y, bz = xi.z - x1.z;
            const bool h0 = j0 < e && ax * ax + ay * ay + az * az < cut2;
            const bool h1 = j1 < e && bx * bx + by * by + bz * bz < cut2;
            const unsigned m0 = __ballot_sync(FULL, h0) >> shift & 0xffu, m1 = __ballot_sync(FULL, h1) >> shift & 0xffu;
            if (h0) queue[n + __popc(m0 & below)] = j0;
            n += __popc(m0);
            if (h1) queue[n + __popc(m1 & below)] = j1;
            n += __popc(m1);
            if (__any_sync(FULL, n > kCellQueue - 2 * kCellLanes)) drain();
        }
    };
    /* lane g finds the slots of column g of the 3 x 3 (lane 0 also those of
     * column 8): one range while the column's cells follow one another in
     * the slots, as they do in a grid sorted by the cell key */
    int s0[2] = {0, 0}, e0[2] = {0, 0};
    bool apart[2] = {false, false};
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int col = t * kCellLanes + g;
        const int X = cx + col % 3 - 1, Y = cy + col / 3 - 1;
        if (col >= 9 || X < 0 || X >= nx || Y < 0 || Y >= ny) continue;
        const int cell = L + (X * ny + Y) * nz + zlo;
        int b[3], f[3];
#pragma unroll
        for (int z = 0; z < 3; ++z) {
            const bool in = zlo + z <= zhi;
            b[z] = in ? __ldg(cells.beg + cell + z) : -1;
            f[z] = in ? __ldg(cells.end + cell + z) : -1;
        }
#pragma unroll
        for (int z = 0; z < 3; ++z) {
            if (b[z] == -1 || f[z] <= b[z]) continue;   /* empty, by either mark */
            if (e0[t] == 0) {
                s0[t] = b[z];
            } else if (b[z] != e0[t]) {
                apart[t] = true;
            }
            e0[t] = f[z];
        }
    }
    const bool any_apart = __any_sync(FULL, apart[0] || apart[1]);
    const int len = e0[0] - s0[0];
    int upto = len;     /* of this lane's and the lanes' before it */
#pragma unroll
    for (int o = 1; o < kCellLanes; o <<= 1) {
        const int v = __shfl_up_sync(FULL, upto, o, kCellLanes);
        if (g >= o) upto += v;
    }
    const int eight = __shfl_sync(FULL, upto, kCellLanes - 1, kCellLanes);
    const int last = __shfl_sync(FULL, s0[1], 0, kCellLanes), last_len = __shfl_sync(FULL, e0[1], 0, kCellLanes) - last;
    if (!any_apart && __all_sync(FULL, eight + last_len <= kCellFew)) {
        /* few candidates: all of them queued untested */
        if (!__any_sync(FULL, eight + last_len > 0)) return r;
        for (int k = 0; __any_sync(FULL, k < len); ++k)
            if (k < len) queue[upto - len + k] = s0[0] + k;
        for (int k = g; k < last_len; k += kCellLanes) queue[eight + k] = last + k;
        n = eight + last_len;
    } else {
        for (int c = 0; c < 9; ++c) {
            const int t = c / kCellLanes, l = c % kCellLanes;
            const int cs = __shfl_sync(FULL, t ? s0[1] : s0[0], l, kCellLanes);
            const int ce = __shfl_sync(FULL, t ? e0[1] : e0[0], l, kCellLanes);
            if (!any_apart) {
                if (__any_sync(FULL, cs < ce)) test(cs, ce);
                continue;
            }
            /* some column's cells are apart: every column cell by cell */
            const bool cell_by_cell = __shfl_sync(FULL, (int)(t ? apart[1] : apart[0]), l, kCellLanes);
            for (int dz = 0; dz < 3; ++dz) {
                int b = dz == 0 ? cs : 0, f = dz == 0 ? ce : 0;
                if (cell_by_cell) {
                    const int z = zlo + dz;
                    b = f = 0;
                    if (z > zhi || !cell_range(cells, L + ((cx + c % 3 - 1) * ny + cy + c / 3 - 1) * nz + z, b, f))
                        b = f = 0;
                }
                test(b, f);
            }
        }
    }
    drain();
    float* v[10] = {&r.S.xx, &r.S.yy, &r.S.zz, &r.S.xy, &r.S.xz, &r.S.yz, &r.acc.x, &r.acc.y, &r.acc.z, &r.acc.w};
#pragma unroll
    for (int k = 0; k < 10; ++k)
#pragma unroll
        for (int o = kCellLanes / 2; o > 0; o >>= 1) *v[k] += __shfl_xor_sync(FULL, *v[k], o, kCellLanes);
    return r;
}

__global__ void __launch_bounds__(kBlock) k_adami(const Parameters* __restrict__ P, int npb, State st, Cells cells)
{
    __shared__ int queue[kBlock / kCellLanes][kCellQueue];
    const int i = lane_target(blockIdx.x, threadIdx.x, kBlock, kCellLanes);
    const bool active = i < npb;
    const float4 xi = active ? __ldg(st.pos + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    const CellSums r = sum_material_cells(P, st, cells, active, xi, queue[threadIdx.x / kCellLanes]);
    if (threadIdx.x % kCellLanes == 0 && r.acc.w > 0.0f) {
        const float rho0 = __ldg(&P->rho0);
        tensor2d out;
        out.xx = (r.S.xx - rho0 * __ldg(&P->acc_x) * r.acc.x) / r.acc.w;
        out.yy = (r.S.yy - rho0 * __ldg(&P->acc_y) * r.acc.y) / r.acc.w;
        out.zz = (r.S.zz - rho0 * __ldg(&P->acc_z) * r.acc.z) / r.acc.w;
        out.xy = r.S.xy / r.acc.w;
        out.xz = r.S.xz / r.acc.w;
        out.yz = r.S.yz / r.acc.w;
        store_t2(st.str, i, out);
    }
}

/* Material layer, self included, no guard on a zero weight sum (reference
 * kernel src/field_smoothing.cu:65-121). */
__global__ void __launch_bounds__(kBlock) k_shepard(const Parameters* __restrict__ P, int np, int npb, State st,
                                                    tensor2d* __restrict__ out_str, Cells cells)
{
    __shared__ int queue[kBlock / kCellLanes][kCellQueue];
    const int i = npb + lane_target(blockIdx.x, threadIdx.x, kBlock, kCellLanes);
    const bool active = i < np;
    const float4 xi = active ? __ldg(st.pos + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    CellSums r = sum_material_cells(P, st, cells, active, xi, queue[threadIdx.x / kCellLanes]);
    if (!active || threadIdx.x % kCellLanes != 0) return;
    const float w = r.acc.w;
    r.S.xx /= w;
    r.S.yy /= w;
    r.S.zz /= w;
    r.S.xy /= w;
    r.S.xz /= w;
    r.S.yz /= w;
    store_t2(out_str, i, r.S);
}

/* A boundary particle's stress from the sums of its extrapolation (sigma_j
 * V_j W in S, x_ij V_j W and V_j W in acc), into both state buffers and both
 * stages' records; a boundary particle's velocity and density stay as the
 * list build packed them, only its stress words change. */
__device__ __forceinline__ void store_wall_stress(const Parameters* __restrict__ P, const State& st, int i,
                                                  const tensor2d& S, const float4& acc, tensor2d* str2,
                                                  const NbrArrays& nb, const NbrArrays& nb2)
{
    const float rho0 = __ldg(&P->rho0);
    const float inv = 1.0f / acc.w;
    tensor2d out;
    out.xx = (S.xx - rho0 * __ldg(&P->acc_x) * acc.x) * inv;
    out.yy = (S.yy - rho0 * __ldg(&P->acc_y) * acc.y) * inv;
    out.zz = (S.zz - rho0 * __ldg(&P->acc_z) * acc.z) * inv;
    out.xy = S.xy * inv;
    out.xz = S.xz * inv;
    out.yz = S.yz * inv;
    store_t2(st.str, i, out);
    store_t2(str2, i, out);
    const float rho = __ldg(&st.vel[i].w);
    store_packed_stress(nb, i, rho, out);
    store_packed_stress(nb2, i, rho, out);
}

/* ------------------------------------------------- list-driven Adami */
/* The Adami extrapolation of k_adami, summed over a boundary particle's
 * list of material neighbours (built with a skin; pairs at q >= 2 add
 * exact zeros, as the cell walk skips them), reading the neighbours from
 * the packed arrays (sigma_j V_j W = s_j rho_j m W with s = sigma / rho^2),
 * and writing the boundary particle's new stress into both state buffers
 * and, scaled, into both stages' packed arrays, which then need no pack of
 * the boundary slots before the pair kernel.  Targets without neighbours
 * keep all of them as they were.
 *
 * The targets are the slots act[0 .. *nact) whose lists can hold entries
 * (launch_boundary_targets): most boundary particles of a wall have no
 * material neighbour.  Their number, which only the device knows, decides
 * how many lanes share a target.  A list of about 20 entries is a chain of
 * dependent gathers: with few targets that is the time (16 us a launch with
 * one lane each, whatever their number), and lanes that share it divide it.
 * With many, the lanes' idle turns and the fewer targets per warp that share
 * a sector cost more than the chain.  So eight lanes while they come to no
 * more than kAdamiLanes, or four to twice that, else one: 9.3 us at the 5 k
 * column (11.3 with 4, 16 with 1), 18.2 with 4 at the 1.97 M cylinder's 70 k
 * targets (21.0 with 8, 23.7 with 1), 44 with 1 at the 2.85 M slope (64 with
 * 2, 88 with 8).  Between 65 k and 131 k targets either of one and four lanes
 * is up to 5 us the better one, with the lists' lengths.  The launch has a lane for every boundary particle, and
 * eight up to kAdamiLanes; blocks beyond the targets end at once (a grid of
 * 12 blocks per SM that strides: 52 us at the slope).
 *
 * Lane g takes entries g, g + G, ..., U at a time: the next turn's entries
 * are fetched ahead and a turn's gathers issued together; a pair at q >= 2
 * and the filler of the last turn, the target's own record, get the kernel
 * factor 0, so the loop has no branch.  From kAdamiPairTargets boundary
 * particles on U is two instead of four (fewer filler entries: 1.17 against
 * 1.28 ms a step at 16.2 M).  The bounds-checked build sets that threshold
 * to 0. */
#ifndef LQ_ADAMI_BLOCK
#define LQ_ADAMI_BLOCK 128
#endif
#ifndef LQ_ADAMI_PAIR_TARGETS
#define LQ_ADAMI_PAIR_TARGETS (4 << 20)
#endif
constexpr int kAdamiPairTargets = LQ_ADAMI_PAIR_TARGETS;
constexpr int kAdamiLanes = 1 << 18;

struct WallSums {
    const Parameters* P;
    State st;
    const int* list;
    const int* count;
    int stride;
    NbrArrays nb, nb2;
    tensor2d* str2;
    const int* act;
};

template <int G, int U>
__device__ __forceinline__ void adami_targets(const WallSums& w, int na)
{
    const int g = threadIdx.x % G;
    const unsigned mates = (unsigned)((1ull << G) - 1ull) << (threadIdx.x & 31 & ~(G - 1));
    const int step = gridDim.x * (LQ_ADAMI_BLOCK / G);
    const int np_all = __ldg(&w.P->np);
    const float ih = __ldg(&w.P->i_h), m = __ldg(&w.P->m), Cw = __ldg(&w.P->kernel_normalization_par);
    for (int a = (blockIdx.x * LQ_ADAMI_BLOCK + threadIdx.x) / G; a < na; a += step) {
        const int i = __ldg(w.act + a);
        const int n = min(__ldg(w.count + i), LQ_NBR_CAP);
        const float4 xi = __ldg(w.st.pos + i);
        tensor2d S = make_tensor2d(0.0f);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        auto entry = [&](int k) {
            const int j = k < n ? __ldg(w.list + (size_t)k * w.stride + i) : i;
            return lq_in_range(j, np_all) ? j : i;
        };
        int nxt[U];
#pragma unroll
        for (int u = 0; u < U; ++u) nxt[u] = entry(g + u * G);
        for (int k = g; k < n; k += U * G) {
            int j[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                j[u] = nxt[u];
                nxt[u] = entry(k + (U + u) * G);
            }
            float4 xr[U], sa[U];
            float2 sb[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                load_xs(w.nb, j[u], xr[u], sa[u]);
                sb[u] = __ldg(reinterpret_cast<const float2*>(w.nb.sb + j[u]));
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float dx = xi.x - xr[u].x, dy = xi.y - xr[u].y, dz = xi.z - xr[u].z;
                /* the approximate square root and quotient of the pair kernel */
                const float q = sqrt_approx(dx * dx + dy * dy + dz * dz) * ih;
                const float t = k + u * G < n ? fmaxf(2.0f - q, 0.0f) : 0.0f;
                const float ker = Cw * t * t * t * t * (q + 0.5f);
                const float kv = ker * __fdividef(m, xr[u].w);
                const float cs = m * xr[u].w * ker;
                S.xx += sa[u].x * cs;
                S.yy += sa[u].y * cs;
                S.zz += sa[u].z * cs;
                S.xy += sa[u].w * cs;
                S.xz += sb[u].x * cs;
                S.yz += sb[u].y * cs;
                acc.x += dx * kv;
                acc.y += dy * kv;
                acc.z += dz * kv;
                acc.w += kv;
            }
        }
        if (G > 1) {
            float* v[10] = {&S.xx, &S.yy, &S.zz, &S.xy, &S.xz, &S.yz, &acc.x, &acc.y, &acc.z, &acc.w};
#pragma unroll
            for (int k = 0; k < 10; ++k)
#pragma unroll
                for (int o = G / 2; o > 0; o >>= 1) *v[k] += __shfl_xor_sync(mates, *v[k], o, G);
        }
        if (g == 0 && acc.w > 0.0f) store_wall_stress(w.P, w.st, i, S, acc, w.str2, w.nb, w.nb2);
    }
}

__global__ void __launch_bounds__(LQ_ADAMI_BLOCK) k_adami_packed(WallSums w, const int* __restrict__ nact, bool pairs)
{
    const int na = __ldg(nact);
    if (pairs)
        adami_targets<1, 2>(w, na);
    else if (na <= kAdamiLanes / 8)
        adami_targets<8, 2>(w, na);
    else if (na <= kAdamiLanes / 2)
        adami_targets<4, 2>(w, na);
    else
        adami_targets<1, 4>(w, na);
}

/* ------------------------------------------ list-driven Shepard filters */
/* The walk of the native driver's two filters over a material target's
 * list, from the packed records (written from the state the filter reads:
 * the corrector packs every material slot, and each filter packs again
 * after changing the state): branch-free groups of four, the next group's
 * entries fetched ahead.  add(W, xr, sa, sb) gets the kernel value of each
 * entry, 0 for boundary neighbours (the filters use the material layer
 * only), for pairs at q >= 2 and for the filler of the last group (the
 * target's own slot); the list holds the target itself at q = 0.  kStress
 * also gathers the sigma / rho^2 words. */
template <bool kStress, class F>
__device__ __forceinline__ void filter_groups(const NbrArrays& nb, const int* p, int n, int stride, int i, int npb,
                                              int np, const float4& xi, float ih, float Cw, F&& add)
{
    int nxt[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) nxt[u] = u < n ? ld_list(p + (size_t)u * stride) : i;
    for (int k = 0; k < n; k += 4) {
        int j[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            j[u] = lq_in_range(nxt[u], np) ? nxt[u] : i;
            nxt[u] = k + 4 + u < n ? ld_list(p + (size_t)(k + 4 + u) * stride) : i;
        }
        float4 xr[4], sa[4];
        float2 sb[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (kStress) {
                load_xs(nb, j[u], xr[u], sa[u]);
                sb[u] = __ldg(reinterpret_cast<const float2*>(nb.sb + j[u]));
            } else {
                xr[u] = __ldg(nb.xs + 2 * (size_t)j[u]);
                sa[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                sb[u] = make_float2(0.f, 0.f);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float dx = xi.x - xr[u].x, dy = xi.y - xr[u].y, dz = xi.z - xr[u].z;
            const float q = sqrt_approx(dx * dx + dy * dy + dz * dz) * ih;
            const float t = (k + u < n && j[u] >= npb) ? fmaxf(2.0f - q, 0.0f) : 0.0f;
            add(Cw * t * t * t * t * (q + 0.5f), xr[u], sa[u], sb[u]);
        }
    }
}

/* The Shepard stress filter of k_shepard over a material particle's list:
 * sum sigma_j V_j W / sum V_j W over the material neighbours, with
 * sigma_j V_j W = s_j rho_j m W from the packed records (s = sigma /
 * rho^2, as Adami reads them).  Targets in the pair kernel's tile order
 * when `order` is set.  A particle whose list overflowed walks its 27
 * cells over the state instead.  Writes the filtered stress of material
 * slots to out_str. */
__global__ void __launch_bounds__(kBlock) k_shepard_list(const Parameters* __restrict__ P, int np, int npb, State st,
                                                         tensor2d* __restrict__ out_str,
                                                         const int* __restrict__ list,
                                                         const int* __restrict__ count, int stride, Cells cells,
                                                         Frames fr, NbrArrays nb, const int* __restrict__ order)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= np - npb) return;
    const int t = order ? __ldg(order + g) : g;
    if (!lq_in_range(t, np - npb)) return;
    const int i = npb + t;
    const int n = __ldg(count + t);
    const float ih = __ldg(&P->i_h), m = __ldg(&P->m), Cw = __ldg(&P->kernel_normalization_par);
    const float4 xi = __ldg(st.pos + i);
    tensor2d S = make_tensor2d(0.0f);
    float w = 0.0f;
    if (n <= LQ_NBR_CAP) {
        filter_groups<true>(nb, list + t, n, stride, i, npb, np, xi, ih, Cw,
                            [&](float ker, const float4& xr, const float4& sa, const float2& sb) {
                                const float cs = m * xr.w * ker;
                                S.xx += sa.x * cs;
                                S.yy += sa.y * cs;
                                S.zz += sa.z * cs;
                                S.xy += sa.w * cs;
                                S.xz += sb.x * cs;
                                S.yz += sb.y * cs;
                                w += ker * __fdividef(m, xr.w);
                            });
    } else {
        /* overflowed list (counted in the health word): the particle itself
         * and its 27-cell walk in the grid the lists were built from, as
         * the pair kernel does */
        auto add = [&](int j) {
            if (j < npb || !lq_in_range(j, np)) return;
            const float4 xj = __ldg(st.pos + j);
            const float3 d = make_float3(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z);
            const float q = norm3df(d.x, d.y, d.z) * ih;
            if (q < 2.0f) {
                const float ker = Cw * (2.0f - q) * (2.0f - q) * (2.0f - q) * (2.0f - q) * (q + 0.5f);
                const float vol = m / __ldg(&st.vel[j].w);
                const tensor2d sj = load_t2(st.str, j);
                S.xx += sj.xx * ker * vol;
                S.yy += sj.yy * ker * vol;
                S.zz += sj.zz * ker * vol;
                S.xy += sj.xy * ker * vol;
                S.xz += sj.xz * ker * vol;
                S.yz += sj.yz * ker * vol;
                w += ker * vol;
            }
        };
        add(i);
        walk_stencil(P, load_pair_const(P), st, cells, i, xi, add, fr);
    }
    const float inv = 1.0f / w;
    S.xx *= inv;
    S.yy *= inv;
    S.zz *= inv;
    S.xy *= inv;
    S.xz *= inv;
    S.yz *= inv;
    store_t2(out_str, i, S);
}

/* Density Shepard filter over a material particle's list (boundary
 * neighbours skipped; the list holds the particle itself, at q = 0):
 * rho~_i = sum m W / sum (m / rho_j) W, from the packed records' positions
 * and densities; targets in tile order when `order` is set. */
__global__ void __launch_bounds__(kBlock) k_density_filter_list(const Parameters* __restrict__ P, int np, int npb,
                                                                State st, float* __restrict__ rho_out,
                                                                const int* __restrict__ list,
                                                                const int* __restrict__ count, int stride,
                                                                Cells cells, Frames fr, NbrArrays nb,
                                                                const int* __restrict__ order)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= np - npb) return;
    const int t = order ? __ldg(order + g) : g;
    if (!lq_in_range(t, np - npb)) return;
    const int i = npb + t;
    const int n = __ldg(count + t);
    const float ih = __ldg(&P->i_h), m = __ldg(&P->m), Cw = __ldg(&P->kernel_normalization_par);
    const float4 xi = __ldg(st.pos + i);
    float num = 0.0f, den = 0.0f;
    if (n <= LQ_NBR_CAP) {
        filter_groups<false>(nb, list + t, n, stride, i, npb, np, xi, ih, Cw,
                             [&](float ker, const float4& xr, const float4&, const float2&) {
                                 num += m * ker;
                                 den += ker * __fdividef(m, xr.w);
                             });
    } else {
        /* overflowed list: the particle itself and its 27-cell walk */
        auto add = [&](int j) {
            if (j < npb || !lq_in_range(j, np)) return;
            const float4 xj = __ldg(st.pos + j);
            const float3 d = make_float3(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z);
            const float q = norm3df(d.x, d.y, d.z) * ih;
            if (q < 2.0f) {
                const float ker = Cw * (2.0f - q) * (2.0f - q) * (2.0f - q) * (2.0f - q) * (q + 0.5f);
                num += m * ker;
                den += ker * (m / __ldg(&st.vel[j].w));
            }
        };
        add(i);
        walk_stencil(P, load_pair_const(P), st, cells, i, xi, add, fr);
    }
    rho_out[i] = num / den;
}

}  // namespace

int launch_density_filter_list(const Parameters* ph, const Parameters* pd, const State& st, float* rho_out,
                               const NeighborList& nl, const Cells& c, cudaStream_t s, const Frames& fr,
                               float* rec, const int* order)
{
    if (ph->npm <= 0) return LQ_OK;
    if (!rec) return set_error(LQ_ERR_ARG, "density filter: the packed neighbour records are required");
    k_density_filter_list<<<blocks_for(ph->npm, kBlock), kBlock, 0, s>>>(pd, ph->np, ph->npb, st, rho_out, nl.list,
                                                                        nl.count, nl.stride, c, fr,
                                                                        nbr_arrays(rec, ph->np), order);
    LQ_TRY_CUDA(cudaGetLastError(), "k_density_filter_list");
    return LQ_OK;
}

/* Launch shapes of the pair kernel: threads per block x resident blocks
 * per SM (the register cap); a negative second entry -G marks the
 * warp-cooperative form with G lanes per target.  Shape 0 is the default. */
const int kPairShapes[kPairShapeCount][3] = {{kBlock, LQ_PAIR_MIN_BLOCKS, 0},
                                             {64, 12, 0},
                                             {256, 3, 0},
                                             {128, 5, 0},
                                             {128, 7, 0},
                                             {128, -8, 0},
                                             {128, -32, 0},
                                             {768, 1, 1},
                                             {384, 2, 1},
                                             {256, 3, 1},
                                             {320, 2, 1}};

/* The native driver's launch shape before any tuning: the tiled 256 x 3
 * shape from 2560 targets per SM on, the 128-thread shape 0 below that (a
 * small case leaves SMs idle at the end of a tiled launch: 230 k targets,
 * plain form, 92 us with shape 0 and 99 with 256 x 3 tiled). */
int default_pair_shape(int npm)
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) !=
                                                  cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return (long long)npm >= 2560LL * sms ? kDefaultTiledShape : 0;
}

/* Tile height (cells) for a block of `threads` targets: a 3 x 3-column
 * tile of that height holds about one block at (2 h / dr)^3 particles per
 * cell. */
static int tile_height(const Parameters* ph, int threads)
{
    const double ppc = std::pow(2.0 * (double)ph->hdr, 3.0);
    const int tz = (int)std::lround((double)threads / (9.0 * (ppc > 1.0 ? ppc : 1.0)));
    return tz < 1 ? 1 : tz;
}

static TileGrid tile_grid_of(const Parameters* ph, int tz)
{
    return tile_grid(ph->cell_num_x, ph->cell_num_y, ph->cell_num_z, ph->ncell_one_layer, tz);
}

int tile_order_scratch(const Parameters* ph, int* nseg, size_t* scan_bytes)
{
    *nseg = tile_grid_of(ph, 1).nseg;   /* the most segments any tile height needs */
    *scan_bytes = 0;
    LQ_TRY_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, *scan_bytes, (const int*)nullptr, (int*)nullptr, *nseg),
                "tile scan scratch query");
    return LQ_OK;
}


int launch_tile_order(const Parameters* ph, const int* start, int shape, const TileOrder& to, cudaStream_t s)
{
    if (shape < 0 || shape >= kPairShapeCount || kPairShapes[shape][2] != 1 || ph->npm <= 0) return LQ_OK;
    if (!to.order || !to.seg) return set_error(LQ_ERR_ARG, "tile order: buffers not allocated");
    const TileGrid tg = tile_grid_of(ph, tile_height(ph, kPairShapes[shape][0]));
    const int nseg = tg.nseg;
    if (nseg > to.nseg_cap) return set_error(LQ_ERR_ARG, "tile order: %d segments > capacity %d", nseg, to.nseg_cap);
    int* beg = to.seg;
    int* len = to.seg + to.nseg_cap;
    int* off = to.seg + 2 * (size_t)to.nseg_cap;
    k_tile_segments<<<blocks_for(nseg, kBlock), kBlock, 0, s>>>(start, tg, ph->npb, ph->np, beg, len);
    LQ_TRY_CUDA(cudaGetLastError(), "k_tile_segments");
    size_t bytes = to.scan_bytes;
    LQ_TRY_CUDA(cub::DeviceScan::ExclusiveSum(to.scan_tmp, bytes, len, off, nseg, s), "tile scan");
    k_tile_fill<<<blocks_for(nseg, kBlock / 32), kBlock, 0, s>>>(nseg, ph->npb, ph->npm, beg, len, off, to.order);
    LQ_TRY_CUDA(cudaGetLastError(), "k_tile_fill");
    return LQ_OK;
}

/* This translation unit's count of bounds violations (always 0 without
 * LQ_CHECKED). */
int bounds_count_sph(unsigned long long* v)
{
#ifdef LQ_CHECKED
    LQ_TRY_CUDA(cudaMemcpyFromSymbol(v, lq_bounds_count, sizeof(*v)), "bounds counter");
#else
    *v = 0;
#endif
    return LQ_OK;
}


int launch_list_refresh(const Parameters* ph, int first, int n, float cut, const float4* pos,
                        const int* inner_count, const NeighborList& shell, const NeighborList& nl, int* health,
                        cudaStream_t s)
{
    if (n <= 0) return LQ_OK;
    if (nl.stride < n || shell.stride != nl.stride)
        return set_error(LQ_ERR_ARG, "list renewal: strides %d / %d, targets %d", nl.stride, shell.stride, n);
    k_list_refresh<<<blocks_for(n, kBlock), kBlock, 0, s>>>(first, n, ph->np, cut * cut, pos, inner_count, shell.list,
                                                           shell.count, nl.list, nl.count, nl.stride, health);
    LQ_TRY_CUDA(cudaGetLastError(), "k_list_refresh");
    return LQ_OK;
}

int launch_neighbor_list_range(const Parameters* ph, const Parameters* pd, int first, int n, int layer_lo, float cut,
                               const float4* pos, const Cells& c, const NeighborList& nl, int* health,
                               cudaStream_t s, const float4* idep, const Frames& fr, const NeighborList* shell,
                               float inner, const int* gate)
{
    if (fr.rows && !idep) return set_error(LQ_ERR_ARG, "neighbour list: frames need the idep array");
    if (n <= 0) return LQ_OK;
    if (nl.stride < n) return set_error(LQ_ERR_ARG, "neighbour list stride %d < targets %d", nl.stride, n);
    if (shell && shell->stride != nl.stride)
        return set_error(LQ_ERR_ARG, "neighbour list: shell stride %d differs from %d", shell->stride, nl.stride);
    const float inner2 = inner > 0.0f ? inner * inner : 0.0f;
    if (shell)
        k_neighbor_list<true><<<blocks_for(n, kBlock), kBlock, 0, s>>>(pd, first, n, layer_lo, cut * cut, pos, c,
                                                                      nl.list, nl.count, nl.stride, health, idep, fr,
                                                                      shell->list, shell->count, inner2, gate);
    else
        k_neighbor_list<false><<<blocks_for(n, kBlock), kBlock, 0, s>>>(pd, first, n, layer_lo, cut * cut, pos, c,
                                                                       nl.list, nl.count, nl.stride, health, idep,
                                                                       fr, nullptr, nullptr, 0.0f, gate);
    LQ_TRY_CUDA(cudaGetLastError(), "k_neighbor_list");
    return LQ_OK;
}

int launch_list_arrange(int n, const NeighborList& nl, cudaStream_t s)
{
    if (n <= 0) return LQ_OK;
    if (nl.stride < n) return set_error(LQ_ERR_ARG, "list order: stride %d < targets %d", nl.stride, n);
    k_list_arrange<<<blocks_for(n, kArrangeBlock), kArrangeBlock, 0, s>>>(n, nl.count, nl.list, nl.stride);
    LQ_TRY_CUDA(cudaGetLastError(), "k_list_arrange");
    return LQ_OK;
}

int launch_pack_neighbors(const Parameters* ph, const State& st, float* rec, int first, cudaStream_t s,
                          bool packed_velocity, float* rec2, int n2)
{
    const int n = ph->np - first;
    if (n <= 0) return LQ_OK;
    const NbrArrays nb = nbr_arrays(rec, ph->np);
    const NbrArrays nb2 = rec2 ? nbr_arrays(rec2, ph->np) : NbrArrays{nullptr, nullptr, nullptr};
    if (packed_velocity)
        k_pack_neighbors<true><<<blocks_for(n, kBlock), kBlock, 0, s>>>(first, ph->np, st, nb, nb2, n2);
    else
        k_pack_neighbors<false><<<blocks_for(n, kBlock), kBlock, 0, s>>>(first, ph->np, st, nb, nb2, n2);
    LQ_TRY_CUDA(cudaGetLastError(), "k_pack_neighbors");
    return LQ_OK;
}

int launch_adami_packed(const Parameters* ph, const Parameters* pd, const State& st, const NeighborList& nl,
                        float* rec, cudaStream_t s, tensor2d* str2, float* rec2, const int* act, const int* nact)
{
    if (ph->npb <= 0) return LQ_OK;
    if (!act || !nact || !str2 || !rec2)
        return set_error(LQ_ERR_ARG, "Adami: the compacted targets and both stages' buffers are required");
    if (nl.stride < ph->npb) return set_error(LQ_ERR_ARG, "Adami: list stride %d < %d targets", nl.stride, ph->npb);
    const bool pairs = ph->npb >= kAdamiPairTargets;
    const long long eight = ph->npb * 8ll, few = eight < kAdamiLanes ? eight : kAdamiLanes;
    const long long lanes = ph->npb > few ? ph->npb : few;
    const int grid = blocks_for(lanes, LQ_ADAMI_BLOCK);
    const WallSums w{pd, st, nl.list, nl.count, nl.stride, nbr_arrays(rec, ph->np), nbr_arrays(rec2, ph->np), str2, act};
    k_adami_packed<<<grid, LQ_ADAMI_BLOCK, 0, s>>>(w, nact, pairs);
    LQ_TRY_CUDA(cudaGetLastError(), "k_adami_packed");
    return LQ_OK;
}

namespace {
/* A boundary list row that holds, or can gain by renewal, an entry. */
struct HasEntries {
    const int* a;
    const int* b;
    __device__ bool operator()(int i) const { return __ldg(a + i) > 0 || (b && __ldg(b + i) > 0); }
};
}   // namespace

size_t boundary_targets_temp_bytes(int npb)
{
    size_t bytes = 0;
    if (npb <= 0) return 0;
    cub::DeviceSelect::If(nullptr, bytes, thrust::counting_iterator<int>(0), (int*)nullptr, (int*)nullptr, npb,
                          HasEntries{nullptr, nullptr});
    return bytes;
}

int launch_boundary_targets(int npb, const int* count, const int* count2, int* act, int* nact, void* temp,
                            size_t temp_bytes, cudaStream_t s)
{
    if (npb <= 0) return LQ_OK;
    if (!count || !act || !nact || !temp)
        return set_error(LQ_ERR_ARG, "boundary targets: missing count, output or scratch");
    size_t bytes = temp_bytes;
    LQ_TRY_CUDA(cub::DeviceSelect::If(temp, bytes, thrust::counting_iterator<int>(0), act, nact, npb,
                                      HasEntries{count, count2}, s),
                "boundary targets (select)");
    return LQ_OK;
}

int launch_shepard_list(const Parameters* ph, const Parameters* pd, const State& st, tensor2d* out_str,
                        const NeighborList& nl, const Cells& c, cudaStream_t s, const Frames& fr, float* rec,
                        const int* order)
{
    if (ph->npm <= 0) return LQ_OK;
    if (!rec) return set_error(LQ_ERR_ARG, "Shepard filter: the packed neighbour records are required");
    k_shepard_list<<<blocks_for(ph->npm, kBlock), kBlock, 0, s>>>(pd, ph->np, ph->npb, st, out_str, nl.list,
                                                                 nl.count, nl.stride, c, fr, nbr_arrays(rec, ph->np),
                                                                 order);
    LQ_TRY_CUDA(cudaGetLastError(), "k_shepard_list");
    return LQ_OK;
}

namespace {

/* Shape 0 gives each target a team of lanes up to this many (us a step with
 * teams and without, plain; mixed): 8000 targets 43.7 and 57.4; 53.2 and 57.5,
 * 9600 53.5 and 57.2; 57.5 and 57.5, 12000 55.6 and 58.0; 67.7 and 59.5. */
#ifndef LQ_TEAM_TARGETS
#define LQ_TEAM_TARGETS 8192
#endif
constexpr int kTeamTargets = LQ_TEAM_TARGETS;

/* The pair kernel of a thread-per-target shape at stage kStage. */
template <bool kKahan, int kStage>
int launch_pair_stage(const Parameters* ph, const Parameters* pd, const State& st, const Rates& r, const Cells& c,
                      const NeighborList& nl, cudaStream_t s, const Frames& fr, const NbrArrays& nb, int shape,
                      const int* order, const int* rows, const StageTail& tail)
{
    if constexpr (kStage != 0)
        if (shape == 0 && ph->npm <= kTeamTargets) {
            k_interaction_team<kKahan, kStage><<<blocks_for(ph->npm, kTeamBlock / kTeam), kTeamBlock, 0, s>>>(
                pd, ph->np, ph->npb, st, r, c, nl.list, nl.count, nl.stride, fr, nb, tail);
            LQ_TRY_CUDA(cudaGetLastError(), "k_interaction_team");
            return LQ_OK;
        }
    const int threads = kPairShapes[shape][0], grid = blocks_for(ph->npm, threads);
#define LQ_PAIR_LAUNCH(T, B)                                                                                          \
    k_interaction_rec<kKahan, T, B, kStage><<<grid, threads, 0, s>>>(pd, ph->np, ph->npb, st, r, c, nl.list, nl.count, \
                                                                     nl.stride, fr, nb, order, rows, tail)
    /* one kernel per register cap, launched with each shape's block */
    if constexpr (kStage == 0) {
        LQ_PAIR_LAUNCH(768, 1);             /* 80 registers */
    } else {
        if (threads * kPairShapes[shape][1] == 768)
            LQ_PAIR_LAUNCH(768, 1);         /* 80 */
        else if (threads * kPairShapes[shape][1] == 640)
            LQ_PAIR_LAUNCH(320, 2);         /* 96 */
        else
            LQ_PAIR_LAUNCH(128, 7);         /* 72 */
    }
#undef LQ_PAIR_LAUNCH
    LQ_TRY_CUDA(cudaGetLastError(), "k_interaction_rec");
    return LQ_OK;
}

}  // namespace

bool integrates_in_pair_kernel(int shape) { return shape != 5 && shape != 6; }

int launch_interaction_list(const Parameters* ph, const Parameters* pd, const State& st, const Rates& r,
                            const Cells& c, const NeighborList& nl, cudaStream_t s, const Frames& fr,
                            bool compensated, float* rec, int shape, bool pack, const int* order,
                            const int* rows, const StageOps* ops)
{
    if (ph->npm <= 0) return LQ_OK;
    if (!rec) return set_error(LQ_ERR_ARG, "interaction: the packed neighbour arrays are required");
    if (reinterpret_cast<uintptr_t>(rec) % 32 != 0)
        return set_error(LQ_ERR_ARG, "interaction: packed neighbour arrays must be 32-byte aligned");
    if (shape < 0 || shape >= kPairShapeCount) return set_error(LQ_ERR_ARG, "interaction: launch shape %d", shape);
    const NbrArrays nb = nbr_arrays(rec, ph->np);
    if (rows && (pack || ops || shape == 5 || shape == 6))
        return set_error(LQ_ERR_ARG, "interaction: list rows need records packed in their order and a "
                         "thread-per-target shape that stores its rates");
    if (pack) LQ_TRY(launch_pack_neighbors(ph, st, rec, 0, s, compensated));
    if (kPairShapes[shape][2] == 1 && !order)
        return set_error(LQ_ERR_ARG, "interaction: launch shape %d needs the tile order", shape);
    if (kPairShapes[shape][2] != 1) order = nullptr;
    if (shape == 5 || shape == 6) {
        if (ops) return set_error(LQ_ERR_ARG, "interaction: launch shape %d stores its rates", shape);
        const int G = shape == 5 ? 8 : 32;
        const int grid = blocks_for((long long)ph->npm * G, 128);
#define LQ_GROUP_LAUNCH(K, G)                                                                                   \
    k_interaction_group<K, G><<<grid, 128, 0, s>>>(pd, ph->np, ph->npb, st, r, c, nl.list, nl.count, nl.stride, fr, nb)
        if (G == 8) {
            if (compensated) LQ_GROUP_LAUNCH(true, 8);
            else LQ_GROUP_LAUNCH(false, 8);
        } else {
            if (compensated) LQ_GROUP_LAUNCH(true, 32);
            else LQ_GROUP_LAUNCH(false, 32);
        }
#undef LQ_GROUP_LAUNCH
        LQ_TRY_CUDA(cudaGetLastError(), "k_interaction_group");
        return LQ_OK;
    }
    if (!ops) {
        if (compensated)
            return set_error(LQ_ERR_ARG, "interaction: the compensated form integrates in the pair kernel");
        return launch_pair_stage<false, 0>(ph, pd, st, r, c, nl, s, fr, nb, shape, order, rows, StageTail());
    }
    const StageTail tail{ops->in,     ops->out,   ops->mt, nbr_arrays(ops->rec_out, ph->np), ops->health,
                         verlet_of(ph, ops->lists), ops->keep_rates || ph->constitutive_model == 3};
    if (compensated)
        return ops->stage == 1 ? launch_pair_stage<true, 1>(ph, pd, st, r, c, nl, s, fr, nb, shape, order, rows, tail)
                               : launch_pair_stage<true, 2>(ph, pd, st, r, c, nl, s, fr, nb, shape, order, rows, tail);
    return ops->stage == 1 ? launch_pair_stage<false, 1>(ph, pd, st, r, c, nl, s, fr, nb, shape, order, rows, tail)
                           : launch_pair_stage<false, 2>(ph, pd, st, r, c, nl, s, fr, nb, shape, order, rows, tail);
}

int launch_adami(const Parameters* ph, const Parameters* pd, const State& st, const Cells& c, cudaStream_t s)
{
    if (ph->npb <= 0) return LQ_OK;
    k_adami<<<blocks_for((long long)ph->npb * kCellLanes, kBlock), kBlock, 0, s>>>(pd, ph->npb, st, c);
    LQ_TRY_CUDA(cudaGetLastError(), "k_adami");
    return LQ_OK;
}

int launch_shepard(const Parameters* ph, const Parameters* pd, const State& st, tensor2d* out_str, const Cells& c,
                   cudaStream_t s)
{
    if (ph->npm <= 0) return LQ_OK;
    k_shepard<<<blocks_for((long long)ph->npm * kCellLanes, kBlock), kBlock, 0, s>>>(pd, ph->np, ph->npb, st, out_str,
                                                                                    c);
    LQ_TRY_CUDA(cudaGetLastError(), "k_shepard");
    return LQ_OK;
}

}  // namespace lqb

/* ------------------------------------------------------------------ C ABI */

namespace {

bool bad_par(const void* ph, const void* pd) { return ph == nullptr || pd == nullptr; }

lqb::State state_of(const float* pos, const float* vel, const float* idep, const float* str, const float* stn)
{
    return lqb::State{(float4*)pos, (float4*)vel, (float4*)idep, (tensor2d*)str, (tensor2d*)stn};
}

}  // namespace

namespace {

/* Launch shape of the drop-in interaction's pair kernel (lqb::kPairShapes):
 * slot order, since each search moves the slots and the tile order would be
 * made anew for every call: the launch takes 308 us at 786 k targets either
 * way, and the tile order took 50. */
constexpr int kDropInShape = 0;
/* Skin of the drop-in interaction's lists (of h) when the caller's grid
 * tracks particle identities: the lists then hold every pair within
 * 2h + skin and are carried across calls until some particle has moved
 * half the skin. */
constexpr float kDropInSkinOverH = 0.05f;

/* Working arrays of the drop-in interaction, one set per device: the
 * neighbour lists, the packed neighbour data and what carries both from
 * call to call.  lq_interaction_reserve sizes them from a
 * Parameters record (the drop-in LoquatGrid's GridConfig calls it, where
 * the reference allocates its arrays); a call that needs more than was
 * reserved grows them itself, synchronising the device before the old
 * arrays are freed.  Calls that overlap on the GPU share the arrays and
 * must not. */
struct DropInWorkspace {
    int np = 0, npm = 0;
    lqb::NeighborList nl;           /* material targets' lists */
    float* rec = nullptr;           /* packed neighbour data, 13 floats per particle */
    /* lists carried across calls (caller grids that track identities) */
    float4* xbuild = nullptr;       /* np: positions at the build, by identity */
    int* build_of = nullptr;        /* np: identity -> slot at the build */
    int* rows = nullptr;            /* npm: target -> its list's row (the target's slot at the build) */
    int* moved = nullptr;           /* device flag: a particle moved half the skin since the build */
    int* tally = nullptr;           /* device counts of [0] builds and [1] reuses of carried lists */
    const int* key = nullptr;       /* the grid (its cell_beg) the carried lists belong to */
    long long gen = -1;
    int np_built = 0, npb_built = 0;
    float h_built = 0.0f;           /* what the lists hold depends on the cut-off and on the cells walked */
    int cells_built[3] = {0, 0, 0};
    bool built = false;
    long long rebuilds = 0, reuses = 0;   /* counts of earlier workspaces (tally holds this one's) */
    std::vector<void*> allocs;
};
std::mutex g_ws_mutex;
std::vector<DropInWorkspace> g_ws;

void free_workspace(DropInWorkspace& w)
{
    for (void* p : w.allocs) cudaFree(p);
    w = DropInWorkspace{};
}

int ws_alloc(DropInWorkspace& w, void** p, size_t bytes)
{
    cudaError_t e = cudaMalloc(p, bytes > 0 ? bytes : 16);
    if (e != cudaSuccess)
        return lqb::set_error(LQ_ERR_ALLOC, "interaction workspace: cudaMalloc(%zu): %s", bytes, cudaGetErrorString(e));
    w.allocs.push_back(*p);
    return LQ_OK;
}

/* Sizes every array for the Parameters' particle counts. */
int size_workspace(DropInWorkspace& w, const Parameters* ph)
{
    const int np = ph->np > 1 ? ph->np : 1, npm = ph->npm > 1 ? ph->npm : 1;
    if (np <= w.np && npm <= w.npm && w.rec) return LQ_OK;
    if (!w.allocs.empty()) LQ_TRY_CUDA(cudaDeviceSynchronize(), "interaction workspace");
    long long rebuilds = w.rebuilds, reuses = w.reuses;
    if (w.tally) {
        int t[2] = {0, 0};
        LQ_TRY_CUDA(cudaMemcpy(t, w.tally, sizeof(t), cudaMemcpyDeviceToHost), "interaction workspace");
        rebuilds += t[0];
        reuses += t[1];
    }
    free_workspace(w);
    DropInWorkspace n;
    n.rebuilds = rebuilds;
    n.reuses = reuses;
    int st = LQ_OK;
    auto A = [&](void** p, size_t bytes) {
        if (st == LQ_OK) st = ws_alloc(n, p, bytes);
    };
    A((void**)&n.rec, sizeof(float) * 13 * (size_t)np);
    n.nl.stride = (npm + 31) / 32 * 32;
    A((void**)&n.nl.list, sizeof(int) * (size_t)LQ_NBR_CAP * n.nl.stride);
    A((void**)&n.nl.count, sizeof(int) * (size_t)n.nl.stride);
    A((void**)&n.xbuild, sizeof(float4) * (size_t)np);
    A((void**)&n.build_of, sizeof(int) * (size_t)np);
    A((void**)&n.rows, sizeof(int) * (size_t)npm);
    A((void**)&n.moved, sizeof(int));
    A((void**)&n.tally, 2 * sizeof(int));
    if (st == LQ_OK) {
        /* done before any stream's call can count */
        cudaError_t e = cudaMemset(n.tally, 0, 2 * sizeof(int));
        if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
        if (e != cudaSuccess) st = lqb::set_error(LQ_ERR_CUDA, "interaction workspace: %s", cudaGetErrorString(e));
    }
    if (st != LQ_OK) {
        free_workspace(n);
        return st;
    }
    n.np = np;
    n.npm = npm;
    w = std::move(n);
    return LQ_OK;
}

int dropin_workspace(const Parameters* ph, DropInWorkspace** out)
{
    int dev = 0;
    LQ_TRY_CUDA(cudaGetDevice(&dev), "interaction workspace");
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    if ((int)g_ws.size() <= dev) g_ws.resize((size_t)dev + 1);
    DropInWorkspace& w = g_ws[(size_t)dev];
    LQ_TRY(size_workspace(w, ph));
    *out = &w;
    return LQ_OK;
}

/* Carrying lists across calls.  The caller's grid gives each slot's
 * particle identity (lqb::identity_*).  A build keeps its lists as they are
 * (rows and entries are slots at the build) and records, by identity, each
 * particle's build slot and position.  Every call packs each particle's
 * neighbour record at its build slot, so the pair kernel gathers through
 * the stored entries as they are, each target reading the row of its build
 * slot; a later call whose particles have all moved less than half the
 * skin only maps slots to build slots (k_carry).  The records stay
 * in the cell order of the build. */
__global__ void __launch_bounds__(256) k_moved_half_skin(int np, const float4* __restrict__ pos,
                                                         const int* __restrict__ ident,
                                                         const float4* __restrict__ xbuild, float half_skin2,
                                                         int* __restrict__ moved)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= np) return;
    const int id = __ldg(ident + c);
    bool far = true;
    if ((unsigned)id < (unsigned)np) {
        const float4 x = __ldg(pos + c), b = __ldg(xbuild + id);
        const float dx = x.x - b.x, dy = x.y - b.y, dz = x.z - b.z;
        far = !(dx * dx + dy * dy + dz * dz < half_skin2);
    }
    if (far) *moved = 1;
}

/* What a call does per slot besides its lists: a build (*moved, or moved
 * null) is recorded, each particle's build slot and position by identity;
 * the particle's neighbour record is packed at its build slot, which in a
 * build is the slot itself (not for a particle that has none); and each
 * material target gets its list's row, that slot less npb (-1: no carried
 * list, the pair kernel walks its stencil).  One thread counts the decision. */
__global__ void __launch_bounds__(256) k_carry(int np, int npb, lqb::State st, const int* __restrict__ ident,
                                               const int* __restrict__ moved, float4* __restrict__ xbuild,
                                               int* __restrict__ build_of, lqb::NbrArrays nb, int* __restrict__ rows,
                                               int* __restrict__ tally)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= np) return;
    const bool build = !moved || *moved;
    if (c == 0) tally[build ? 0 : 1] += 1;
    const int id = __ldg(ident + c);
    const float4 x = __ldg(st.pos + c);
    int o = build ? c : -1;     /* a build's lists name its own slots, every one of them */
    if ((unsigned)id < (unsigned)np) {
        if (build) {
            xbuild[id] = x;
            build_of[id] = c;
        } else {
            o = build_of[id];
            if ((unsigned)o >= (unsigned)np) o = -1;
        }
    }
    if (c >= npb) rows[c - npb] = o >= npb ? o - npb : -1;
    if (o >= 0) lqb::pack_slot<false>(nb, o, x, __ldg(st.vel + c), lqb::load_t2(st.str, c));
}

}  // namespace

extern "C" int lq_interaction_stats(long long* rebuilds, long long* reuses)
{
    if (!rebuilds || !reuses) return lqb::set_error(LQ_ERR_ARG, "lq_interaction_stats: null argument");
    int dev = 0;
    LQ_TRY_CUDA(cudaGetDevice(&dev), "interaction stats");
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    *rebuilds = 0;
    *reuses = 0;
    if (dev < (int)g_ws.size()) {
        const DropInWorkspace& w = g_ws[(size_t)dev];
        int t[2] = {0, 0};
        if (w.tally) {
            /* the decisions are counted on the device by the calls' streams */
            LQ_TRY_CUDA(cudaDeviceSynchronize(), "interaction stats");
            LQ_TRY_CUDA(cudaMemcpy(t, w.tally, sizeof(t), cudaMemcpyDeviceToHost), "interaction stats");
        }
        *rebuilds = w.rebuilds + t[0];
        *reuses = w.reuses + t[1];
    }
    return LQ_OK;
}

extern "C" int lq_interaction_reserve(const void* par_host)
{
    if (!par_host) return lqb::set_error(LQ_ERR_ARG, "lq_interaction_reserve: null Parameters");
    const Parameters* ph = static_cast<const Parameters*>(par_host);
    if (ph->np < 0 || ph->npm < 0 || ph->ncell < 1)
        return lqb::set_error(LQ_ERR_ARG, "lq_interaction_reserve: bad sizes np=%d npm=%d ncell=%d", ph->np, ph->npm,
                              ph->ncell);
    DropInWorkspace* w = nullptr;
    return dropin_workspace(ph, &w);
}

/* The reference's ParticleInteraction (src/particle_interaction.h:27-40).
 * The caller's grid (cell_beg / cell_end: every particle sorted into its
 * cell, cells in key order) gives the material targets' neighbours within
 * 2h, found by the 27-cell walk into lists, and the pair kernel sums over
 * the lists from the packed neighbour data, in plain FP32 as the reference
 * computes. */
extern "C" int lq_particle_interaction(const void* par_host, const void* par_device, const float* pospres,
                                       const float* velrhop, const float* idep, const float* str, const float* stn,
                                       float* accad, float* spin, float* acestn, const int* cell_beg,
                                       const int* cell_end, void* stream)
{
    if (bad_par(par_host, par_device)) return lqb::set_error(LQ_ERR_ARG, "lq_particle_interaction: null Parameters");
    const Parameters* ph = static_cast<const Parameters*>(par_host);
    if (ph->npm > 0 && (!pospres || !velrhop || !str || !accad || !spin || !acestn || !cell_beg || !cell_end))
        return lqb::set_error(LQ_ERR_ARG, "lq_particle_interaction: null array");
    if (ph->npm <= 0) return LQ_OK;
    lqb::Rates r{(float4*)accad, (float4*)spin, (tensor2d*)acestn};
    const Parameters* pd = static_cast<const Parameters*>(par_device);
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    const lqb::State st = state_of(pospres, velrhop, idep, str, stn);
    DropInWorkspace* w = nullptr;
    LQ_TRY(dropin_workspace(ph, &w));
    const lqb::Cells c{nullptr, cell_beg, cell_end};
    const int np = ph->np, npb = ph->npb, npm = ph->npm;
    const int nb256 = (np + 255) / 256;
    lqb::GridIdentity gi;
    if (lqb::identity_find(cell_beg, &gi) && gi.np == np) {
        /* the caller's grid tracks its particles: carry the lists while
         * every particle stays within half the skin of its build position.
         * The device decides (no host synchronisation): the list build is
         * enqueued and returns at once when it is not taken. */
        const float skin = kDropInSkinOverH * ph->h;
        const bool carried = w->built && w->key == cell_beg && w->gen == gi.gen && w->np_built == np &&
                             w->npb_built == npb && w->h_built == ph->h && w->cells_built[0] == ph->cell_num_x &&
                             w->cells_built[1] == ph->cell_num_y && w->cells_built[2] == ph->cell_num_z;
        const int* moved = nullptr;
        if (carried) {
            LQ_TRY_CUDA(cudaMemsetAsync(w->moved, 0, sizeof(int), s), "moved flag");
            k_moved_half_skin<<<nb256, 256, 0, s>>>(np, st.pos, gi.ident, w->xbuild, 0.25f * skin * skin, w->moved);
            LQ_TRY_CUDA(cudaGetLastError(), "k_moved_half_skin");
            moved = w->moved;
        }
        /* a build: fresh lists in the current slots, kept with each
         * particle's build slot and position */
        LQ_TRY(lqb::launch_neighbor_list_range(ph, pd, npb, npm, 0, 2.0f * ph->h + skin, st.pos, c, w->nl, nullptr,
                                               s, nullptr, lqb::Frames(), nullptr, 0.0f, moved));
        /* either way the pair kernel reads the lists of the last build,
         * each target at the row of its build slot, with the records
         * packed at the build slots: a reuse maps only slots */
        k_carry<<<nb256, 256, 0, s>>>(np, npb, st, gi.ident, moved, w->xbuild, w->build_of,
                                      lqb::nbr_arrays(w->rec, np), w->rows, w->tally);
        LQ_TRY_CUDA(cudaGetLastError(), "k_carry");
        w->built = true;
        w->key = cell_beg;
        w->gen = gi.gen;
        w->np_built = np;
        w->npb_built = npb;
        w->h_built = ph->h;
        w->cells_built[0] = ph->cell_num_x;
        w->cells_built[1] = ph->cell_num_y;
        w->cells_built[2] = ph->cell_num_z;
        return lqb::launch_interaction_list(ph, pd, st, r, c, w->nl, s, lqb::Frames(), false, w->rec, kDropInShape,
                                            false, nullptr, w->rows);
    }
    /* a grid of the caller's own: lists built in its slots at every call,
     * with the pair body's own cut-off test (q < 2 with the candidate
     * slack of the cell walk) */
    const float cut = 2.0f * ph->h * sqrtf(1.0001f);
    LQ_TRY(lqb::launch_neighbor_list_range(ph, pd, npb, npm, 0, cut, st.pos, c, w->nl, nullptr, s));
    w->built = false;
    return lqb::launch_interaction_list(ph, pd, st, r, c, w->nl, s, lqb::Frames(), false, w->rec, kDropInShape, true);
}

extern "C" int lq_adami_boundary(const void* par_host, const void* par_device, const float* pospres,
                                 const float* velrhop, float* str, const int* cell_beg, const int* cell_end,
                                 void* stream)
{
    if (bad_par(par_host, par_device)) return lqb::set_error(LQ_ERR_ARG, "lq_adami_boundary: null Parameters");
    const Parameters* ph = static_cast<const Parameters*>(par_host);
    if (ph->npb > 0 && (!pospres || !velrhop || !str || !cell_beg || !cell_end))
        return lqb::set_error(LQ_ERR_ARG, "lq_adami_boundary: null array");
    lqb::Cells c{nullptr, cell_beg, cell_end};
    return lqb::launch_adami(ph, static_cast<const Parameters*>(par_device),
                             state_of(pospres, velrhop, nullptr, str, nullptr), c, static_cast<cudaStream_t>(stream));
}

extern "C" int lq_stress_regularization(const void* par_host, const void* par_device, const float* pospres,
                                        const float* velrhop, float* str, float* tensor2d_cache, const int* cell_beg,
                                        const int* cell_end, void* stream)
{
    if (bad_par(par_host, par_device))
        return lqb::set_error(LQ_ERR_ARG, "lq_stress_regularization: null Parameters");
    const Parameters* ph = static_cast<const Parameters*>(par_host);
    if (ph->npm <= 0) return LQ_OK;
    if (!pospres || !velrhop || !str || !tensor2d_cache || !cell_beg || !cell_end)
        return lqb::set_error(LQ_ERR_ARG, "lq_stress_regularization: null array");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    lqb::Cells c{nullptr, cell_beg, cell_end};
    LQ_TRY(lqb::launch_shepard(ph, static_cast<const Parameters*>(par_device),
                               state_of(pospres, velrhop, nullptr, str, nullptr), (tensor2d*)tensor2d_cache, c, s));
    /* copy the filtered material stress back (reference src/field_smoothing.cu:144) */
    LQ_TRY_CUDA(cudaMemcpyAsync((tensor2d*)str + ph->npb, (tensor2d*)tensor2d_cache + ph->npb,
                                sizeof(tensor2d) * (size_t)ph->npm, cudaMemcpyDeviceToDevice, s),
                "Shepard copy back");
    return LQ_OK;
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

void ParticleInteraction(Parameters* par_host, Parameters* par_device, float4* pospres, float4* velrhop,
                         float4* idep, tensor2d* str, tensor2d* stn, float4* accad, float4* spin, tensor2d* acestn,
                         const int* cell_beg, const int* cell_end)
{
    check_or_die(lq_particle_interaction(par_host, par_device, (const float*)pospres, (const float*)velrhop,
                                         (const float*)idep, (const float*)str, (const float*)stn, (float*)accad,
                                         (float*)spin, (float*)acestn, cell_beg, cell_end, nullptr),
                 "ParticleInteraction");
}

void AdamiBoundary(Parameters* par_host, Parameters* par_device, float4* pospres, float4* velrhop, tensor2d* str,
                   const int* cell_beg, const int* cell_end)
{
    check_or_die(lq_adami_boundary(par_host, par_device, (const float*)pospres, (const float*)velrhop, (float*)str,
                                   cell_beg, cell_end, nullptr),
                 "AdamiBoundary");
}

void StressRegularization(Parameters* par_host, Parameters* par_device, float4* pospres, float4* velrhop,
                          tensor2d* str, tensor2d* tensor2d_cache, const int* cell_beg, const int* cell_end)
{
    check_or_die(lq_stress_regularization(par_host, par_device, (const float*)pospres, (const float*)velrhop,
                                          (float*)str, (float*)tensor2d_cache, cell_beg, cell_end, nullptr),
                 "StressRegularization");
}

extern "C" int lq_debug_bounds_violations(long long* count)
{
    if (!count) return lqb::set_error(LQ_ERR_ARG, "lq_debug_bounds_violations: null argument");
#ifdef LQ_CHECKED
    LQ_TRY_CUDA(cudaDeviceSynchronize(), "bounds counter");
    unsigned long long a = 0, b = 0, c = 0;
    LQ_TRY(lqb::bounds_count_sph(&a));
    LQ_TRY(lqb::bounds_count_grid(&b));
    LQ_TRY(lqb::bounds_count_integrate(&c));
    *count = (long long)(a + b + c);
#else
    *count = -1;
#endif
    return LQ_OK;
}
