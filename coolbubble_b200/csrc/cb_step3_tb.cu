/* cb_step3_tb.cu -- two leapfrog steps per HBM pass on static 3-D lattices.
 *
 * Temporal blocking of the step of cb_step3.cu (reference Bubble::oneStep,
 * src/bubble.cpp:849-876, static background: a = 1, no step between two
 * reported ones needs a global sum). One launch reads phi_n, pi_{n-1/2} and
 * writes phi_{n+2}, pi_{n+3/2}: half the DRAM bytes per step.
 *
 *  - Float and double; rows of a warp or more, padded to whole 16-byte vectors.
 *    Tiles of TJ full rows of axis 1, TJ even (axis-2 neighbours wrap in shared
 *    memory; the last tile may hang over the lattice's end and repeat its first
 *    rows); work items (plane part, tile) taken from a device-wide queue,
 *    part-major with tiles fastest (the items in flight share their halo rows
 *    in L2), one block per SM.
 *  - Input planes arrive by TMA bulk copies into a 4- to 6-stage ring: phi
 *    rows [j0 - 2, j0 + TJ + 2), pi rows [j0 - 1, j0 + TJ + 1) (periodic).
 *  - Each consumer thread owns the same positions in every plane (two vectors of
 *    the tile, a share of the two halo rows) and marches them along axis 0:
 *    its own columns of input phi, of level-1 phi and of level-1 pi stay in
 *    registers, so shared memory holds only what other threads read -- the
 *    input planes and two level-1 planes (TJ + 2 rows each). That leaves room
 *    for 8-row tiles at 512^3 (level-1 rows 1.25x the output rows).
 *  - Round q (input plane q landed): per position, level 1 (the first step) at
 *    plane q - 1 and level 2 (the second step, to HBM) at plane q - 2; one
 *    consumer barrier per round orders the level-1 planes' writes and reuse.
 *    Axis-2 neighbours come from the adjacent lanes by shuffle.
 *  - An item computing planes [p0, p1) streams input planes p0 - 2 .. p1 + 1
 *    (overlapped tiling: neighbouring items recompute the halo, no block
 *    talks to another). The input ring runs on from one item to the next.
 *  - The per-site results are those of the single-step kernel (float: packed
 *    f32x2, the same rounded operations), so two blocked steps give the fields
 *    of two single steps bit for bit.
 *  - What bounds it: the latency of a round (load, two dependent updates, a
 *    barrier) over 16 warps, ncu on 256^3: float FMA pipe 48 % busy (a quarter of
 *    it register moves), issue 49 %; double FP64 pipe 36 %, issue 50 %; DRAM
 *    41-47 %. us per step, one step per pass -> here: 192^3 float 19.0 -> 14.7,
 *    250^3 48 -> 26.2, 256^3 50.0 -> 24.0, 512^3 336 -> 170; double 192^3 44.7 ->
 *    28.3, 256^3 89 -> 56. A barrier split into arriving and waiting half a round
 *    later, with two or three level-1 planes, cost more in registers than it hid
 *    (250^3 30.4 and 34.1, 512^3 184 and 212).
 *  - Waits are bounded (clock64 limit, sleeping retries); a timed-out block
 *    records an error word; consumer warps leave together (a vote in the
 *    per-round barrier).
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <type_traits>

#include "cb_internal.h"
#include "cb_launch.cuh"
#include "cb_march.cuh"
#include "cb_step_common.cuh"
#include "cb_tma.cuh"

namespace cb {

namespace {

constexpr int TB_MAXT = 512;             /* threads per block (all of them compute) */
constexpr int TB_NTS = 2;                 /* tile positions per thread */
constexpr int TB_HDR = 256;               /* full[nstage] mbarriers (nstage <= 8) */
constexpr int TB_IQ = 8;

/* One leapfrog step on the static background: pi' = pi + dt F(phi), phi' =
 * phi + dt pi' (bubble.cpp:716-743, 853-856, 867-870 with a = 1), for the
 * sites c of a row with its neighbour rows um / up along axis 1 and im / ip
 * along axis 0 and the sites left / right of it along axis 2 -- the results
 * of the single-step kernel bit for bit. */
template <typename T, int BY>
struct Step;

/* float: packed pairs (f32x2) */
template <int BY>
struct Step<float, BY> {
    F2 idx2, dt, nc2, c3, nc4, m2;
    __device__ __forceinline__ explicit Step(const StepConst &k)
        : idx2(f2_splat(k.inv_dx2f)), dt(f2_splat(k.dtf)), nc2(f2_splat(-k.c2f)), c3(f2_splat(k.c3f)),
          nc4(f2_splat(-k.c4f)), m2(f2_splat(-2.f)) {}
    /* the axis-2 term of site c between a and b: in scalars, since the neighbours
     * of a pair straddle the pairs they are held in (packing them took six moves
     * per vector) */
    static __device__ __forceinline__ float along(float a, float c, float b) {
        return __fadd_rn(__fmaf_rn(c, -2.f, b), a);
    }
    __device__ __forceinline__ void pair(F2 cc, F2 umm, F2 upp, F2 imm, F2 ipp, F2 t2, F2 pp, F2 &phi2,
                                         F2 &pi2) const {
        /* x - 2 c in one rounding: 2 c is exact */
        const F2 t0 = f2_add(f2_fma(cc, m2, ipp), imm);
        const F2 t1 = f2_add(f2_fma(cc, m2, upp), umm);
        const F2 lap = f2_add(f2_add(t0, t1), t2);
        /* -V'(f)/f = -(c2 + f (-c3 + f c4)) with every operand negated: the
         * exact negation of the one-step kernel's rounded h (round to nearest
         * is symmetric); with a^(d-2) = a^d = 1 the force fma(1 lap, 1/dx^2,
         * -1 (f h)) is then fma(lap, 1/dx^2, f (-h)), bit for bit */
        const F2 nh = f2_fma(cc, f2_fma(cc, nc4, c3), nc2);
        const F2 force = f2_fma(lap, idx2, f2_mul(cc, nh));
        pi2 = f2_fma(dt, force, pp);
        phi2 = f2_fma(dt, pi2, cc);
    }
    __device__ __forceinline__ void operator()(const float4 &c, const float4 &um, const float4 &up, const float4 &im,
                                               const float4 &ip, float left, float right, const float4 &pv,
                                               float4 &phi, float4 &pi) const {
        F2 phi01, pi01, phi23, pi23;
        pair(f2_pack(c.x, c.y), f2_pack(um.x, um.y), f2_pack(up.x, up.y), f2_pack(im.x, im.y), f2_pack(ip.x, ip.y),
             f2_pack(along(left, c.x, c.y), along(c.x, c.y, c.z)), f2_pack(pv.x, pv.y), phi01, pi01);
        pair(f2_pack(c.z, c.w), f2_pack(um.z, um.w), f2_pack(up.z, up.w), f2_pack(im.z, im.w), f2_pack(ip.z, ip.w),
             f2_pack(along(c.y, c.z, c.w), along(c.z, c.w, right)), f2_pack(pv.z, pv.w), phi23, pi23);
        phi = make_float4(f2_lo(phi01), f2_hi(phi01), f2_lo(phi23), f2_hi(phi23));
        pi = make_float4(f2_lo(pi01), f2_hi(pi01), f2_lo(pi23), f2_hi(pi23));
    }
    __device__ __forceinline__ void operator()(const float2 &c, const float2 &um, const float2 &up, const float2 &im,
                                               const float2 &ip, float left, float right, const float2 &pv,
                                               float2 &phi, float2 &pi) const {
        F2 p2, q2;
        pair(f2_pack(c.x, c.y), f2_pack(um.x, um.y), f2_pack(up.x, up.y), f2_pack(im.x, im.y), f2_pack(ip.x, ip.y),
             f2_pack(along(left, c.x, c.y), along(c.x, c.y, right)), f2_pack(pv.x, pv.y), p2, q2);
        phi = make_float2(f2_lo(p2), f2_hi(p2));
        pi = make_float2(f2_lo(q2), f2_hi(q2));
    }
    /* one site: the same operations in scalars */
    __device__ __forceinline__ void operator()(float c, float um, float up, float im, float ip, float left,
                                               float right, float pv, float &phi, float &pi) const {
        const float lap = __fadd_rn(__fadd_rn(along(im, c, ip), along(um, c, up)), along(left, c, right));
        const float nh = __fmaf_rn(c, __fmaf_rn(c, f2_lo(nc4), f2_lo(c3)), f2_lo(nc2));
        const float force = __fmaf_rn(lap, f2_lo(idx2), __fmul_rn(c, nh));
        pi = __fmaf_rn(f2_lo(dt), force, pv);
        phi = __fmaf_rn(f2_lo(dt), pi, c);
    }
};

/* double: the single-step kernel's rounded operations in its order, without
 * its products with a^(d-2) = a^d = 1 (exact) */
template <int BY>
struct Step<double, BY> {
    const StepConst &k;
    __device__ __forceinline__ explicit Step(const StepConst &kk) : k(kk) {}
    __device__ __forceinline__ void operator()(double c, double um, double up, double im, double ip, double left,
                                               double right, double pv, double &phi, double &pi) const {
        using A = Ar<double>;
        /* x - 2 c in one rounding: 2 c is exact */
        const double t0 = A::add(__fma_rn(c, -2.0, ip), im);
        const double t1 = A::add(__fma_rn(c, -2.0, up), um);
        const double t2 = A::add(__fma_rn(c, -2.0, right), left);
        const double lap = A::add(A::add(t0, t1), t2);
        pi = A::add(pv, A::mul(k.dt, A::sub(over_dx2<BY>(k, lap), dV<double>(k, c))));
        phi = A::add(c, A::mul(k.dt, pi));
    }
    __device__ __forceinline__ void operator()(const double2 &c, const double2 &um, const double2 &up,
                                               const double2 &im, const double2 &ip, double left, double right,
                                               const double2 &pv, double2 &phi, double2 &pi) const {
        (*this)(c.x, um.x, up.x, im.x, ip.x, left, c.y, pv.x, phi.x, pi.x);
        (*this)(c.y, um.y, up.y, im.y, ip.y, c.x, right, pv.y, phi.y, pi.y);
    }
};

/* A tile position of a thread (row r1 of the level-1 rows j0 - 1 .. j0 + tj,
 * vector kv of the row), updated at both levels in every plane of an item,
 * with its columns along axis 0 kept in registers:
 *   x_m, x_c  input phi at planes m - 1, m (level 1 at plane m reads phi at
 *             m + 1 from the stage that just landed);
 *   y_c, y_p  level-1 phi at planes m', m' + 1 (level 2 at m');
 *   z, zz     level-1 pi at planes m', m' + 1.
 * The halo rows (j0 - 1, j0 + tj) are updated at level 1 only; a thread's
 * share of them keeps only x_m, x_c. */
template <typename V>
struct Slot {
    V x_m, x_c, y_c, y_p, z, zz;
};

/* Two leapfrog steps per pass (see the file comment). Thread c owns the tile
 * positions c and c + half the tile's (the same site of the row half a tile
 * further, so one set of offsets and row ends serves both) and HW sites of
 * the halo rows (row j0 - 1, then row j0 + tj), sites HW c .. HW c + HW - 1:
 * HW = 2 n / NT (1 or 2) gives every thread the same share; HW = 4 gives
 * threads c < 2 n / 4 one vector each (where 2 n / NT is not 1 or 2). Rows hold a
 * multiple of 32 vectors, so a warp's 32 positions of a slot are 32
 * consecutive vectors of one row: the axis-2 neighbours come from the next
 * lanes by shuffle (the end lanes read them from shared memory), and the
 * branch on the halo slot is uniform across the warp.
 * NV: the vectors of a row where they are a power of two (32, 64, 128) and the
 * tile has 1024 of them: every shared offset of a round is then a constant
 * (512^3 float 193 -> 177 us per step, 256^3 27.4 -> 24.9, in double 60 -> 55;
 * with the axis-2 terms in scalars 170 and 24.0).
 * The streamed input planes are counted g = 0, 1, ... over all the block's
 * items (plane g in stage g mod nstage); round g waits for plane g. An item
 * computing planes [p0, p1) streams planes p0 - 2 .. p1 + 1: its first two
 * rounds load the register queues, then round q (input plane q) runs, per
 * position, level 1 at plane q - 1 and level 2 at plane q - 2. Every round
 * ends with one barrier of all threads; plane g's stage is free once round
 * g + 1 has ended, so at the start of round g thread 0 issues the copies of
 * planes up to g + nstage - 2 (no other wait). */
template <typename T, int BY, int HW, bool WHOLE, int NV = 0>
__global__ void __launch_bounds__(TB_MAXT, 1)
    k_step3_t2(StepConst k, int tj_, int nstage, int parts, const T *__restrict__ phi_in, const T *__restrict__ pi_in,
               T *__restrict__ phi_out, T *__restrict__ pi_out, DevState *st) {
    using V = typename Vec<T>::V;
    constexpr int W = Vec<T>::W;
    constexpr uint32_t ES = sizeof(T);
    /* level-1 phi at plane m' - 1 from registers only where offsets are constants:
     * elsewhere they are too few and keeping it costs more than reading it back (250^3 float 27.7 -> 26.3 us per step,
     * 192^3 15.6 -> 14.7; 512^3, NV, 170 -> 174) */
    constexpr bool KEEP_Y = NV != 0;
    extern __shared__ __align__(128) unsigned char smraw[];
    __shared__ int abort_flag;
    __shared__ int item_q[TB_IQ];

    static_assert(NV == 0 || WHOLE, "a constant row length is for whole-warp rows");
    const int n = NV ? NV * W : k.n, np = WHOLE ? n : k.pitch;   /* sites and elements of a row */
    const int tj = NV ? TB_NTS * TB_MAXT / NV : tj_;
    const int R0 = tj + 4;                 /* input phi rows: j0 - 2 .. j0 + tj + 1 */
    const int R0p = tj + 2;                /* input pi rows: j0 - 1 .. j0 + tj */
    const int R1 = tj + 2;                 /* level-1 phi rows: j0 - 1 .. j0 + tj */
    const int stage_n = (R0 + R0p) * np;    /* elements per input stage */
    const int slot_n = R1 * np;             /* elements per level-1 slot */
    uint64_t *full = reinterpret_cast<uint64_t *>(smraw);
    T *ring = reinterpret_cast<T *>(smraw + TB_HDR);
    T *l1 = ring + (size_t)nstage * stage_n;

    const int ntiles = (n + tj - 1) / tj;
    const int items = ntiles * parts;
    const size_t row_bytes = (size_t)np * sizeof(T);
    const size_t plane = (size_t)n * np;
    const uint32_t tx_bytes = (uint32_t)((size_t)(R0 + R0p) * row_bytes);
    const int lane = threadIdx.x & 31;
    const int NT = NV ? TB_MAXT : blockDim.x;
    auto item_of = [&](int it, int &t, int &p0, int &p1) {
        const int c = it / ntiles;
        t = it % ntiles;
        p0 = (int)((long long)c * n / parts);
        p1 = (int)((long long)(c + 1) * n / parts);
    };

    /* ---- the copies (thread 0): planes are issued in stream order; the
     *      producer's item j is published in item_q[j % TB_IQ] before its
     *      first plane is issued ---- */
    int pr_j = 0, pr_it = -1, pr_pl = 0, pr_p1 = 0;              /* producer: item, next plane */
    /* the item's source rows, as element offsets within a plane and counts of
     * rows: phi rows j0 - 2 .. j0 + tj + 1 and pi rows j0 - 1 .. j0 + tj, each from
     * its start up to the lattice's last row, then the rest from row 0 */
    __shared__ size_t pr_r[2];   /* thread 0's only: kept out of the registers */
    __shared__ int pr_c[2];
    int issued = 0;                                              /* planes issued so far */
    int is_stage = 0;                                            /* its stage: issued mod nstage */
    bool pr_done = false;
    auto next_item = [&]() {
        /* a block's first item is its own index (the grid never exceeds the
         * items); later ones come from the queue */
        const int cur = pr_j == 0 ? (int)blockIdx.x : (int)gridDim.x + (int)atomicAdd(&st->item_next, 1u);
        pr_it = cur < items ? cur : -1;
        item_q[pr_j % TB_IQ] = pr_it;
        ++pr_j;
        if (pr_it < 0) {
            pr_done = true;
            return;
        }
        int t, p0, p1;
        item_of(pr_it, t, p0, p1);
        pr_pl = p0 - 2;
        pr_p1 = p1;
        const int j0 = t * tj;
        const int r0 = (j0 - 2 + n) % n, r1 = (j0 - 1 + n) % n;
        pr_r[0] = (size_t)r0 * np;
        pr_r[1] = (size_t)r1 * np;
        pr_c[0] = min(R0, n - r0);
        pr_c[1] = min(R0p, n - r1);
    };
    auto issue_upto = [&](int last) {
        while (!pr_done && issued <= last) {
            const int s = is_stage;
            const int pw = pr_pl < 0 ? pr_pl + n : (pr_pl >= n ? pr_pl - n : pr_pl);
            T *dst = ring + (size_t)s * stage_n;
            T *dpi = dst + (size_t)R0 * np;
            const T *gphi = phi_in + (size_t)pw * plane;
            const T *gpi = pi_in + (size_t)pw * plane;
            const uint32_t rb = (uint32_t)row_bytes;
            fence_proxy_async();
            mbar_arrive_expect_tx(&full[s], tx_bytes);
            const int c0 = pr_c[0], c1 = pr_c[1];
            bulk_g2s(dst, gphi + pr_r[0], (uint32_t)c0 * rb, &full[s]);
            if (c0 < R0) bulk_g2s(dst + (size_t)c0 * np, gphi, (uint32_t)(R0 - c0) * rb, &full[s]);
            bulk_g2s(dpi, gpi + pr_r[1], (uint32_t)c1 * rb, &full[s]);
            if (c1 < R0p) bulk_g2s(dpi + (size_t)c1 * np, gpi, (uint32_t)(R0p - c1) * rb, &full[s]);
            ++issued;
            if (++is_stage == nstage) is_stage = 0;
            if (++pr_pl > pr_p1 + 1) next_item();
        }
    };

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < nstage; ++s) mbar_init(&full[s], 1);
        fence_mbar_init();
    }
    __syncthreads();
    pdl_wait();          /* the previous step's fields, device state and work queue */
    if (threadIdx.x == 0) {
        next_item();
        issue_upto(nstage - 2);
    }
    __syncthreads();

    const Step<T, BY> step(k);
    /* the positions as offsets r1 np + kk in an array of level-1 rows (row r1,
     * first site kk; rows hold np = W nvr elements, so tile position u sits at
     * np + W u): tile slot s, which is half a tile's rows, at off0 + s tj / 2 np,
     * the halo slot at offh. Where a slot's positions are fewer than the threads
     * (!WHOLE), the spare threads repeat the last position and store nothing. */
    const int npos = tj / TB_NTS * (np / W), slot_step = WHOLE ? W * NT : W * npos;
    const bool own = WHOLE || (int)threadIdx.x < npos;
    const int off0 = np + W * (own ? (int)threadIdx.x : npos - 1);
    using HT = typename Part<T, HW>::V;
    /* whole warps take part in the halo rows (they shuffle) */
    const bool has_h = HW * (int)(WHOLE ? threadIdx.x : threadIdx.x & ~31) < 2 * np;
    const bool own_h = HW * (int)threadIdx.x < 2 * np;
    const int fh = own_h ? HW * (int)threadIdx.x : 2 * np - HW;   /* first halo site, counted over both rows */
    const int offh = fh + (fh < np ? 0 : tj * np);
    /* the axis-2 neighbours of the vector at shared byte address a: from the
     * neighbouring lanes, at the warp's ends and the row's ends from the row
     * (periodic; a row's pad holds the images of its first sites, which advance
     * as those do). Both slots of a thread start at the same site of their rows
     * (they are whole rows apart). WHOLE: a row is whole warps. */
    const int kk0 = off0 % np;
    const uint32_t from_l = lane == 0 || (!WHOLE && kk0 == 0), from_r = lane == 31 || (!WHOLE && kk0 + W == np);
    const int ladj_b = (int)ES * ((kk0 == 0 ? n : 0) - 1), radj_b = (int)ES * ((kk0 + W == np ? -n : 0) + W);
    /* the same for the halo share (first site kk_h of its row, HW sites) */
    const int kk_h = fh % np;
    const uint32_t from_lh = lane == 0 || (!WHOLE && kk_h == 0), from_rh = lane == 31 || (!WHOLE && kk_h + HW == np);
    const int ladjh_b = (int)ES * ((kk_h == 0 ? n : 0) - 1), radjh_b = (int)ES * ((kk_h + HW == np ? -n : 0) + HW);
    auto sides = [&](const V &c, uint32_t a, T &left, T &right) {
        left = __shfl_up_sync(0xffffffffu, last(c), 1);
        right = __shfl_down_sync(0xffffffffu, first(c), 1);
        lds_if(left, a + ladj_b, from_l);
        lds_if(right, a + radj_b, from_r);
    };
    const uint32_t ring_a = smem_u32(ring), l1_a = smem_u32(l1);
    const uint32_t stage_b = ES * (uint32_t)stage_n, slot_b = ES * (uint32_t)slot_n, nb = ES * (uint32_t)np;
    const uint32_t pi_b = ES * (uint32_t)(R0 * np);
    /* the stage and phase parity of round g's plane, advanced once per round */
    int gs = 0, gs_prev = 0;
    uint32_t gph = 0u;
    auto advance = [&]() {
        gs_prev = gs;
        if (++gs == nstage) {
            gs = 0;
            gph ^= 1u;
        }
    };
    /* Round g: wait for input plane g; a wait that ran out sets the abort flag and
     * bad, which the vote at the round's end makes the block's. The round's shuffles
     * need every lane of a warp whatever its own wait gave, so in float the round
     * runs in any case (what it stores belongs to a step reported as failed); in
     * double, where the registers come out better for it, whole warps skip it.
     * us per step with the skip and without, float: 192^3 14.9 and 14.2, 250^3 26.4
     * and 25.5, 512^3 172 and 172; double: 192^3 28.4 and 27.2, 250^3 60.9 and 63.4,
     * 320^3 127 and 130. */
    constexpr bool SKIP = std::is_same<T, double>::value;
    bool bad = false;
    auto acquire = [&]() -> bool {
        const bool ok = mbar_wait(&full[gs], gph, WAIT_LIMIT);
        if (!ok) {
            atomicExch(&abort_flag, 1);
            if (SKIP) bad = true;
        }
        if (!SKIP) bad = !ok;
        return !SKIP || warp_all(ok);
    };
    /* end of round g: every thread's reads of the planes and level-1 slots are
     * done and its level-1 writes visible; thread 0 then issues the planes
     * whose stages that freed. Returns whether any thread's wait ran out. */
    auto end_round = [&](int g, bool bad) -> bool {
        const bool any_bad = tb_any(bad);
        if (!any_bad && threadIdx.x == 0) issue_upto(g + nstage - 1);
        return any_bad;
    };
    Slot<V> sl[TB_NTS];
    HT hxm, hxc;
    auto at = [&](int s) { return off0 + s * slot_step; };
    int g = 0;   /* the round: index of the input plane it waits for */
    for (int j = 0;; ++j) {
        const int it = item_q[j % TB_IQ];
        if (it < 0) break;
        int t, p0, p1;
        item_of(it, t, p0, p1);
        const int j0 = t * tj;
        /* the slots whose level-2 row is the lattice's (the last tile may hang over) */
        bool keep[TB_NTS];
#pragma unroll
        for (int s = 0; s < TB_NTS; ++s) keep[s] = WHOLE || (own && j0 * np + at(s) - np < n * np);
        /* input planes p0 - 2 and p0 - 1: this thread's phi into the register queues */
        if (acquire()) {
            const uint32_t S = ring_a + gs * stage_b + nb;
#pragma unroll
            for (int s = 0; s < TB_NTS; ++s) sl[s].x_m = lds<V>(S + ES * at(s));
            if (has_h) hxm = lds<HT>(S + ES * offh);
        }
        if (end_round(g, bad)) break;
        ++g;
        advance();
        if (acquire()) {
            const uint32_t S = ring_a + gs * stage_b + nb;
#pragma unroll
            for (int s = 0; s < TB_NTS; ++s) sl[s].x_c = lds<V>(S + ES * at(s));
            if (has_h) hxc = lds<HT>(S + ES * offh);
        }
        if (end_round(g, bad)) break;
        ++g;
        advance();
        /* two rounds per loop trip: the register queues of period two (input
         * phi, level-1 pi) then trade places without moves (512^3: 0.2288 ->
         * 0.2225 ms per step) */
#pragma unroll 2
        for (int q = p0; q <= p1 + 1; ++q, ++g, advance()) {
            if (acquire()) {
                const uint32_t Sn = ring_a + gs * stage_b;        /* plane q */
                const uint32_t S0 = ring_a + gs_prev * stage_b;   /* plane q - 1 */
                const uint32_t D1 = l1_a + ((q - p0) & 1) * slot_b;   /* level-1 plane q - 1 */
                /* level 1 at plane q - 1, at one position with input queue (xm, xc) */
                auto level1 = [&](V &xm, V &xc, int s, V &ym, V &phi1, V &pi1) {
                    /* input phi row 0 is level-1 row -1: the centre sits at n + off */
                    const uint32_t ob = ES * (uint32_t)at(s);
                    const V x_p = lds<V>(Sn + nb + ob);
                    const V um = lds<V>(S0 + ob);
                    const V up = lds<V>(S0 + 2u * nb + ob);
                    const V pv = lds<V>(S0 + pi_b + ob);
                    T left, right;
                    sides(xc, S0 + nb + ob, left, right);
                    step(xc, um, up, xm, x_p, left, right, pv, phi1, pi1);
                    /* the slot still holds this position's level-1 plane q - 3 */
                    if (!KEEP_Y) ym = lds<V>(D1 + ob);
                    if (own) sts(D1 + ob, phi1);
                    xm = xc;
                    xc = x_p;
                };
                /* level 2 at plane q - 2 (from level-1 planes q - 3 .. q - 1) at one tile
                 * position; level-1 plane q - 2 was written in the last round */
                const int m2 = q - 2;
                const uint32_t L0 = l1_a + ((m2 - p0 + 1) & 1) * slot_b;
                /* global row j0 - 1 + r1 of plane m2: the tile position's offset from row j0 - 1 */
                const size_t gbase = ((size_t)m2 * n + (size_t)j0) * np - (size_t)np;
                auto level2 = [&](Slot<V> &x, const V &ym, int s) {
                    const uint32_t ob = L0 + ES * (uint32_t)at(s);
                    const V um = lds<V>(ob - nb);
                    const V up = lds<V>(ob + nb);
                    T left, right;
                    sides(x.y_c, ob, left, right);
                    V phi2, pi2;
                    step(x.y_c, um, up, ym, x.y_p, left, right, x.z, phi2, pi2);
                    if (keep[s]) {
                        *reinterpret_cast<V *>(phi_out + (gbase + at(s))) = phi2;
                        *reinterpret_cast<V *>(pi_out + (gbase + at(s))) = pi2;
                    }
                };
                /* per tile position: level 1 at plane q - 1, then level 2 at plane q - 2,
                 * which needs the position's own level-1 plane q - 1 just computed */
#pragma unroll
                for (int s = 0; s < TB_NTS; ++s) {
                    Slot<V> &x = sl[s];
                    V ym, phi1, pi1;
                    level1(x.x_m, x.x_c, s, ym, phi1, pi1);
                    if (KEEP_Y) ym = x.y_c;
                    x.y_c = x.y_p;
                    x.y_p = phi1;
                    x.z = x.zz;
                    x.zz = pi1;
                    if (m2 >= p0) level2(x, ym, s);
                }
                if (has_h) {
                    /* level 1 at plane q - 1 on the halo share */
                    const uint32_t ob = ES * (uint32_t)offh;
                    const HT xp = lds<HT>(Sn + nb + ob);
                    const HT um = lds<HT>(S0 + ob);
                    const HT up = lds<HT>(S0 + 2u * nb + ob);
                    const HT pv = lds<HT>(S0 + pi_b + ob);
                    const uint32_t a = S0 + nb + ob;
                    T left = __shfl_up_sync(0xffffffffu, last(hxc), 1);
                    T right = __shfl_down_sync(0xffffffffu, first(hxc), 1);
                    lds_if(left, a + ladjh_b, from_lh);
                    lds_if(right, a + radjh_b, from_rh);
                    HT phi1, pi1;
                    step(hxc, um, up, hxm, xp, left, right, pv, phi1, pi1);
                    if (WHOLE || own_h) sts(D1 + ob, phi1);
                    hxm = hxc;
                    hxc = xp;
                }
            }
            if (end_round(g, bad)) {
                bad = true;
                break;
            }
        }
        if (bad) break;
    }
    __syncthreads();
    /* this block's items are done: the next step may be scheduled */
    pdl_allow_next();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&st->item_done, 1u) == gridDim.x - 1) {
            st->item_next = 0u;
            st->item_done = 0u;
        }
    }
    if (abort_flag) {
        /* record, then let every issued copy land before the block exits */
        if (threadIdx.x == 0) {
            atomicExch(&st->err, ERR_TMA_TIMEOUT);
            for (int q = max(issued - nstage, 0); q < issued; ++q)
                mbar_wait(&full[q % nstage], (uint32_t)((q / nstage) & 1), WAIT_LIMIT / 8);
        }
        __syncthreads();
    }
}

}  // namespace

int sm_count();

/* Geometry of the two-step pass (d = 3, static background, rows of whole
 * 16-byte vectors (padded, where n is no multiple of one), rows of at least one warp: with shorter ones a round's
 * latency is all there is, 100^3 in float 6.5 us per step against 6.7). A tile is TJ rows; its TJ n / W positions are two per
 * thread, at most 512 threads (so TJ n <= 4096 floats or 2048 doubles), and
 * the halo rows' 2 n / W positions are no more than the threads (TJ >= 4).
 * Shared memory: 4 to 6 input stages of 2 TJ + 6 rows and 2 level-1 planes of
 * TJ + 2 rows in the 227 KB of one block per SM. TJ and the plane parts P are
 * those of the least modelled time: whole rounds of items over the SMs, times
 * the planes an item streams (n / P and four beyond them), times a plane's
 * time, 1 us (the chain of its loads, updates and barrier; 1.15 in general) and 0.036 us (float)
 * or 0.05 us (double) per vector of a scheduler's warps (64^3 1.1 us a plane,
 * 512^3 1.63, 256^3 in double 1.86). So 512^3 takes 9 parts in 4 rounds (198.6
 * us per step; 16 parts in 7 rounds 213). Double needs dx^2 to divide in one
 * or two operations (one step per pass otherwise). */
bool step3tb_geometry(const StepConst &k, int prec, int tl, int &tj, int &nstage, size_t &smem, unsigned &grid,
                      int &parts) {
    const int W = prec == P_FP64 ? 2 : 4;
    const int n = k.n, np = k.pitch;
    if (k.d != 3 || k.expanding || tl != 2 || np % W != 0 || np / W < 32 || n > 1024) return false;
    if (prec == P_FP64 && !k.dx2_pow2 && !k.dx2_pair) return false;
    const size_t row = (size_t)np * (prec == P_FP64 ? 8 : 4);
    const size_t budget = 227 * 1024 - 1024 - TB_HDR;   /* dynamic share of 227 KB, room for the static variables */
    const int nv = np / W;
    const long long slots = sm_count();
    double best = 0.0;
    for (int t = 4; t <= 32 && t * nv <= TB_NTS * TB_MAXT; t += TB_NTS) {
        const size_t stage = (size_t)(2 * t + 6) * row, lev = (size_t)2 * (t + 2) * row;
        if (lev + 4 * stage > budget) break;
        const long long ntiles = (n + t - 1) / t;
        const int per_sched = (t * nv + 255) / 256;   /* warps per scheduler, two vectors each */
        /* rows of whole warps in whole tiles save the masks and per-slot wraps (launch below) */
        const bool whole = whole_rows(n, np, prec, t);
        const double round = (whole ? 1.0 : 1.15) + (prec == P_FP64 ? 0.05 : 0.036) * (4.0 * per_sched + (2 * nv + 127) / 128);
        for (long long w = 1; w <= 8; ++w) {
            const long long P = std::min<long long>(w * slots / ntiles, n / 4);
            if (P < 1) continue;
            const long long waves = (ntiles * P + slots - 1) / slots;
            const double cost = (double)waves * ((double)((n + P - 1) / P) + 4.0) * round;
            if (best == 0.0 || cost < best) {
                best = cost;
                tj = t;
                parts = (int)P;
                nstage = (int)std::min<size_t>((budget - lev) / stage, 6);
                smem = TB_HDR + (size_t)nstage * stage + lev;
            }
        }
    }
    if (best == 0.0) return false;
    const char *env = std::getenv("CB_STEP3TB_PARTS");
    if (env && std::atoi(env) >= 1 && std::atoi(env) <= n) parts = std::atoi(env);
    const long long nitems = (long long)((n + tj - 1) / tj) * parts;
    grid = (unsigned)std::min(nitems, slots);
    return true;
}

cudaError_t launch_step3_tb(int prec, const StepConst &k, int tl, const void *phi_in, const void *pi_in,
                            void *phi_out, void *pi_out, DevState *st, cudaStream_t s) {
    int tj, nstage, parts;
    size_t smem;
    unsigned grid;
    if (!step3tb_geometry(k, prec, tl, tj, nstage, smem, grid, parts)) return cudaErrorInvalidValue;
    const int W = prec == P_FP64 ? 2 : 4;
    const int npos = tj * (k.pitch / W);
    const int nc = (npos + 64 - 1) / 64 * 32;
    /* rows of whole warps, whole tiles, every thread two positions: the halo rows'
     * 2 n sites then spread as 1, 2 (float: 4) per thread where that comes out even.
     * Other rows spread them as one pair of floats or one double per thread where the
     * threads suffice (250^3 float 29.3 us per step with whole vectors on some of the
     * warps, 28.4 with pairs, 31.5 site by site; 200^3 double 34.9 -> 33.7) */
    const bool whole = whole_rows(k.n, k.pitch, prec, tj);
    auto go = [&](auto t, auto by, auto hw, auto wh) -> cudaError_t {
        using T = decltype(t);
        constexpr int HW = decltype(hw)::value;
        auto fn = k_step3_t2<T, decltype(by)::value, HW, decltype(wh)::value>;
        if constexpr (decltype(wh)::value) {
            /* rows of 2^5, 2^6, 2^7 vectors; the halo share that goes with each */
            constexpr int per_w = 16 / (int)sizeof(T);
            if (nc == TB_MAXT && k.n == 32 * per_w && HW == per_w) fn = k_step3_t2<T, decltype(by)::value, HW, true, 32>;
            if (nc == TB_MAXT && k.n == 64 * per_w) fn = k_step3_t2<T, decltype(by)::value, HW, true, 64>;
            if (nc == TB_MAXT && k.n == 128 * per_w) fn = k_step3_t2<T, decltype(by)::value, HW, true, 128>;
        }
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        return launch_pdl(fn, dim3(grid), dim3(nc), smem, s, k, tj, nstage, parts, (const T *)phi_in,
                          (const T *)pi_in, (T *)phi_out, (T *)pi_out, st);
    };
    using std::integral_constant;
    constexpr std::true_type yes{};
    constexpr std::false_type no{};
    constexpr integral_constant<int, 1> one{};
    constexpr integral_constant<int, 2> two{};
    constexpr integral_constant<int, 4> four{};
    if (prec != P_FP64) {
        constexpr integral_constant<int, BY_MUL> mul{};
        if (!whole) return k.pitch <= nc ? go(0.f, mul, two, no) : go(0.f, mul, four, no);
        return 2 * k.n == nc ? go(0.f, mul, one, yes) : k.n == nc ? go(0.f, mul, two, yes) : go(0.f, mul, four, yes);
    }
    auto doubles = [&](auto by) {
        if (!whole) return 2 * k.pitch <= nc ? go(0.0, by, one, no) : go(0.0, by, two, no);
        return 2 * k.n == nc ? go(0.0, by, one, yes) : go(0.0, by, two, yes);
    };
    return k.dx2_pow2 ? doubles(integral_constant<int, BY_MUL>{}) : doubles(integral_constant<int, BY_PAIR>{});
}

}  // namespace cb
