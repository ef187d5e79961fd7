/* cb_step3_df.cu -- plain steps of an expanding background (d = 3): the pending
 * drift, the kick, and the sums of the Friedmann update (reference
 * Bubble::oneStep, src/bubble.cpp:849-876). A step that reports every box
 * average runs on cb_step3.cu.
 *
 * Drift-first ordering as there: the stored phi is one drift behind, and a
 * step first applies phi += (dt pi) p to every site it reads.
 *
 *  - Tiles of TJ full rows; work items (tile, plane part); input planes -- phi
 *    and pi rows j0 - 1 .. j0 + TJ -- arrive by TMA bulk copies into a ring.
 *  - A thread owns two vectors of the tile (and a share of the halo rows) in
 *    every plane and marches them along axis 0. Round q drifts its vectors of
 *    plane q, once, into one of two shared planes (for the neighbours) and into
 *    registers, then computes plane q - 1: its own column (planes q - 2 .. q of
 *    phi, plane q - 1 of pi) is in registers, the neighbours along axis 2 come
 *    by shuffle, and only the two neighbour rows are read back. One barrier of
 *    the block per round; it also frees plane q's stage, whose refill one thread
 *    issues.
 *  - Successive steps march the planes in opposite directions: what a step
 *    wrote last is what the next one reads first, and is still in L2.
 *  - The sums of an item go to its own row of partial sums, added in a fixed
 *    order; the background is updated in double by one warp.
 *  - MS: one cooperative launch runs many steps. After each, every block waits
 *    (bounded) until all have counted it done, forms the totals itself and
 *    updates its own copy of the background (block 0 also the run's), while the
 *    first planes of the next step are on their way.
 *  - What bounds it: the chains of a round (load, drift, kick, barrier) over 16
 *    warps; ncu on 256^3: issue 41 %, FP64 pipe 33 % (double), DRAM 47-52 %. Four
 *    vectors per thread spill, three blocks of 80 registers too; rows of a thread
 *    one below the other (a third fewer shared reads) measured the same.
 *  - Waits are bounded; a timed-out block records an error word and leaves with
 *    its copies landed.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "cb_internal.h"
#include "cb_launch.cuh"
#include "cb_march.cuh"
#include "cb_step_common.cuh"
#include "cb_tma.cuh"

namespace cb {

int sm_count();

namespace {

constexpr int DF_MAXT = 512;    /* threads per block */
constexpr int DF_NTS = 2;       /* tile vectors per thread */
constexpr int DF_HDR = 256;     /* full[nstage] mbarriers (nstage <= 8) */
constexpr int DF_IQ = 8;

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

/* Wait (bounded) until *ctr reaches target; false if the wait ran out. Only
 * blocks of one cooperative launch, resident together, wait so. */
__device__ __forceinline__ bool grid_wait(const unsigned *ctr, unsigned target) {
    if (ld_acquire(ctr) >= target) return true;
    const long long t0 = clock64();
    while (ld_acquire(ctr) < target) {
        __nanosleep(64);
        if (clock64() - t0 > WAIT_LIMIT) return false;
    }
    return true;
}

/* The per-site arithmetic of one step, with the sums' terms. */
template <typename T, int BY, bool EG, bool RAG>
struct Site;

template <int BY, bool EG, bool RAG>
struct Site<float, BY, EG, RAG> {
    using V = float4;
    F2 fl, idx2, nfv, dt, c2, nc3, c4, v2, nv3, v4, dv, kw, eg, p;
    struct Pairs {   /* Kahan-compensated packed pair; c: the compensation, negated */
        F2 s{0ull}, c{0ull};
        __device__ __forceinline__ void add(F2 x) {
            const F2 y = f2_add(x, c);
            const F2 t = f2_add(s, y);
            c = f2_sub(y, f2_sub(t, s));
            s = t;
        }
        __device__ __forceinline__ double value() const {
            return __dadd_rn(__dadd_rn((double)f2_lo(s), (double)f2_lo(c)), __dadd_rn((double)f2_hi(s), (double)f2_hi(c)));
        }
    };
    /* the sums of a vector's pairs, compensated; padded rows, which the generic kernel took
     * before: every site's term in double (322^3 110.2 us per step, 109.6 with sums of pairs) */
    using Sum = std::conditional_t<RAG, Acc<double>, Pairs>;
    __device__ __forceinline__ static Sum zero() { return Sum{}; }
    __device__ __forceinline__ Site(const StepConst &k, const DevState *st)
        : fl(f2_splat((float)st->fl)), idx2(f2_splat(k.inv_dx2f)), nfv(f2_splat(-(float)st->fv)), dt(f2_splat(k.dtf)),
          c2(f2_splat(k.c2f)), nc3(f2_splat(-k.c3f)), c4(f2_splat(k.c4f)), v2(f2_splat(k.v2f)), nv3(f2_splat(-k.v3f)),
          v4(f2_splat(k.v4f)), dv(f2_splat(k.dvf)), kw(f2_splat((float)st->kin_w)),
          eg(f2_splat((float)(0.5 * (double)(float)st->inv_adx * (double)(float)st->inv_adx))),
          p(f2_splat((float)st->drift_p)) {}
    __device__ __forceinline__ V drift(const V &f, const V &m) const {
        const F2 a = f2_add(f2_pack(f.x, f.y), f2_mul(f2_mul(dt, f2_pack(m.x, m.y)), p));
        const F2 b = f2_add(f2_pack(f.z, f.w), f2_mul(f2_mul(dt, f2_pack(m.z, m.w)), p));
        return make_float4(f2_lo(a), f2_hi(a), f2_lo(b), f2_hi(b));
    }
    struct Terms {
        F2 ek, ep, eg;
    };
    __device__ __forceinline__ F2 pair(F2 cc, F2 um, F2 up, F2 im, F2 ip, F2 km, F2 kp, F2 pp, Terms &t) const {
        const F2 two = f2_add(cc, cc);
        const F2 t0 = f2_add(f2_sub(ip, two), im);
        const F2 t1 = f2_add(f2_sub(up, two), um);
        const F2 t2 = f2_add(f2_sub(kp, two), km);
        const F2 lap = f2_add(f2_add(t0, t1), t2);
        const F2 h = f2_fma(cc, f2_fma(cc, c4, nc3), c2);
        const F2 force = f2_fma(f2_mul(fl, lap), idx2, f2_mul(nfv, f2_mul(cc, h)));
        const F2 pn = f2_fma(dt, force, pp);
        t.ek = f2_mul(f2_mul(kw, pn), pn);
        t.ep = f2_fma(f2_mul(cc, cc), f2_fma(cc, f2_fma(cc, v4, nv3), v2), dv);
        if (EG) {
            const F2 gx = f2_sub(up, cc), gy = f2_sub(ip, cc), gz = f2_sub(kp, cc);
            t.eg = f2_mul(eg, f2_fma(gz, gz, f2_fma(gy, gy, f2_mul(gx, gx))));
        }
        return pn;
    }
    /* pi after the kick; with `count` the vector enters the sums (RAG: its first `sites`; the
     * others are images in a row's pad) */
    __device__ __forceinline__ V kick(const V &c, const V &um, const V &up, const V &im, const V &ip, float l, float r,
                                      const V &pv, bool count, int sites, Sum (&acc)[3]) const {
        const F2 mid = f2_pack(c.y, c.z);
        Terms a, b;
        const F2 pa = pair(f2_pack(c.x, c.y), f2_pack(um.x, um.y), f2_pack(up.x, up.y), f2_pack(im.x, im.y),
                           f2_pack(ip.x, ip.y), f2_pack(l, c.x), mid, f2_pack(pv.x, pv.y), a);
        const F2 pb = pair(f2_pack(c.z, c.w), f2_pack(um.z, um.w), f2_pack(up.z, up.w), f2_pack(im.z, im.w),
                           f2_pack(ip.z, ip.w), mid, f2_pack(c.w, r), f2_pack(pv.z, pv.w), b);
        if (count) {
            auto put = [&](Sum &s, F2 x, F2 y) {
                if constexpr (RAG) {
                    s.add((double)f2_lo(x));
                    s.add((double)(sites > 1 ? f2_hi(x) : 0.f));
                    s.add((double)(sites > 2 ? f2_lo(y) : 0.f));
                    s.add((double)(sites > 3 ? f2_hi(y) : 0.f));
                } else {
                    s.add(f2_add(x, y));
                }
            };
            put(acc[S_EK], a.ek, b.ek);
            put(acc[S_EP], a.ep, b.ep);
            if (EG) put(acc[S_EG], a.eg, b.eg);
        }
        return make_float4(f2_lo(pa), f2_hi(pa), f2_lo(pb), f2_hi(pb));
    }
};

template <int BY, bool EG, bool RAG>
struct Site<double, BY, EG, RAG> {
    using V = double2;
    using A = Ar<double>;
    using Sum = Acc<double>;
    __device__ __forceinline__ static Sum zero() { return Sum{}; }
    const StepConst &k;
    double fl, fv, kw, p, adx, inv_adx;
    bool adx_pow2;
    __device__ __forceinline__ Site(const StepConst &kk, const DevState *st)
        : k(kk), fl(st->fl), fv(st->fv), kw(st->kin_w), p(st->drift_p), adx(st->adx), inv_adx(st->inv_adx),
          adx_pow2(st->adx_pow2 != 0) {}
    __device__ __forceinline__ double grad(double x) const { return adx_pow2 ? A::mul(x, inv_adx) : A::div(x, adx); }
    __device__ __forceinline__ V drift(const V &f, const V &m) const {
        return make_double2(A::add(f.x, A::mul(A::mul(k.dt, m.x), p)), A::add(f.y, A::mul(A::mul(k.dt, m.y), p)));
    }
    /* m: 1, or 0 for an image in a row's pad */
    __device__ __forceinline__ double site(double c, double um, double up, double im, double ip, double l, double r,
                                           double pv, bool count, double m, Sum (&acc)[3]) const {
        const double two = A::add(c, c);
        const double t0 = A::add(A::sub(ip, two), im);
        const double t1 = A::add(A::sub(up, two), um);
        const double t2 = A::add(A::sub(r, two), l);
        const double lap = A::add(A::add(t0, t1), t2);
        const double force = A::sub(over_dx2<BY>(k, A::mul(fl, lap)), A::mul(fv, dV<double>(k, c)));
        const double pn = A::add(pv, A::mul(k.dt, force));
        if (count) {
            auto put = [&](int i, double x) { acc[i].s = __fma_rn(m, x, acc[i].s); };   /* a plain add for m = 1 */
            put(S_EK, A::mul(A::mul(kw, pn), pn));
            put(S_EP, Vpot<double>(k, c));
            if (EG) {
                const double gx = grad(A::sub(up, c)), gy = grad(A::sub(ip, c)), gz = grad(A::sub(r, c));
                put(S_EG, A::mul(0.5, A::add(A::add(A::sq(gx), A::sq(gy)), A::sq(gz))));
            }
        }
        return pn;
    }
    __device__ __forceinline__ V kick(const V &c, const V &um, const V &up, const V &im, const V &ip, double l, double r,
                                      const V &pv, bool count, int sites, Sum (&acc)[3]) const {
        const double a = site(c.x, um.x, up.x, im.x, ip.x, l, c.y, pv.x, count, 1.0, acc);
        const double b = site(c.y, um.y, up.y, im.y, ip.y, c.x, r, pv.y, count, RAG && sites < 2 ? 0.0 : 1.0, acc);
        return make_double2(a, b);
    }
};

/* All threads of a block: tot[s] = sum over rows r of partials[r * NSUM + s] for
 * s < NS (the rest 0), in a fixed order for a block size: threads stride the
 * rows, lanes by shuffle, warps in order. Valid in every thread on return. */
template <int NS>
__device__ void df_totals(const double *partials, unsigned rows, double *tot, double (*red)[3]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double acc[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) acc[s] = 0.0;
    for (unsigned b = threadIdx.x; b < rows; b += blockDim.x) {
#pragma unroll
        for (int s = 0; s < NS; ++s) acc[s] = __dadd_rn(acc[s], __ldcg(partials + (size_t)b * NSUM + s));
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        double x = acc[s];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x = __dadd_rn(x, __shfl_down_sync(0xffffffffu, x, o));
        if (lane == 0) red[w][s] = x;
    }
    __syncthreads();
    if (threadIdx.x < NSUM) {
        double x = 0.0;
        if (threadIdx.x < NS)
            for (int i = 0; i < nw; ++i) x = __dadd_rn(x, red[i][threadIdx.x]);
        tot[threadIdx.x] = x;
    }
    __syncthreads();
}

/* FORM: 0 WHOLE rows, 1 rows of whole vectors, 2 padded rows (RAG) */
template <typename T, int BY, bool EG, bool MS, int FORM>
__global__ void __launch_bounds__(DF_MAXT, 1)
    k_step3_df(StepConst k, int tj, int nstage, int parts, int nsteps, int keep_l2, const T *phi_a, const T *pi_a,
               T *phi_b, T *pi_b, DevState *st, double *partials) {
    using S = Site<T, BY, EG, FORM == 2>;
    using V = typename S::V;
    constexpr int W = Vec<T>::W, NS = EG ? 3 : 2;
    constexpr bool WHOLE = FORM == 0, RAG = FORM == 2;
    constexpr uint32_t ES = sizeof(T);
    extern __shared__ __align__(128) unsigned char smraw[];
    __shared__ int abort_flag;
    __shared__ int item_q[DF_IQ];
    __shared__ double item_red[2][DF_MAXT / 32][3];
    __shared__ double tot[NSUM];
    __shared__ DevState ls;   /* the block's copy of the background */

    const int n = k.n, np = RAG ? k.pitch : n;
    const int rows = tj + 2;                     /* phi and pi rows j0 - 1 .. j0 + tj of a stage */
    const int half_n = rows * np;                /* elements of either */
    uint64_t *full = reinterpret_cast<uint64_t *>(smraw);
    T *ring = reinterpret_cast<T *>(smraw + DF_HDR);
    T *drifted = ring + (size_t)nstage * 2 * half_n;   /* the drifted phi rows of two planes */
    const bool issuer = (int)threadIdx.x == (int)blockDim.x - 32;   /* its warp has no halo rows to drift */
    const int ntiles = (n + tj - 1) / tj;
    const int items = ntiles * parts;
    const size_t row_bytes = (size_t)np * ES, plane = (size_t)n * np;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, NT = blockDim.x, nw = NT >> 5;
    T *const fphi[2] = {const_cast<T *>(phi_a), phi_b}, *const fpi[2] = {const_cast<T *>(pi_a), pi_b};
    auto item_of = [&](int it, int &t, int &p0, int &p1) {
        const int c = it / ntiles;
        t = it % ntiles;
        p0 = (int)((long long)c * n / parts);
        p1 = (int)((long long)(c + 1) * n / parts);
    };

    /* ---- the copies (one thread), in the order the block streams its planes ---- */
    const uint64_t pol = keep_l2 ? l2_evict_first() : l2_evict_normal();
    int pr_j = 0, pr_u = 0, pr_n = 0, is_stage = 0, issued = 0, sp_issue = 0;
    bool pr_done = false;
    __shared__ int pr_s[4];   /* the issuer's: first plane, plane step, source row, rows before the wrap */
    /* a block's first item of a step is its own index (the grid never exceeds
     * the items); later ones come from the queue (MS: one item per block) */
    auto next_item = [&](bool first) {
        int cur = (int)blockIdx.x;
        if (!first) cur = MS ? items : (int)gridDim.x + (int)atomicAdd(&st->item_next, 1u);
        const int it = cur < items ? cur : -1;
        item_q[pr_j % DF_IQ] = it;
        ++pr_j;
        if (it < 0) {
            pr_done = true;
            return;
        }
        int t, p0, p1;
        item_of(it, t, p0, p1);
        const bool rev = (k.odd + sp_issue) & 1;
        pr_s[0] = rev ? p1 : p0 - 1;
        pr_s[1] = rev ? -1 : 1;
        pr_s[2] = (t * tj - 1 + n) % n;
        pr_s[3] = min(rows, n - pr_s[2]);
        pr_u = 0;
        pr_n = p1 - p0 + 2;
    };
    auto issue_upto = [&](int last) {
        while (!pr_done && issued <= last) {
            const int pl = pr_s[0] + pr_s[1] * pr_u;
            const size_t base = (size_t)(pl < 0 ? pl + n : pl >= n ? pl - n : pl) * plane;
            const T *gphi = fphi[sp_issue & 1] + base, *gpi = fpi[sp_issue & 1] + base;
            const int r0 = pr_s[2], c0 = pr_s[3];
            T *dst = ring + (size_t)is_stage * 2 * half_n;
            uint64_t *bar = &full[is_stage];
            mbar_arrive_expect_tx(bar, (uint32_t)(2 * rows * row_bytes));
            bulk_g2s(dst, gphi + (size_t)r0 * np, (uint32_t)(c0 * row_bytes), bar, pol);
            bulk_g2s(dst + half_n, gpi + (size_t)r0 * np, (uint32_t)(c0 * row_bytes), bar, pol);
            if (c0 < rows) {
                bulk_g2s(dst + (size_t)c0 * np, gphi, (uint32_t)((rows - c0) * row_bytes), bar, pol);
                bulk_g2s(dst + half_n + (size_t)c0 * np, gpi, (uint32_t)((rows - c0) * row_bytes), bar, pol);
            }
            ++issued;
            if (++is_stage == nstage) is_stage = 0;
            if (++pr_u == pr_n) next_item(false);
        }
    };

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < nstage; ++s) mbar_init(&full[s], 1);
        fence_mbar_init();
    }
    __syncthreads();
    pdl_wait();   /* the previous step's fields, device state and work queue */
    if (issuer) {
        ls = *st;
        next_item(true);
        issue_upto(nstage - 1);
    }
    __syncthreads();

    /* this thread's vectors: element offsets in a plane's phi rows (row 0 is
     * j0 - 1, so tile vector u sits at np + W u); spare threads repeat the last
     * vector and store nothing. The axis-2 neighbours come from the adjacent
     * lanes, at the warp's and the row's ends from the row (periodic; a row's pad
     * holds the images of its first sites). WHOLE: rows of whole warps in whole
     * tiles, every slot of a thread at the same place of its row. */
    const int npos = tj * (np / W), slot_step = W * NT;
    int offs[DF_NTS], ladj_b[DF_NTS], radj_b[DF_NTS];
    uint32_t from_l[DF_NTS], from_r[DF_NTS];
    bool own[DF_NTS];
#pragma unroll
    for (int s = 0; s < DF_NTS; ++s) {
        const int u = threadIdx.x + s * NT;
        own[s] = WHOLE || u < npos;
        offs[s] = np + W * (own[s] ? u : npos - 1);
        const int kk = offs[s] % np;
        from_l[s] = lane == 0 || (!WHOLE && kk == 0);
        from_r[s] = lane == 31 || (!WHOLE && kk + W == np);
        ladj_b[s] = (int)ES * ((kk == 0 ? n : 0) - 1);
        radj_b[s] = (int)ES * ((kk + W == np ? -n : 0) + W);
    }
    auto at = [&](int s) { return WHOLE ? offs[0] + s * slot_step : offs[s]; };
    const uint32_t ring_a = smem_u32(ring), drifted_a = smem_u32(drifted), nb = ES * (uint32_t)np, half_b = ES * (uint32_t)half_n;
    const uint32_t stage_b = 2u * half_b;

    int gs = 0;                /* stage of this round's plane */
    uint32_t gph = 0u;
    int g = 0;                 /* the round, counted over all items and steps */
    bool bad = false;
    int j = 0;
    typename S::Sum acc[3];
    V xm[DF_NTS], xc[DF_NTS], z[DF_NTS];
    for (int sp = 0; !bad && sp < (MS ? nsteps : 1); ++sp) {
        const S site(k, &ls);
        T *const phi_o = fphi[(sp + 1) & 1], *const pi_o = fpi[(sp + 1) & 1];
        for (;; ++j) {
            const int it = item_q[j % DF_IQ];
            if (it < 0) {
                ++j;
                break;
            }
            int t, p0, p1;
            item_of(it, t, p0, p1);
            const int j0 = t * tj;
            /* the slots whose row is the lattice's (the last tile may hang over) */
            bool keep[DF_NTS];
#pragma unroll
            for (int s = 0; s < DF_NTS; ++s) keep[s] = WHOLE || (own[s] && j0 * np + offs[s] - np < n * np);
#pragma unroll
            for (int s = 0; s < 3; ++s) acc[s] = S::zero();
            auto march = [&](auto dir) {
                constexpr bool REV = decltype(dir)::value;
#pragma unroll 2
                for (int u = 0; u <= p1 - p0 + 1; ++u, ++g) {
                    /* the round's shuffles need every lane of a warp whatever its own wait gave:
                     * the round runs in any case, and the vote at its end stops the block
                     * (what it stored belongs to a step reported as failed). In double 192^3
                     * 45.4 us per step; 46.7 with a warp's vote before the round instead. */
                    if (!mbar_wait(&full[gs], gph, WAIT_LIMIT)) {
                        atomicExch(&abort_flag, 1);
                        bad = true;
                    }
                    const uint32_t Sq = ring_a + gs * stage_b;
                    const uint32_t Dq = drifted_a + (g & 1) * half_b, Dp = drifted_a + (~g & 1) * half_b;
                    const int i = REV ? p1 + 1 - u : p0 - 2 + u;   /* the plane to compute */
                    /* element 0 of row j0 - 1 of plane i */
                    const size_t gbase = ((size_t)i * n + (size_t)j0) * np - (size_t)np;
#pragma unroll
                    for (int s = 0; s < DF_NTS; ++s) {
                        const uint32_t ob = ES * (uint32_t)at(s);
                        const V m = lds<V>(Sq + half_b + ob);
                        const V xp = site.drift(lds<V>(Sq + ob), m);
                        if (own[s]) sts(Dq + ob, xp);
                        if (u >= 2) {
                            const V um = lds<V>(Dp + ob - nb), up = lds<V>(Dp + ob + nb);
                            const int q = WHOLE ? 0 : s;
                            T left = __shfl_up_sync(0xffffffffu, last(xc[s]), 1);
                            T right = __shfl_down_sync(0xffffffffu, first(xc[s]), 1);
                            lds_if(left, Dp + ob + ladj_b[q], from_l[q]);
                            lds_if(right, Dp + ob + radj_b[q], from_r[q]);
                            const int sites = RAG ? min(W, n - offs[s] % np) : W;
                            const V pn = site.kick(xc[s], um, up, REV ? xp : xm[s],
                                                   REV ? xm[s] : xp, left, right, z[s], keep[s], sites, acc);
                            if (keep[s]) {
                                *reinterpret_cast<V *>(pi_o + (gbase + at(s))) = pn;
                                *reinterpret_cast<V *>(phi_o + (gbase + at(s))) = xc[s];
                            }
                        }
                        xm[s] = xc[s];
                        xc[s] = xp;
                        z[s] = m;
                    }
                    /* the halo rows' drift */
                    for (int h = threadIdx.x; h < 2 * (np / W); h += NT) {
                        const uint32_t ob = ES * (uint32_t)(W * h + (W * h < np ? 0 : tj * np));
                        const uint32_t from = ring_a + gs * stage_b + ob;
                        sts(drifted_a + (g & 1) * half_b + ob, site.drift(lds<V>(from), lds<V>(from + half_b)));
                    }
                    /* end of the round: the drifted plane is visible, its stage and the drifted
                     * plane before it are free */
                    bad = tb_any(bad);
                    if (!bad && issuer) issue_upto(g + nstage);
                    if (++gs == nstage) {
                        gs = 0;
                        gph ^= 1u;
                    }
                    if (bad) break;
                }
            };
            if ((k.odd + sp) & 1) march(std::true_type{});
            else march(std::false_type{});
            if (bad) break;
            /* the item's sums: lanes by shuffle, warps in order, to the item's own row */
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                double x = acc[s].value();
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) x = __dadd_rn(x, __shfl_down_sync(0xffffffffu, x, o));
                if (lane == 0) item_red[j & 1][warp][s] = x;
            }
            __syncthreads();
            if (threadIdx.x < NSUM) {
                double x = 0.0;
                if (threadIdx.x < NS)
                    for (int q = 0; q < nw; ++q) x = __dadd_rn(x, item_red[j & 1][q][threadIdx.x]);
                partials[((size_t)(MS ? (sp & 1) * items : 0) + it) * NSUM + threadIdx.x] = x;
            }
        }
        if (MS && !bad) {
            /* all blocks' fields and rows of this step, then its totals and the update */
            __threadfence();
            __syncthreads();
            if (issuer) {
                atomicAdd(&st->step_bar, 1u);
                if (!grid_wait(&st->step_bar, gridDim.x * (unsigned)(sp + 1))) {
                    atomicExch(&abort_flag, 1);
                    bad = true;
                } else if (sp + 1 < nsteps) {
                    asm volatile("fence.proxy.async.global;" ::: "memory");
                    sp_issue = sp + 1;
                    pr_done = false;
                    next_item(true);
                    issue_upto(g + nstage - 1);
                }
            }
            bad = tb_any(bad);
            if (bad) break;
            __threadfence();
            df_totals<NS>(partials + (size_t)(sp & 1) * items * NSUM, (unsigned)items, tot, item_red[0]);
            if (warp == 0) epilogue(k, &ls, tot, false, false, lane);
            if (warp == 1 && blockIdx.x == 0) epilogue(k, st, tot, false, false, lane);
            __syncthreads();
        }
    }
    __threadfence();
    __syncthreads();
    pdl_allow_next();
    __shared__ bool is_last;
    if (threadIdx.x == 0) {
        is_last = atomicAdd(&st->item_done, 1u) == gridDim.x - 1;
        if (is_last) {
            st->item_next = 0u;
            st->item_done = 0u;
            st->step_bar = 0u;
        }
    }
    __syncthreads();
    if (abort_flag) {
        /* record, then let every issued copy land before the block exits */
        if (issuer) {
            atomicExch(&st->err, ERR_TMA_TIMEOUT);
            for (int q = issued > nstage ? issued - nstage : 0; q < issued; ++q)
                mbar_wait(&full[q % nstage], (uint32_t)((q / nstage) & 1), WAIT_LIMIT / 8);
        }
        __syncthreads();
        return;
    }
    if (!MS && is_last) {
        __threadfence();
        df_totals<NS>(partials, (unsigned)items, tot, item_red[0]);
        if (warp == 0) epilogue(k, st, tot, false, false, lane);
    }
}

}  // namespace

namespace {

/* Tiles, plane parts and ring of a step. */
struct PlanDF {
    int tj = 0, nstage = 0, parts = 0, threads = 0, items = 0;
    bool whole = false;
    size_t smem = 0;
    unsigned grid = 0;
};

/* One block per SM of two vectors per thread (TJ n / W <= 1024), with at least
 * three stages of the ring beside the two drifted planes. TJ and the parts are
 * those of the least modelled time: whole rounds of items over the SMs, times
 * an item's planes (its own and two), times a round's time, which the warps'
 * chains set (256^3 in double, 16 warps 1.41 us, 192^3 with 12 1.18, 128^3 with
 * 8 0.93; rows that are no whole warps 8 % more). So 256^3 takes 32 tiles in 9
 * parts, two rounds of 31 planes: 94 us per step, 99 in 4 parts of 66. */
bool plan_df(const StepConst &k, int prec, PlanDF &best) {
    const int W = prec == P_FP64 ? 2 : 4;
    const int n = k.n, nv = k.pitch / W;
    if (k.d != 3 || !k.expanding || k.force_generic || k.pitch % W != 0 || n < 64) return false;
    const size_t row = (size_t)k.pitch * (prec == P_FP64 ? 8 : 4), budget = 222 * 1024 - DF_HDR;
    const long long slots = sm_count();
    double least = 0.0;
    for (int t = 2; t + 2 <= n; ++t) {
        const int threads = (t * nv + 63) / 64 * 32;
        const size_t stage = 2 * (size_t)(t + 2) * row;
        if (threads > DF_MAXT || 4 * stage > budget) break;
        const bool whole = whole_rows(n, k.pitch, prec, t);
        const double round = (0.55 + 0.05 * ((threads + 127) / 128 * 4)) * (whole ? 1.0 : 1.08);
        const long long ntiles = (n + t - 1) / t;
        for (long long w = 1; w <= 6; ++w) {
            const long long P = std::min<long long>(w * slots / ntiles, n / 2);
            if (P < 1) continue;
            const long long rounds = (ntiles * P + slots - 1) / slots;
            /* several rounds: launches between the steps */
            const double us = (rounds > 1 ? 4.0 : 0.0) + (double)rounds * ((double)((n + P - 1) / P) + 2.0) * round;
            if (least != 0.0 && us >= least) continue;
            least = us;
            best.tj = t;
            best.parts = (int)P;
            best.threads = threads;
            best.whole = whole;
            best.nstage = (int)std::min<size_t>(budget / stage - 1, 8);
            best.smem = DF_HDR + (size_t)(best.nstage + 1) * stage;
            best.items = (int)(ntiles * P);
            best.grid = (unsigned)std::min<long long>(best.items, slots);
        }
    }
    return least > 0.0;
}

}  // namespace

/* Whether a run's plain expanding steps take this kernel: double from 128^3,
 * float beyond 256^3. Below, a step is a few short rounds and the staged
 * kernel's two blocks per SM start faster. us per step, staged -> here, double:
 * 96^3 12.4 -> 12.9, 112^3 16.0 -> 17.4, 128^3 19.7 -> 18.9, 192^3 52.4 -> 45.7,
 * 256^3 117 -> 94, 320^3 256 -> 196, 400^3 445 -> 371; float: 192^3 27.1 -> 28.3,
 * 256^3 51.7 -> 51.0 to 52.6, 264^3 68.5 -> 58.7, 320^3 118 -> 101, 400^3 211 ->
 * 173. */
bool step3df_applies(const StepConst &k, int prec) {
    PlanDF p;
    return k.n >= (prec == P_FP64 ? 128 : 257) && plan_df(k, prec, p);
}

size_t step3df_partial_rows(const StepConst &k, int prec) {
    PlanDF p;
    return plan_df(k, prec, p) ? 2 * (size_t)p.items : 0;
}

cudaError_t launch_step3_df(int prec, const StepConst &k, int nsteps, bool cooperative, void *phi_a, void *pi_a,
                            void *phi_b, void *pi_b, DevState *st, double *partials, cudaStream_t s) {
    PlanDF p;
    if (nsteps < 1 || (nsteps > 1 && !cooperative) || !plan_df(k, prec, p)) return cudaErrorNotSupported;
    /* many steps per launch only where a step is one item per block: with several the
     * launch between steps costs less than the blocks waiting for the last one */
    if (cooperative && (unsigned)p.items > p.grid) return cudaErrorNotSupported;
    /* what a step reads is not read again: while its outputs then fit the L2 for the
     * most part (four fields within 2.5 times its 126 MB) let them stay there */
    const size_t fields = 4 * field_elems(k) * (prec == P_FP64 ? 8 : 4);
    const int keep = fields <= (size_t)320 << 20 ? 1 : 0;
    auto go = [&](auto t, auto by, auto eg, auto ms, auto wh) -> cudaError_t {
        using T = decltype(t);
        auto fn = k_step3_df<T, decltype(by)::value, decltype(eg)::value, decltype(ms)::value, decltype(wh)::value>;
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem);
        if (e != cudaSuccess) return e;
        if (!decltype(ms)::value)
            return launch_pdl(fn, dim3(p.grid), dim3(p.threads), p.smem, s, k, p.tj, p.nstage, p.parts, 1, keep,
                              (const T *)phi_a, (const T *)pi_a, (T *)phi_b, (T *)pi_b, st, partials);
        int per_sm = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, p.threads, p.smem);
        if (e != cudaSuccess) return e;
        if ((long long)per_sm * sm_count() < (long long)p.grid) return cudaErrorNotSupported;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(p.grid);
        cfg.blockDim = dim3(p.threads);
        cfg.dynamicSmemBytes = p.smem;
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, fn, k, p.tj, p.nstage, p.parts, nsteps, keep, (const T *)phi_a,
                                  (const T *)pi_a, (T *)phi_b, (T *)pi_b, st, partials);
    };
    using Yes = std::true_type;
    using No = std::false_type;
    using std::integral_constant;
    auto with_form = [&](auto t, auto by, auto eg, auto ms) {
        return p.whole              ? go(t, by, eg, ms, integral_constant<int, 0>{})
               : k.pitch == k.n     ? go(t, by, eg, ms, integral_constant<int, 1>{})
                                    : go(t, by, eg, ms, integral_constant<int, 2>{});
    };
    auto with_ms = [&](auto t, auto by, auto eg) {
        return cooperative ? with_form(t, by, eg, Yes{}) : with_form(t, by, eg, No{});
    };
    auto with_eg = [&](auto t, auto by) { return k.alpha == 1 ? with_ms(t, by, Yes{}) : with_ms(t, by, No{}); };
    if (prec != P_FP64) return with_eg(0.f, integral_constant<int, BY_MUL>{});
    return k.dx2_pow2   ? with_eg(0.0, integral_constant<int, BY_MUL>{})
           : k.dx2_pair ? with_eg(0.0, integral_constant<int, BY_PAIR>{})
                        : with_eg(0.0, integral_constant<int, BY_DIV>{});
}

}  // namespace cb
