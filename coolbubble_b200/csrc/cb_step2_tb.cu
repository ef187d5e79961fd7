/* cb_step2_tb.cu -- several leapfrog steps per launch on static 1-D and 2-D
 * lattices (Bubble::oneStep, src/bubble.cpp:849-876, for D = 1, 2; these
 * backgrounds never expand, bubble.hpp:77, so between two reported lines no
 * step needs a global sum).
 *
 * Overlapped tiling in registers. A block takes a tile of the lattice with a
 * halo as deep as the number of steps, every thread holds a patch of it -- K
 * rows of one 16-byte vector, phi and pi -- and the block advances the whole
 * tile step by step; only the sites that no tile edge has reached yet are
 * written back. Fields cross memory once per launch instead of once per step.
 *
 *  - d = 2: a warp holds K full rows of a tile (32 vectors wide), the block's
 *    warps lie one below the other. Neighbours along axis 1 come from the
 *    adjacent lanes by shuffle, along axis 0 from the thread's own registers;
 *    only a patch's first and last rows go through shared memory, in two
 *    buffers used in turn, so a step has one barrier.
 *  - A row of 8, 16 or 32 vectors is held whole, on as many lanes: its neighbours
 *    wrap within them and it needs no halo of columns (64^2 float 0.45 -> 0.35 us
 *    per step, 128 such lattices in one launch 2.9 -> 1.4).
 *  - d = 1: a warp holds K vectors of a row of 32 K vectors; a step has no
 *    barrier and no shared memory.
 *  - Coordinates wrap, so tiles that hang over the lattice's end and lattices
 *    smaller than a tile need no special case. n that is no multiple of the
 *    vector width loads and stores site by site (once per launch).
 *  - The last step of a launch may measure the box averages (bubble.cpp:
 *    761-844), in double per thread and across threads, in a fixed order.
 *
 * What bounds it: the arithmetic of the tile, halo included. ncu, 8 steps on
 * 4096^2 floats: FMA pipe 62 % busy (the packed operations occupy it two
 * cycles), DRAM 21 %; 4 steps on 3072^2 doubles: FP64 pipe 60-65 %, DRAM 32 %.
 * us per step, one launch per step -> here: 512^2 double 2.72 -> 1.05, 1000^2
 * float 6.69 -> 1.23, 3072^2 double (dx^2 no power of two) 52.2 -> 24.6,
 * 4096^2 float 47.3 -> 13.4; 4096 sites (d = 1, double) 2.19 -> 0.14.
 *
 * The per-site operations are those of the one-step kernels (cb_step.cu,
 * cb_step2.cu) for a = 1, where a^(d-2) = a^d = 1 and the products with them
 * are exact: fields are identical to theirs bit for bit.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <type_traits>
#include <vector>

#include "cb_internal.h"
#include "cb_launch.cuh"
#include "cb_step_common.cuh"
#include "cb_tma.cuh"

namespace cb {

int sm_count();

namespace {

constexpr int TB2_MAXW = 16;    /* warps per block at most */

/* constants of the update (a = 1) */
template <typename T>
struct Cst;
template <>
struct Cst<float> {
    F2 idx2, dt, nc2, c3, nc4, m2;
    __device__ __forceinline__ explicit Cst(const StepConst &k)
        : idx2(f2_splat(k.inv_dx2f)), dt(f2_splat(k.dtf)), nc2(f2_splat(-k.c2f)), c3(f2_splat(k.c3f)),
          nc4(f2_splat(-k.c4f)), m2(f2_splat(-2.f)) {}
};
template <>
struct Cst<double> {
    const StepConst &k;
    __device__ __forceinline__ explicit Cst(const StepConst &kk) : k(kk) {}
};

/* One packed pair: the force with the periodic Laplacian and V'(phi) (the
 * exact negation of the one-step kernel's rounded V'/phi), kick and drift. */
template <int D>
__device__ __forceinline__ void pair2(const Cst<float> &K, F2 cc, F2 um, F2 up, F2 km, F2 kp, F2 &pi, F2 &phi) {
    /* x - 2 c in one rounding: 2 c is exact */
    F2 lap = f2_add(f2_fma(cc, K.m2, kp), km);
    if (D == 2) lap = f2_add(f2_add(f2_fma(cc, K.m2, up), um), lap);
    const F2 nh = f2_fma(cc, f2_fma(cc, K.nc4, K.c3), K.nc2);
    const F2 force = f2_fma(lap, K.idx2, f2_mul(cc, nh));
    pi = f2_fma(K.dt, force, pi);
    phi = f2_fma(K.dt, pi, cc);
}

/* One vector of one step: c its sites, um / up the vectors one row before and
 * after along axis 0 (d = 2), l / r the sites beside it; pi advances in place. */
template <int D, int BY>
__device__ __forceinline__ float4 update(const Cst<float> &K, const float4 &c, const float4 &um, const float4 &up,
                                         float l, float r, float4 &p) {
    const F2 mid = f2_pack(c.y, c.z);
    F2 pa = f2_pack(p.x, p.y), pb = f2_pack(p.z, p.w), fa, fb;
    pair2<D>(K, f2_pack(c.x, c.y), f2_pack(um.x, um.y), f2_pack(up.x, up.y), f2_pack(l, c.x), mid, pa, fa);
    pair2<D>(K, f2_pack(c.z, c.w), f2_pack(um.z, um.w), f2_pack(up.z, up.w), mid, f2_pack(c.w, r), pb, fb);
    p = make_float4(f2_lo(pa), f2_hi(pa), f2_lo(pb), f2_hi(pb));
    return make_float4(f2_lo(fa), f2_hi(fa), f2_lo(fb), f2_hi(fb));
}
template <int D, int BY>
__device__ __forceinline__ double site(const StepConst &k, double c, double um, double up, double l, double r,
                                       double &p) {
    using A = Ar<double>;
    /* x - 2 c in one rounding: 2 c is exact */
    const double tk = A::add(__fma_rn(c, -2.0, r), l);
    const double lap = D == 2 ? A::add(A::add(__fma_rn(c, -2.0, up), um), tk) : tk;
    p = A::add(p, A::mul(k.dt, A::sub(over_dx2<BY>(k, lap), dV<double>(k, c))));
    return A::add(c, A::mul(k.dt, p));
}
template <int D, int BY>
__device__ __forceinline__ double2 update(const Cst<double> &K, const double2 &c, const double2 &um,
                                          const double2 &up, double l, double r, double2 &p) {
    double2 f;
    f.x = site<D, BY>(K.k, c.x, um.x, up.x, l, c.y, p.x);
    f.y = site<D, BY>(K.k, c.y, um.y, up.y, c.x, r, p.y);
    return f;
}

/* The box sums of one vector (the one-step kernels' expressions); pn: pi after
 * the kick, po: before it. */
template <typename T, int D>
struct Measure {
    using A = Ar<T>;
    using V = typename Vec<T>::V;
    T kin_w, vel_w, adx, inv_adx;
    bool mul;   /* multiply by 1 / (a dx): float, or exact */
    __device__ __forceinline__ T grad(T x) const { return mul ? A::mul(x, inv_adx) : A::div(x, adx); }
    __device__ __forceinline__ void add(const StepConst &k, const V &c, const V &dn, T right, const V &pn, const V &po,
                                        bool whole, int valid, double (&acc)[NSUM]) const {
        constexpr int W = Vec<T>::W;
#pragma unroll
        for (int s = 0; s < W; ++s) {
            if (!whole && s >= valid) break;
            const T cur = Vec<T>::get(c, s);
            const T gx = grad(A::sub(s == W - 1 ? right : Vec<T>::get(c, s < W - 1 ? s + 1 : s), cur));
            const T gy = D == 2 ? grad(A::sub(Vec<T>::get(dn, s), cur)) : (T)0;
            const T gz = (T)0;
            const T eg = A::mul((T)0.5, A::add(A::add(A::sq(gx), A::sq(gy)), A::sq(gz)));
            const T ep = Vpot<T>(k, cur);
            const T pin = Vec<T>::get(pn, s), pio = Vec<T>::get(po, s);
            const T ek = A::mul(A::mul(kin_w, pin), pin);
            const T v = A::mul(pin, vel_w);
            const T et = A::add(A::add(ek, eg), ep);
            auto put = [&](int i, T x) { acc[i] = __dadd_rn(acc[i], (double)x); };
            put(S_EK, ek);
            put(S_EP, ep);
            put(S_EG, eg);
            put(S_PHI, cur);
            put(S_V, v);
            put(Q_EK, A::sq(ek));
            put(Q_EP, A::sq(ep));
            put(Q_EG, A::sq(eg));
            put(Q_ET, A::sq(et));
            put(Q_PHI, A::sq(cur));
            put(Q_V, A::sq(v));
            put(S_EKIN_IN, A::mul(A::mul(kin_w, pio), pio));
        }
    }
};

template <int B>
__device__ __forceinline__ void cp_async(uint32_t to, const void *from) {
    if constexpr (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(to), "l"(from), "n"(B) : "memory");
}

/* tx x ty: the sites a tile writes (columns x rows), hx its column halo (a
 * multiple of the vector width, at least `steps`), tiles_x x tiles_y tiles. */
struct Tiles {
    int tx, ty, hx, tiles_x, tiles;
};

/* How a row of a tile lies on the lanes: 32 vectors loaded site by site (n no
 * multiple of the vector) or as vectors, with a halo of columns; or the
 * lattice's whole row on 8, 16 or 32 lanes, which needs none. */
enum { BY_SITE = 0, VECTORS = 1, WHOLE_ROWS = 2 };

/* A thread's place in a tile: column of vector r, and row of it, counted from
 * the first site the tile (d = 1: the warp's part of it) writes. */
template <int W, int K, int D>
struct Place {
    int lane, w, hx, steps;   /* lane and number of the thread's (part of a) warp */
    __device__ __forceinline__ int col(int r) const { return (lane + (D == 1 ? 32 * r : 0)) * W - hx; }
    __device__ __forceinline__ int row(int r) const { return D == 1 ? 0 : w * K + r - steps; }
};

/* The steps of one tile whose patch the threads hold, and its sites written
 * back; edge: the block's shared rows, two buffers used in turn (buf). With
 * SUMS the last step's terms enter acc. */
template <typename T, int D, int K, int FORM, int BY, bool SUMS>
__device__ __forceinline__ void run_tile(const StepConst &k, const Cst<T> &C, const Tiles &g, int steps, int x0, int y0,
                                         typename Vec<T>::V (&phi)[K], typename Vec<T>::V (&pi)[K],
                                         typename Vec<T>::V *edge, int &buf, const Measure<T, D> &M,
                                         double (&acc)[NSUM], T *__restrict__ phi_out, T *__restrict__ pi_out) {
    using VV = Vec<T>;
    using V = typename VV::V;
    constexpr int W = VV::W;
    constexpr bool ALIGNED = FORM != BY_SITE;
    const int n = k.n, lanes = FORM == WHOLE_ROWS ? n / W : 32;   /* of a row of a tile */
    const int lane = (int)threadIdx.x % lanes, w = (int)threadIdx.x / lanes, nw = (int)blockDim.x / lanes;
    const Place<W, K, D> at{lane, w, g.hx, steps};
    /* WHOLE_ROWS: a row's neighbours wrap within its lanes */
    const int base_lane = (int)(threadIdx.x & 31) - lane;
    const int from_l = base_lane + (lane == 0 ? lanes - 1 : lane - 1), from_r = base_lane + (lane + 1 == lanes ? 0 : lane + 1);
    auto col = [&](int r) { return at.col(r); };
    auto row = [&](int r) { return at.row(r); };
    /* sites of vector r that this tile writes: none, or the first `valid` */
    auto valid_of = [&](int r) -> int {
        const int c = col(r), y = row(r);
        if (c < 0 || c >= g.tx || (D == 2 && (y < 0 || y >= g.ty || y0 + y >= n))) return 0;
        return min(W, n - (x0 + c));
    };
    auto step = [&](auto measure) {
        constexpr bool MEASURE = decltype(measure)::value;
        V prev = phi[0], below = phi[K - 1];
        if (D == 2) {
            V *const e = edge + buf * (2 * lanes * nw);
            buf ^= 1;
            e[(2 * w) * lanes + lane] = phi[0];
            e[(2 * w + 1) * lanes + lane] = phi[K - 1];
            __syncthreads();
            if (w > 0) prev = e[(2 * w - 1) * lanes + lane];
            if (w + 1 < nw) below = e[(2 * w + 2) * lanes + lane];
        }
        T last = VV::get(phi[0], W - 1);   /* d = 1: the last site of the row's previous vector */
#pragma unroll
        for (int r = 0; r < K; ++r) {
            const V cur = phi[r];
            const V next = r < K - 1 ? phi[r < K - 1 ? r + 1 : r] : below;
            T left = FORM == WHOLE_ROWS ? __shfl_sync(0xffffffffu, VV::get(cur, W - 1), from_l)
                                        : __shfl_up_sync(0xffffffffu, VV::get(cur, W - 1), 1);
            T right = FORM == WHOLE_ROWS ? __shfl_sync(0xffffffffu, VV::get(cur, 0), from_r)
                                         : __shfl_down_sync(0xffffffffu, VV::get(cur, 0), 1);
            if (D == 1) {
                const T before = __shfl_sync(0xffffffffu, last, 31);
                const T after = __shfl_sync(0xffffffffu, VV::get(next, 0), 0);
                if (lane == 0) left = before;
                if (lane == 31) right = after;
                last = VV::get(cur, W - 1);
            }
            const V before_kick = pi[r];
            phi[r] = update<D, BY>(C, cur, prev, next, left, right, pi[r]);
            if (MEASURE) {
                const int valid = valid_of(r);
                if (valid > 0) M.add(k, cur, next, right, pi[r], before_kick, ALIGNED, valid, acc);
            }
            prev = cur;
        }
    };
    const int plain = SUMS ? steps - 1 : steps;
    for (int s = 0; s < plain; ++s) step(std::false_type{});
    if (SUMS) step(std::true_type{});
#pragma unroll
    for (int r = 0; r < K; ++r) {
        const int valid = valid_of(r);
        if (valid <= 0) continue;
        const size_t o = (size_t)(y0 + row(r)) * n + x0 + col(r);
        if (ALIGNED) {
            *reinterpret_cast<V *>(phi_out + o) = phi[r];
            *reinterpret_cast<V *>(pi_out + o) = pi[r];
        } else {
#pragma unroll
            for (int s = 0; s < W; ++s)
                if (s < valid) {
                    phi_out[o + s] = VV::get(phi[r], s);
                    pi_out[o + s] = VV::get(pi[r], s);
                }
        }
    }
}

/* A block's sums: its row of partial sums (row of nrows), then, in the block
 * that finishes last, the total -- warps by shuffle, warps in order, rows in a
 * fixed order -- and the step's line; rec (may be NULL) receives the record. */
__device__ void finish_sums(const StepConst &k, double (&acc)[NSUM], DevState *st, double *partials, unsigned row,
                            unsigned nrows, DevState *rec) {
    __shared__ double red[TB2_MAXW][NSUM];
    __shared__ double tot[NSUM];
    __shared__ bool is_last;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int s = 0; s < NSUM; ++s) {
        double x = acc[s];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x = __dadd_rn(x, __shfl_down_sync(0xffffffffu, x, o));
        if (lane == 0) red[w][s] = x;
    }
    __syncthreads();
    if (threadIdx.x < NSUM) {
        double x = 0.0;
        for (int i = 0; i < nw; ++i) x = __dadd_rn(x, red[i][threadIdx.x]);
        partials[(size_t)row * NSUM + threadIdx.x] = x;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        is_last = atomicAdd(&st->counter, 1u) == nrows - 1;
        if (is_last) st->counter = 0u;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    /* warp w adds sums w, w + nw, ...: lane l the rows l, l + 32, ... */
    for (int s = w; s < NSUM; s += nw) {
        double x = 0.0;
        for (unsigned b = lane; b < nrows; b += 32) x = __dadd_rn(x, __ldcg(partials + (size_t)b * NSUM + s));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x = __dadd_rn(x, __shfl_down_sync(0xffffffffu, x, o));
        if (lane == 0) tot[s] = x;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        epilogue(k, st, tot, true, true, lane);
        if (rec && lane == 0) *rec = *st;   /* lane 0 wrote it */
    }
}

/* The measured values' scales, from the run's record. */
template <typename T, int D>
__device__ __forceinline__ Measure<T, D> measure_of(const DevState *st) {
    Measure<T, D> M;
    M.kin_w = (T)st->kin_w;
    M.vel_w = (T)st->vel_w;
    M.adx = (T)st->adx;
    M.inv_adx = (T)st->inv_adx;
    M.mul = std::is_same<T, float>::value || st->adx_pow2 != 0;
    return M;
}

template <typename T, int D, int K, int FORM, int BY, bool SUMS>
__global__ void __launch_bounds__(TB2_MAXW * 32, 1)
    k_step2_tb(StepConst k, Tiles g, int steps, const T *__restrict__ phi_in, const T *__restrict__ pi_in,
               T *__restrict__ phi_out, T *__restrict__ pi_out, DevState *st, double *partials) {
    using VV = Vec<T>;
    using V = typename VV::V;
    constexpr int W = VV::W;
    /* first and last rows of every warp's patch, two buffers */
    extern __shared__ __align__(16) unsigned char smraw[];
    V *const edge = reinterpret_cast<V *>(smraw);
    constexpr bool ALIGNED = FORM != BY_SITE;
    const int n = k.n, lanes = FORM == WHOLE_ROWS ? n / W : 32;
    const int lane = (int)threadIdx.x % lanes, w = (int)threadIdx.x / lanes, nw = (int)blockDim.x >> 5;
    const Cst<T> C(k);
    double acc[NSUM];
    Measure<T, D> M{};
    pdl_wait();   /* the previous launch's fields and device state */
    if (SUMS) {
#pragma unroll
        for (int s = 0; s < NSUM; ++s) acc[s] = 0.0;
        M = measure_of<T, D>(st);
    }
    /* where a tile starts, and this thread's column of vector r and row of it,
     * counted from the first site the tile (d = 1: the warp's part of it) writes */
    auto x_of = [&](int tile) { return (D == 1 ? tile * nw + w : tile % g.tiles_x) * g.tx; };
    auto y_of = [&](int tile) { return D == 1 ? 0 : tile / g.tiles_x * g.ty; };
    auto col = [&](int r) { return (lane + (D == 1 ? 32 * r : 0)) * W - g.hx; };
    auto row = [&](int r) { return D == 1 ? 0 : w * K + r - steps; };
    auto wrap = [&](int i) {
        i %= n;
        return i < 0 ? i + n : i;
    };
    /* each thread copies its own patch of the next tile into its own shared
     * slots while the block computes the current one: no barrier is involved */
    V *const mine = edge + (D == 2 ? 2 * 64 * nw : 0) + threadIdx.x;
    auto fetch = [&](int tile) {
        const int x0 = x_of(tile);
        int c = wrap(x0 + col(0)), y = wrap(y_of(tile) + row(0));
#pragma unroll
        for (int r = 0; r < K; ++r) {
            const size_t base = (size_t)y * n;
            const uint32_t to = smem_u32(mine + 2 * r * blockDim.x), step_b = 16u * blockDim.x;
            if (ALIGNED) {
                cp_async<16>(to, phi_in + base + c);
                cp_async<16>(to + step_b, pi_in + base + c);
            } else {
                int cs = c;
#pragma unroll
                for (int s = 0; s < W; ++s) {
                    cp_async<sizeof(T)>(to + s * sizeof(T), phi_in + base + cs);
                    cp_async<sizeof(T)>(to + step_b + s * sizeof(T), pi_in + base + cs);
                    if (++cs == n) cs = 0;
                }
            }
            if (D == 1) c = wrap(x0 + col(r + 1));
            else if (++y == n) y = 0;
        }
    };
    if ((int)blockIdx.x < g.tiles) fetch(blockIdx.x);
    int buf = 0;   /* the edge rows' buffer of the next step: in turn, over all the block's tiles */
    for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x) {
        /* this thread's patch: column of vector r, and row of it, counted from
         * the first site the tile (d = 1: the warp's part of it) writes */
        const int x0 = x_of(tile), y0 = y_of(tile);
        V phi[K], pi[K];
        asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
        for (int r = 0; r < K; ++r) {
            phi[r] = mine[2 * r * blockDim.x];
            pi[r] = mine[(2 * r + 1) * blockDim.x];
        }
        if (tile + gridDim.x < g.tiles) fetch(tile + gridDim.x);
        run_tile<T, D, K, FORM, BY, SUMS>(k, C, g, steps, x0, y0, phi, pi, edge, buf, M, acc, phi_out, pi_out);
    }
    pdl_allow_next();
    if (SUMS) finish_sums(k, acc, st, partials, blockIdx.x, gridDim.x, nullptr);
}

constexpr size_t BATCH2_MOST = 65535;   /* lattices of a launch: gridDim.y */

/* One launch of `steps` steps over many lattices of one kind (ensembles):
 * block (x, y) takes tile x of lattice y, where it has one. */
template <typename T, int K, int FORM, int BY, bool SUMS>
__global__ void __launch_bounds__(TB2_MAXW * 32, 1)
    k_step2_batch(const Batch2Member *__restrict__ members, Tiles g0, int steps, int flip, int event,
                  double *partials) {
    using VV = Vec<T>;
    using V = typename VV::V;
    constexpr int W = VV::W;
    extern __shared__ __align__(16) unsigned char smraw[];
    V *const edge = reinterpret_cast<V *>(smraw);
    const Batch2Member &mb = members[blockIdx.y];
    const StepConst k = mb.k;
    constexpr bool ALIGNED = FORM != BY_SITE;
    const int n = k.n, lanes = FORM == WHOLE_ROWS ? n / W : 32;
    Tiles g = g0;
    if (FORM == WHOLE_ROWS) {
        g.tx = n;
        g.ty = (int)blockDim.x / lanes * K - 2 * steps;
    }
    g.tiles_x = (n + g.tx - 1) / g.tx;
    g.tiles = g.tiles_x * ((n + g.ty - 1) / g.ty);
    if ((int)blockIdx.x >= g.tiles) return;
    const T *const phi_in = static_cast<const T *>(mb.phi[flip]), *const pi_in = static_cast<const T *>(mb.pi[flip]);
    const Cst<T> C(k);
    double acc[NSUM];
    Measure<T, 2> M{};
    pdl_wait();   /* the previous launch's fields and records */
    if (SUMS) {
#pragma unroll
        for (int s = 0; s < NSUM; ++s) acc[s] = 0.0;
        M = measure_of<T, 2>(mb.st);
    }
    const int x0 = (int)blockIdx.x % g.tiles_x * g.tx, y0 = (int)blockIdx.x / g.tiles_x * g.ty;
    const Place<W, K, 2> at{(int)threadIdx.x % lanes, (int)threadIdx.x / lanes, g.hx, steps};
    auto wrap = [&](int i) {
        i %= n;
        return i < 0 ? i + n : i;
    };
    V phi[K], pi[K];
    const int c = wrap(x0 + at.col(0));
    int y = wrap(y0 + at.row(0));
#pragma unroll
    for (int r = 0; r < K; ++r) {
        const size_t base = (size_t)y * n;
        if (ALIGNED) {
            phi[r] = *reinterpret_cast<const V *>(phi_in + base + c);
            pi[r] = *reinterpret_cast<const V *>(pi_in + base + c);
        } else {
            int cs = c;
#pragma unroll
            for (int s = 0; s < W; ++s) {
                VV::set(phi[r], s, phi_in[base + cs]);
                VV::set(pi[r], s, pi_in[base + cs]);
                if (++cs == n) cs = 0;
            }
        }
        if (++y == n) y = 0;
    }
    int buf = 0;
    run_tile<T, 2, K, FORM, BY, SUMS>(k, C, g, steps, x0, y0, phi, pi, edge, buf, M, acc,
                                         static_cast<T *>(mb.phi[1 - flip]), static_cast<T *>(mb.pi[1 - flip]));
    pdl_allow_next();
    if (SUMS)
        finish_sums(k, acc, mb.st, partials + (size_t)mb.row * NSUM, blockIdx.x, g.tiles, mb.records + event);
}

}  // namespace

namespace {

/* How a launch of `steps` steps tiles the lattice. */
struct Plan2 {
    int rows = 0, warps = 0;   /* K of the patches, warps per block */
    Tiles g{};
    unsigned grid = 0;
    double us = 0.0;           /* modelled time */
};

constexpr int TB2_STEPS = 20;   /* d = 2: steps per launch at most (the halo eats the tile beyond) */

/* d = 2: the patch height and block size whose modelled time is least. A
 * launch costs a start, then per round of resident blocks a load and a store
 * of the rows the busiest SM holds, and per step a latency and an issue time
 * per row (a row: 32 vectors; 8-row patches pay for 128 registers with fewer
 * warps to hide latency). The coefficients, in us, were fitted to 418 timed
 * (n, K, warps, steps) combinations of each precision, n from 64 to 3072:
 * 7 % rms off, and the plan it picks within 6 % of the fastest one timed
 * (9 % at 3072^2 in double). Small lattices so get small blocks on many SMs
 * and few steps per launch, large ones tall tiles whose halo costs less. */
template <class TilesOf>
bool plan_tiles(int prec, int form, int steps, TilesOf &&tiles_of, Plan2 &best) {
    struct Cost { double start, load, load_row, step, row4, row8, wide; };
    static constexpr Cost cost[2] = {{1.60, -0.16, 0.030, 0.120, 0.0079, 0.0100, 0.061},    /* double */
                                     {1.54, 0.11, 0.027, 0.066, 0.0049, 0.0069, 0.088}};    /* float */
    static constexpr int shape[5][2] = {{4, 4}, {4, 8}, {4, 16}, {8, 8}, {8, 16}};
    const Cost &c = cost[prec == P_FP64 ? 0 : 1];
    const int W = prec == P_FP64 ? 2 : 4, sms = sm_count();
    best.us = 0.0;
    for (const auto &s : shape) {
        Plan2 p;
        p.rows = s[0];
        p.warps = s[1];
        p.g.hx = form == WHOLE_ROWS ? 0 : (steps + W - 1) / W * W;
        p.g.tx = 32 * W - 2 * p.g.hx;
        p.g.ty = p.rows * p.warps - 2 * steps;   /* WHOLE_ROWS: of rows of 32 lanes; more of shorter ones */
        if (p.g.tx <= 0) continue;
        const long long tiles = tiles_of(p.g, p.rows * p.warps);
        if (tiles <= 0) continue;
        const int per_sm = TB2_MAXW / p.warps;
        p.g.tiles = (int)tiles;
        p.grid = (unsigned)std::min<long long>(tiles, (long long)sms * per_sm);
        const long long busiest = (tiles + sms - 1) / sms;
        auto round_us = [&](long long blocks) {
            const double rows = (double)blocks * p.rows * p.warps;
            return c.load + c.load_row * rows +
                   steps * (c.step + (p.rows == 4 ? c.row4 : c.row8) * rows + (p.warps == TB2_MAXW ? c.wide : 0.0));
        };
        p.us = c.start + (double)(busiest / per_sm) * round_us(per_sm) +
               (busiest % per_sm ? round_us(busiest % per_sm) : 0.0);
        if (best.us == 0.0 || p.us < best.us) best = p;
    }
    return best.us > 0.0;
}

/* the tiles of one lattice of n^2; h: rows of 32 lanes in a block. 0: none fits. */
long long tiles_of_one(Tiles &g, int n, int W, int form, int steps, int h) {
    if (form == WHOLE_ROWS) {
        g.tx = n;
        g.ty = h * (32 / (n / W)) - 2 * steps;
    }
    if (g.ty <= 0) return 0;
    g.tiles_x = (n + g.tx - 1) / g.tx;
    return (long long)g.tiles_x * ((n + g.ty - 1) / g.ty);
}

int form_of(const StepConst &k, int prec) {
    const int W = prec == P_FP64 ? 2 : 4, nv = k.n / W;
    if (k.n % W != 0) return BY_SITE;
    return k.d == 2 && (nv == 8 || nv == 16 || nv == 32) ? WHOLE_ROWS : VECTORS;
}

bool plan_2d(const StepConst &k, int prec, int steps, Plan2 &p) {
    const int form = form_of(k, prec);
    return plan_tiles(prec, form, steps, [&](Tiles &g, int h) {
        return tiles_of_one(g, k.n, prec == P_FP64 ? 2 : 4, form, steps, h);
    }, p);
}

/* the tiles of lattices of these sizes; each: of every one of them (may be NULL) */
bool plan_batch(const std::vector<int> &ns, int prec, int form, int steps, Plan2 &p, std::vector<int> *each) {
    const int W = prec == P_FP64 ? 2 : 4;
    if (!plan_tiles(prec, form, steps, [&](Tiles &g, int h) -> long long {
            long long all = 0;
            int last = 0;
            long long of_last = 0;
            for (int n : ns) {   /* sorted: equal ones are neighbours */
                if (n != last) {
                    of_last = tiles_of_one(g, n, W, form, steps, h);
                    last = n;
                }
                if (of_last == 0) return 0;
                all += of_last;
            }
            return all <= INT_MAX ? all : 0;
        }, p))
        return false;
    if (each) {
        each->clear();
        for (int n : ns) {
            Tiles g = p.g;
            g.ty = p.rows * p.warps - 2 * steps;
            each->push_back((int)tiles_of_one(g, n, W, form, steps, p.rows * p.warps));
        }
    }
    return true;
}

/* of `left` steps: an even split into launches whose modelled time is least */
template <class Us>
int even_split(int left, Us &&us_of) {
    int steps = 0;
    double least = 0.0;
    for (int t = std::min(left, TB2_STEPS); t >= 1; --t) {
        const int launches = (left + t - 1) / t;
        if ((left + launches - 1) / launches != t) continue;   /* not the even split of its launches */
        const double us = us_of(t);
        if (us <= 0.0) continue;
        if (steps == 0 || launches * us < least) {
            steps = t;
            least = launches * us;
        }
    }
    return steps;
}

/* d = 1: warps are independent, so only the patch length matters: two vectors
 * per thread below 2^18 sites (more warps: 4096 double sites 0.15 us per step,
 * 0.17 with four), four from there on (2^20 floats 0.49 against 0.55 us). */
constexpr int TB1_STEPS = 32;
bool plan_1d(const StepConst &k, int prec, int steps, Plan2 &p) {
    const int W = prec == P_FP64 ? 2 : 4;
    p.rows = k.n < (1 << 18) ? 2 : 4;
    p.warps = 4;
    p.g.hx = (steps + W - 1) / W * W;
    p.g.tx = 32 * W * p.rows - 2 * p.g.hx;
    if (p.g.tx <= 0) return false;
    p.g.ty = 1;
    p.g.tiles_x = (k.n + p.g.tx - 1) / p.g.tx;
    p.g.tiles = (p.g.tiles_x + p.warps - 1) / p.warps;
    p.grid = (unsigned)std::min(p.g.tiles, sm_count() * (TB2_MAXW / p.warps));
    return true;
}

bool plan2(const StepConst &k, int prec, int steps, Plan2 &p) {
    return k.d == 1 ? plan_1d(k, prec, steps, p) : plan_2d(k, prec, steps, p);
}

}  // namespace

/* The steps of the next launch when `left` steps are to come, the last of them
 * with sums or not: launches of nearly equal depth, as many as the modelled
 * time is least for. A single step without sums is left to the one-step
 * kernels (512^2 double: 2.7 us, here 3.1). */
int step2tb_steps(const StepConst &k, int prec, int left, bool sums) {
    if (k.d > 2 || k.force_generic || k.temporal == 1 || left < 1 || (left == 1 && !sums)) return 0;
    if (k.d == 1) {
        /* in double a halo of 32 of 256 sites costs more than a launch from 2^18 sites on */
        const int most = prec == P_FP64 && k.n >= (1 << 18) ? TB1_STEPS / 2 : TB1_STEPS;
        const int launches = (left + most - 1) / most;
        return (left + launches - 1) / launches;
    }
    /* The start and the block-wide sums of a launch here are not earned back by the one
     * step of a small lattice (in us, double: 64^2 9.0, one-step kernel 7.7; 256^2 10.5
     * and 9.5; 320^2 11.2 and 11.3; 512^2 13.9 and 18.0), by two of a very small one
     * (32^2 8.8 and 8.6; 64^2 9.4 and 9.3), nor by one or two where the strips' kernel has
     * one per row (1024^2 float 17.0 and 13.7; calls of two 43.1 and 36.6). Large lattices
     * read their halo for one step only: strips from 4096^2 on in float and where double
     * divides by the compiler's division (calls of one step, float: 3072^2 82.0 here, 81.3
     * in strips; 3584^2 94 and 106; 4096^2 118 and 111; 8192^2 340 and 315; double that
     * divides: 3584^2 153 and 154; 4096^2 191 and 180; 8192^2 638 and 597; other double
     * 8192^2 576 and 597). */
    const bool strip = step2_one_strip(k, prec);
    const bool large = k.n >= 4096 && step2_applies(k, prec, false) && (prec != P_FP64 || !(k.dx2_pow2 || k.dx2_pair));
    if (sums && ((left == 1 && (k.n <= 288 || strip || large)) || (left == 2 && (k.n <= 64 || strip)))) return 0;
    return even_split(left, [&](int t) {
        Plan2 p;
        return plan_2d(k, prec, t, p) ? p.us : 0.0;
    });
}

cudaError_t launch_step2_tb(int prec, const StepConst &k, int steps, bool sums, const void *phi_in, const void *pi_in,
                            void *phi_out, void *pi_out, DevState *st, double *partials, cudaStream_t s) {
    Plan2 p;
    if (steps < 1 || !plan2(k, prec, steps, p)) return cudaErrorInvalidValue;
    /* a block with sums writes a row of partial sums: no more of them than a run's
     * one-step launches have (blocks take several tiles then) */
    if (sums) p.grid = (unsigned)std::min<size_t>(p.grid, step_blocks(k));
    const int form = form_of(k, prec);
    const size_t smem = ((k.d == 2 ? (size_t)2 * 64 * p.warps : 0) + (size_t)2 * p.rows * 32 * p.warps) * 16;
    auto go = [&](auto t, auto d, auto rows, auto al, auto dv, auto su) -> cudaError_t {
        using T = decltype(t);
        auto fn = k_step2_tb<T, decltype(d)::value, decltype(rows)::value, decltype(al)::value, decltype(dv)::value,
                             decltype(su)::value>;
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        return launch_pdl(fn, dim3(p.grid), dim3(p.warps * 32), smem, s, k, p.g, steps, (const T *)phi_in,
                          (const T *)pi_in, (T *)phi_out, (T *)pi_out, st, partials);
    };
    using Yes = std::true_type;
    using No = std::false_type;
    auto with_rows = [&](auto t, auto d, auto al, auto dv, auto su) {
        constexpr int less = decltype(d)::value == 1 ? 2 : 8;   /* d = 1: 2 or 4, d = 2: 4 or 8 */
        return p.rows == 4 ? go(t, d, std::integral_constant<int, 4>{}, al, dv, su)
                           : go(t, d, std::integral_constant<int, less>{}, al, dv, su);
    };
    auto with_sums = [&](auto t, auto d, auto al, auto dv) {
        return sums ? with_rows(t, d, al, dv, Yes{}) : with_rows(t, d, al, dv, No{});
    };
    auto with_al = [&](auto t, auto d, auto dv) {
        if constexpr (decltype(d)::value == 2)
            if (form == WHOLE_ROWS) return with_sums(t, d, std::integral_constant<int, WHOLE_ROWS>{}, dv);
        return form == BY_SITE ? with_sums(t, d, std::integral_constant<int, BY_SITE>{}, dv)
                               : with_sums(t, d, std::integral_constant<int, VECTORS>{}, dv);
    };
    auto with_t = [&](auto d) {
        using std::integral_constant;
        if (prec != P_FP64) return with_al(0.f, d, integral_constant<int, BY_MUL>{});
        if (k.dx2_pow2) return with_al(0.0, d, integral_constant<int, BY_MUL>{});
        return k.dx2_pair ? with_al(0.0, d, integral_constant<int, BY_PAIR>{})
                          : with_al(0.0, d, integral_constant<int, BY_DIV>{});
    };
    return k.d == 1 ? with_t(std::integral_constant<int, 1>{}) : with_t(std::integral_constant<int, 2>{});
}

int batch2_steps(const std::vector<int> &ns, int prec, int kind, int left) {
    return even_split(left, [&](int t) {
        Plan2 p;
        return plan_batch(ns, prec, kind % 3, t, p, nullptr) ? p.us : 0.0;
    });
}

std::vector<int> batch2_tiles(const std::vector<int> &ns, int prec, int kind, int steps) {
    Plan2 p;
    std::vector<int> each;
    plan_batch(ns, prec, kind % 3, steps, p, &each);
    return each;
}

int batch2_threads(const std::vector<int> &ns, int prec, int kind, int steps) {
    Plan2 p;
    return plan_batch(ns, prec, kind % 3, steps, p, nullptr) ? p.warps * 32 : 0;
}

int batch2_kind(const StepConst &k, int prec) {
    const int by = prec != P_FP64 || k.dx2_pow2 ? BY_MUL : k.dx2_pair ? BY_PAIR : BY_DIV;
    return by * 3 + form_of(k, prec);
}

cudaError_t launch_step2_batch(int prec, int kind, const Batch2Member *members, const std::vector<int> &ns, int steps,
                               int flip, int event, double *partials, cudaStream_t s) {
    Plan2 p;
    std::vector<int> tiles;
    if (steps < 1 || ns.empty() || !plan_batch(ns, prec, kind % 3, steps, p, &tiles)) return cudaErrorInvalidValue;
    const size_t smem = (size_t)2 * 64 * p.warps * 16;
    auto go = [&](auto t, auto rows, auto al, auto dv, auto su) -> cudaError_t {
        using T = decltype(t);
        auto fn = k_step2_batch<T, decltype(rows)::value, decltype(al)::value, decltype(dv)::value, decltype(su)::value>;
        /* a grid has at most 65535 lattices; the first of each is its largest */
        for (size_t at = 0; at < ns.size(); at += BATCH2_MOST) {
            const unsigned count = (unsigned)std::min(ns.size() - at, BATCH2_MOST);
            const cudaError_t e = launch_pdl(fn, dim3((unsigned)tiles[at], count), dim3(p.warps * 32), smem, s,
                                             members + at, p.g, steps, flip, event, partials);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    };
    using std::integral_constant;
    using Yes = std::true_type;
    using No = std::false_type;
    auto with_rows = [&](auto t, auto al, auto dv, auto su) {
        return p.rows == 4 ? go(t, integral_constant<int, 4>{}, al, dv, su) : go(t, integral_constant<int, 8>{}, al, dv, su);
    };
    auto with_sums = [&](auto t, auto al, auto dv) {
        return event >= 0 ? with_rows(t, al, dv, Yes{}) : with_rows(t, al, dv, No{});
    };
    auto with_al = [&](auto t, auto dv) {
        switch (kind % 3) {
            case BY_SITE: return with_sums(t, integral_constant<int, BY_SITE>{}, dv);
            case VECTORS: return with_sums(t, integral_constant<int, VECTORS>{}, dv);
            default: return with_sums(t, integral_constant<int, WHOLE_ROWS>{}, dv);
        }
    };
    if (prec != P_FP64) return with_al(0.f, integral_constant<int, BY_MUL>{});
    switch (kind / 3) {
        case BY_MUL: return with_al(0.0, integral_constant<int, BY_MUL>{});
        case BY_PAIR: return with_al(0.0, integral_constant<int, BY_PAIR>{});
        default: return with_al(0.0, integral_constant<int, BY_DIV>{});
    }
}

}  // namespace cb
