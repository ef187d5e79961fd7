/* cb_internal.h -- structures shared by the host glue and the CUDA kernels. */
#ifndef CB_INTERNAL_H
#define CB_INTERNAL_H

#include <cstddef>
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

namespace cb {

/* Per-site sums accumulated by the step kernel (factor dxLD applied at the end). */
enum SumIdx {
    S_EK = 0,   /* sum 0.5 a_kin^(-2d) pi_{n+1/2}^2     (bubble.cpp:810) */
    S_EP,       /* sum V(phi_n)                          (808) */
    S_EG,       /* sum 0.5 |grad_+ phi_n / (a dx)|^2     (794-807) */
    S_PHI,      /* sum phi_n                             (816) */
    S_V,        /* sum pi_{n+1/2} a_kin^(-d)             (817) */
    Q_EK,       /* sums of squares for the spreads       (820-825) */
    Q_EP,
    Q_EG,
    Q_ET,
    Q_PHI,
    Q_V,
    S_EKIN_IN,  /* static background: sum 0.5 pi_{n-1/2}^2, the previous step's raw kinetic sum */
    NSUM
};

/* Background state on the device. The last block of each step kernel that
 * measures sums rewrites it (Friedmann update, bubble.cpp:858-875), so
 * consecutive launches on one stream chain without the host. */
struct DevState {
    /* background at the start of the next step */
    double a, ap, H, C;
    double ekin_half_prev;
    /* coefficients the next step uses */
    double fl;       /* a^(d-2+alpha)                (bubble.cpp:740) */
    double fv;       /* a^(d+alpha)                  (741) */
    double a_kin;    /* a + dt/2 a'                  (765) */
    double kin_w;    /* 0.5 a_kin^(-2d)              (810) */
    double vel_w;    /* a_kin^(-d)                   (817) */
    double adx;      /* a dx                         (794) */
    double inv_adx;
    double drift_p;  /* pending drift factor a_half^(-d+alpha) (870); 0: none pending */
    int adx_pow2;    /* a dx is a power of two: multiplying by 1/(a dx) is exact */
    int pad0;
    /* the last measured line (sums times dxLD; *_var = sums of squares times dxLD^2) */
    double etot, ekin, egrad, epot;
    double etot_var, ekin_var, egrad_var, epot_var;
    double avphi, avphi_var, avphip, avphip_var;
    /* checks of the last measured line: equation of state, energy drift against
     * etot0 (the t = 0 total energy; 0 until known), C / H^2 */
    double w, etot_drift, c_rel, etot0;
    /* last-block-done ticket and error word */
    unsigned int counter;
    int err;
    /* work queue of the staged d = 3 step: next item, and blocks finished
     * (the last block to finish sets both back to zero for the next launch) */
    unsigned int item_next;
    unsigned int item_done;
    /* steps counted done by the blocks of a multi-step launch (reset at its end) */
    unsigned int step_bar;
    unsigned int pad1;
};

/* Constants of one run, passed by value to every launch.
 * Its size decides what a launch costs the host: with the bytes of all arguments
 * at 24 or 32 beyond a multiple of 64 a launch takes 1.9 us, else 2.2 to 2.3
 * (216 to 416 bytes tried, every 8). The 1-D and 2-D kernels, whose calls the host
 * paces, add 72 or 80 bytes of their own (a call of one plain step: 3.4 us with 304
 * bytes in all, 2.9 with 280). */
struct StepConst {
    int d, n;
    int ni, nj, nk;     /* extents mapped onto (march axis, tile rows, tile columns) */
    int cz;             /* planes per block along the march axis (generic d = 3 kernel) */
    double dt;
    double c2, c3, c4;  /* V'(f) = c2 f - c3 f^2 + c4 f^3, coefficients as bubble.cpp:76 forms them */
    double v2, v3, v4, dv; /* V(f) = v2 f^2 - v3 f^3 + v4 f^4 + DeltaV (bubble.cpp:71) */
    /* the same coefficients rounded to float once on the host, so float kernels
     * read them straight from the parameter bank instead of converting per site */
    float c2f, c3f, c4f, v2f, v3f, v4f, dvf;
    float dtf;
    int odd;            /* the step's index is odd: expanding steps march the planes in turn forwards and
                           backwards */
    float dx2f, inv_dx2f;
    int want_local;
    double dx, dx2;
    double inv_dx2;     /* 1/dx2, rounded (dx2_pair: down) */
    int dx2_pow2;
    int dx2_pair;       /* fma(x, inv_dx2, x inv_dx2_lo) is x / dx2 rounded (reciprocal_pair, cb_api.cpp) */
    double dxLD, mpl;
    int alpha, expanding;
    short force_generic;  /* 1: always use the generic tile kernel (diagnostics and cross-checks) */
    short temporal;       /* steps per pass of static 3-D lattices (1: one step per launch on every static lattice) */
    int pitch;            /* elements from a row of the last axis to the next: n, or (d = 3 runs) n rounded
                             up to whole 16-byte vectors. The pad holds the periodic images of the row's
                             first sites: every kernel that writes phi or pi keeps them equal. Here, behind
                             what the kernels load in groups of 16 bytes: among those the generic kernel
                             came out with 40 registers instead of 48 (expanding float 48^3 29.0 us per
                             step, here 21.8) */
    double inv_dx2_lo;    /* 1/dx2 - inv_dx2, rounded */
};
static_assert((sizeof(StepConst) + 72) % 64 == 24, "dear to launch");

bool reciprocal_pair(double d, double &zh, double &zl);

/* The checks of one line from its energies, in double and in this order (the
 * step epilogue does the same operations with explicit rounding):
 * w = (Ekin - (d-2)/d Egrad - Epot) / Etot (python/plot_SummaryPlots.py:91-95);
 * drift = Etot / Etot0 - 1 (plot_SummaryPlots.py:80-81), 0 while Etot0 is
 * unknown; C / H^2 when H != 0. Host code (lines assembled on the host). */
struct LineChecks {
    double w, drift, c_rel;
};
inline LineChecks line_checks(int d, double ekin, double egrad, double epot, double etot, double etot0, double H,
                              double C) {
    LineChecks r;
    const double q = (double)(d - 2) / (double)d;
    r.w = (ekin - q * egrad - epot) / etot;
    r.drift = etot0 != 0.0 ? etot / etot0 - 1.0 : 0.0;
    r.c_rel = H != 0.0 ? C / (H * H) : 0.0;
    return r;
}

/* Kernel launchers (cb_step.cu). Each returns the cudaError_t of the launch. */
enum Prec { P_FP64 = 0, P_FP32 = 1 };

/* Which sums a step kernel accumulates (the `sums` argument of the launchers).
 * SUM_FRIEDMANN_EG: the Friedmann sums with the gradient energy (conformal
 * time, alpha = 1); the staged d = 3 kernel takes it as its own variant so
 * the choice is made at compile time. */
/* SUM_LINE: every box average and no local energy arrays -- the staged d = 3
 * kernel's own variant in double, with the sums' terms formed in fewer
 * operations than the arrays' values. */
enum SumMode { SUM_NONE = 0, SUM_FRIEDMANN = 1, SUM_FULL = 2, SUM_FRIEDMANN_EG = 3, SUM_LINE = 4 };

/* sums: 0 none, 1 only what the Friedmann update needs, 2 every box average */
cudaError_t launch_step(int prec, const StepConst &k, bool drift_first, int sums, const void *phi_in,
                        const void *pi_in, void *phi_out, void *pi_out, void *loc_ek, void *loc_eg, void *loc_ep,
                        DevState *st, double *partials, cudaStream_t s);
/* Number of blocks (and so of partial-sum slots) a step launch may use. */
size_t step_blocks(const StepConst &k);

/* d = 2 kernel marching column strips down the rows (cb_step2.cu), also run
 * on the single row of d = 1: static background, n a multiple of the vector
 * width, lattices of at least STEP2_MIN_SITES (d = 2) / STEP1_MIN_SITES
 * (d = 1) sites; below that the generic tile kernel. */
constexpr size_t STEP2_MIN_SITES = size_t(1) << 20;   /* below 1024^2 both are launch-bound; the tiles win at 128^2 */
constexpr size_t STEP1_MIN_SITES = size_t(1) << 20;   /* d = 1: at 2^18 sites the tiles still win (4.5 vs 5.7 us) */
bool step2_applies(const StepConst &k, int prec, bool drift_first);
bool step2_one_strip(const StepConst &k, int prec);   /* and a row is one block's strip */
size_t step2_blocks(const StepConst &k);
cudaError_t launch_step2(int prec, const StepConst &k, int sums, const void *phi_in, const void *pi_in,
                         void *phi_out, void *pi_out, void *le, void *lg, void *lp, DevState *st, double *partials,
                         cudaStream_t s);

/* Several steps per launch on static 1-D and 2-D lattices (cb_step2_tb.cu).
 * step2tb_steps: how many of the next `left` steps one launch takes, the last
 * of the `left` measuring sums or not (0: the one-step kernels). */
int step2tb_steps(const StepConst &k, int prec, int left, bool sums);
cudaError_t launch_step2_tb(int prec, const StepConst &k, int steps, bool sums, const void *phi_in, const void *pi_in,
                            void *phi_out, void *pi_out, DevState *st, double *partials, cudaStream_t s);

/* Many static d = 2 lattices of one precision and kind per launch: steps at a
 * time (batch2_steps of the `left` to come), the last with sums into record
 * `event` of each (< 0: none). flip: which of a member's buffers hold the
 * fields now. ns: the members' n, largest first. partials: as many rows as all
 * members have tiles (batch2_tiles, of a launch of so many steps), a member's
 * from its `row` on. */
struct Batch2Member {
    StepConst k;
    void *phi[2], *pi[2];
    DevState *st, *records;
    int row;
};
int batch2_kind(const StepConst &k, int prec);   /* members of a launch share it: form of the rows, division by dx^2 */
int batch2_steps(const std::vector<int> &ns, int prec, int kind, int left);
int batch2_threads(const std::vector<int> &ns, int prec, int kind, int steps);   /* of a block */
std::vector<int> batch2_tiles(const std::vector<int> &ns, int prec, int kind, int steps);
cudaError_t launch_step2_batch(int prec, int kind, const Batch2Member *members, const std::vector<int> &ns, int steps,
                               int flip, int event, double *partials, cudaStream_t s);

/* d = 3 kernel with TMA-staged row tiles (cb_step3.cu). */
bool step3_geometry(const StepConst &k, int prec, int &tj, int &nstage, size_t &smem, unsigned &grid);
size_t step3_partial_rows(const StepConst &k, int prec);
cudaError_t launch_step3(int prec, const StepConst &k, bool drift_first, int sums, const void *phi_in,
                         const void *pi_in, void *phi_out, void *pi_out, void *loc_ek, void *loc_eg, void *loc_ep,
                         DevState *st, double *partials, cudaStream_t s);
cudaError_t launch_step3_ms(int prec, const StepConst &k, int nsteps, void *phi_a, void *pi_a, void *phi_b,
                            void *pi_b, DevState *st, double *partials, cudaStream_t s);

/* Plain steps of an expanding background (cb_step3_df.cu): one step, or with
 * `cooperative` nsteps >= 1 of them in one launch (A = the fields now, B = the
 * other buffers; the fields end in B for odd nsteps). cudaErrorNotSupported
 * where the kernel does not apply, or its blocks cannot all be resident. */
cudaError_t launch_step3_df(int prec, const StepConst &k, int nsteps, bool cooperative, void *phi_a, void *pi_a,
                            void *phi_b, void *pi_b, DevState *st, double *partials, cudaStream_t s);
bool step3df_applies(const StepConst &k, int prec);
size_t step3df_partial_rows(const StepConst &k, int prec);

/* TL steps per pass, static 3-D lattices (cb_step3_tb.cu). */
bool step3tb_geometry(const StepConst &k, int prec, int tl, int &tj, int &nstage, size_t &smem, unsigned &grid,
                      int &parts);
cudaError_t launch_step3_tb(int prec, const StepConst &k, int tl, const void *phi_in, const void *pi_in,
                            void *phi_out, void *pi_out, DevState *st, cudaStream_t s);

cudaError_t launch_ic_energies(int prec, const StepConst &k, const void *phi, const void *pi, void *loc_ek,
                               void *loc_eg, void *loc_ep, DevState *st, double *partials, cudaStream_t s);
cudaError_t launch_ic_backkick(int prec, const StepConst &k, const void *phi, void *pi, DevState *st,
                               double *partials, cudaStream_t s);
size_t ic_blocks(const StepConst &k);

/* phi_out = phi + (dt * pi) * drift_p; then drift_p = 0 (applies a pending drift). */
cudaError_t launch_flush_drift(int prec, const StepConst &k, const void *phi, const void *pi, void *phi_out,
                               DevState *st, cudaStream_t s);
cudaError_t launch_convert(int from_prec, int to_prec, const void *src, void *dst, size_t n, cudaStream_t s);
/* `rows` rows of n elements between a field's rows (k.pitch apart) and dense
 * ones, converted on the way; a padded destination gets its images */
cudaError_t launch_repitch(int from_prec, int to_prec, const void *src, size_t src_pitch, void *dst, size_t dst_pitch,
                           int n, size_t rows, cudaStream_t s);
/* elements of a field's buffer, pads included */
inline size_t field_elems(const StepConst &k) {
    size_t e = (size_t)k.pitch;
    for (int i = 1; i < k.d; ++i) e *= (size_t)k.n;
    return e;
}
/* Rows of n elements in tiles of t rows on the marching kernels, two vectors a thread (u and
 * u + half the tile's): whether every warp's vectors are consecutive in one row, all tiles are
 * whole, and both vectors of a thread start at the same site of their rows -- half a tile is
 * then whole rows, so t is even. One set of row-end offsets serves both. */
inline bool whole_rows(int n, int pitch, int prec, int t) {
    const int W = prec == 0 ? 2 : 4;
    return pitch == n && n % W == 0 && n / W % 32 == 0 && t % 2 == 0 && n % t == 0;
}
/* a d = 3 run's row pitch: whole 16-byte vectors where the staged kernels apply */
inline int run_pitch(int d, int n, int prec) {
    const int W = prec == 0 ? 2 : 4;
    return d == 3 && n >= 64 ? (n + W - 1) / W * W : n;
}

}  // namespace cb

#endif
