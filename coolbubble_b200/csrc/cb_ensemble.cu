/* cb_ensemble.cu -- many independent lattices advanced together.
 *
 * The reference evolves one lattice per process (its run parameters are
 * process globals, main.cpp:45-50). An ensemble here is a set of runs
 * (cb_handle) stepped together: thermal-fluctuation ensembles and parameter
 * scans of different n, c and start.
 *
 * Two-dimensional static members are stepped in batches: one launch advances
 * every lattice of a precision by several steps (cb_step2_tb.cu, tiles with
 * halos in registers), tile by tile, so a mix of sizes fills the GPU like one
 * large lattice, and fields cross memory once per several steps. The lines of
 * an event are measured by the last step of a launch and each member's step
 * record is kept on the device until the call ends. 48 lattices of 128^2,
 * 256^2 and 512^2 in float, 400 steps: 2.1 ms (5.2 with every lattice held in
 * the shared memory of a cluster, whose barrier per step and issue rate set
 * 3.2 us per step and lattice), with lines every 40 steps 3.2 (6.6); 128 of
 * 64^2 1.4 us per step (2.1), 64 of 256^2 4.6 (6.7).
 *
 * Other members (d = 1, 3, large lattices, a static background that did not start at a = 1)
 * are stepped by their own handles on their own streams, concurrently.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "cb_handle.h"

using namespace cb;

struct cb_ensemble {
    std::vector<cb_handle *> members;
    /* members of one precision and kind, stepped by the same launches */
    struct Batch {
        int prec = 0, kind = 0;
        std::vector<int> idx, ns;      /* member indices, largest lattices first, and their n */
        Batch2Member *dev = nullptr;   /* device array */
        double *partials = nullptr;    /* partial sums, `rows` rows */
        size_t rows = 0;
        cudaStream_t stream = nullptr;
        int launches = 0;              /* of the running call */
        /* the plan, which only the members' sizes decide: steps of the next launch by the
         * steps left of an interval, and every member's tiles in launches of tiles_of steps */
        std::map<int, int> cut;
        std::vector<int> tiles;
        int tiles_of = 0;
        int next(int left) {
            if (left > 1024) return batch2_steps(ns, prec, kind, left);   /* the plan kept stays small */
            int &t = cut[left];
            if (t == 0) t = batch2_steps(ns, prec, kind, left);
            return t;
        }
    };
    std::vector<Batch> batches;
    std::vector<int> own;              /* members stepped by their own handles */
    DevState *records = nullptr;       /* the lines' step records of a call, member by member */
    size_t records_cap = 0;
};

namespace {

/* The size class of a 2-D lattice: how many 200 KB shares (1, 2, 4, 8, 16)
 * three of its fields fill in whole rows; 0 beyond, or for other rows. A way for
 * callers to tell sizes apart; no launch depends on it. */
int size_class(int prec, int d, int n) {
    const size_t esz = prec == P_FP64 ? 8 : 4;
    if (d != 2 || n % (16 / esz) != 0) return 0;
    for (int cs = 1; cs <= 16; cs *= 2) {
        if (n % cs != 0) return 0;
        if (3 * (size_t)(n / cs) * n * esz <= 200 * 1024) return cs;
    }
    return 0;
}

constexpr int LONG_INTERVAL = 64;   /* steps whose launches cb_ensemble_member_plan speaks of */

/* Members stepped in batches. A large lattice fills the GPU by itself, and its own
 * launches choose kernel and depth for it alone: in double from 2048^2 on, in float
 * from 3072^2 (one member, us in a batch and on its own stream; ten steps with a line
 * each: double 1448^2 491 and 400, 2048^2 752 and 464, 8192^2 9472 and 4560, float
 * 2048^2 524 and 370, 3072^2 738 and 670, 8192^2 5388 and 2974; 40 steps and one line:
 * double 2048^2 547 and 499, float 2048^2 214 and 214; 40 plain steps: double 2048^2
 * 488 and 466, float 2048^2 170 and 180, 3072^2 347 and 347). */
bool batched(const cb_handle *h) {
    const int most = h->prec == P_FP64 ? 2048 : 3072;
    return h->p.d == 2 && h->p.n_grids < most && h->unit_scale && !h->k.force_generic && h->k.temporal != 1;
}

cudaError_t grow_partials(cb_ensemble::Batch &b, size_t rows) {
    if (rows <= b.rows) return cudaSuccess;
    if (b.partials) cudaFreeAsync(b.partials, b.stream);
    b.partials = nullptr;
    b.rows = 0;
    const cudaError_t e = cudaMallocAsync((void **)&b.partials, rows * NSUM * sizeof(double), b.stream);
    if (e == cudaSuccess) b.rows = rows;
    return e;
}

/* The members' buffers, records of the call and, for launches of `steps` steps
 * with sums (0: none), rows of partial sums to the batch's array. */
cudaError_t upload_members(cb_ensemble *e, cb_ensemble::Batch &b, int nev, int steps) {
    std::vector<Batch2Member> host(b.idx.size());
    size_t rows = 0;
    if (steps > 0 && steps != b.tiles_of) {
        b.tiles = batch2_tiles(b.ns, b.prec, b.kind, steps);
        b.tiles_of = steps;
    }
    if (steps > 0 && b.tiles.empty()) return cudaErrorInvalidValue;
    for (size_t q = 0; q < b.idx.size(); ++q) {
        const cb_handle *h = e->members[b.idx[q]];
        Batch2Member &m = host[q];
        m.k = h->k;
        m.k.want_local = 0;
        for (int i = 0; i < 2; ++i) {   /* [0]: the fields now */
            m.phi[i] = h->phi[i == 0 ? h->cphi : 1 - h->cphi];
            m.pi[i] = h->pi[i == 0 ? h->cpi : 1 - h->cpi];
        }
        m.st = h->st;
        m.records = e->records + (size_t)b.idx[q] * nev;
        m.row = (int)rows;
        if (steps > 0) rows += (size_t)b.tiles[q];
    }
    const cudaError_t err = grow_partials(b, rows);
    if (err != cudaSuccess) return err;
    return cudaMemcpyAsync(b.dev, host.data(), host.size() * sizeof(Batch2Member), cudaMemcpyHostToDevice, b.stream);
}

/* All steps of a call for one batch: intervals of sums_every steps (the last
 * one may be shorter and has no line), each in launches of several steps. */
cudaError_t run_batch(cb_ensemble *e, cb_ensemble::Batch &b, int nsteps, int sums_every, int nev) {
    /* every interval with a line is cut alike, so all launches with sums have the same steps */
    int last = 0;
    for (int left = nev > 0 ? sums_every : 0; left > 0; left -= last)
        if ((last = b.next(left)) < 1) return cudaErrorInvalidValue;
    cudaError_t err = upload_members(e, b, nev, last);
    b.launches = 0;
    for (int done = 0, j = 0; done < nsteps && err == cudaSuccess;) {
        const int span = nev > 0 ? std::min(sums_every, nsteps - done) : nsteps - done;
        const bool line = nev > 0 && span == sums_every && j < nev;
        for (int left = span; left > 0 && err == cudaSuccess;) {
            const int t = b.next(left);
            if (t < 1) return cudaErrorInvalidValue;
            err = launch_step2_batch(b.prec, b.kind, b.dev, b.ns, t, b.launches & 1, line && t == left ? j : -1,
                                     b.partials, b.stream);
            b.launches++;
            left -= t;
        }
        if (line) ++j;
        done += span;
    }
    return err;
}

}  // namespace

extern "C" {

int cb_ensemble_create(int count, cb_handle *const *members, cb_ensemble **out) {
    return cb::guard(nullptr, [&]() -> int {
        if (count < 1 || !members || !out) return fail(nullptr, CB_EINVAL, "cb_ensemble_create: bad arguments");
        *out = nullptr;
        for (int i = 0; i < count; ++i)
            if (!members[i]) return fail(nullptr, CB_EINVAL, "cb_ensemble_create: NULL member");
        cb_ensemble *e = new cb_ensemble();
        e->members.assign(members, members + count);
        std::map<int, int> of;   /* (prec, kind) -> batch */
        std::vector<int> order(count);
        for (int i = 0; i < count; ++i) order[i] = i;
        std::stable_sort(order.begin(), order.end(),
                         [&](int x, int y) { return members[x]->p.n_grids > members[y]->p.n_grids; });
        for (int i : order) {
            cb_handle *h = members[i];
            if (!batched(h)) {
                e->own.push_back(i);
                continue;
            }
            const int kind = batch2_kind(h->k, h->prec), key = kind * 2 + h->prec;
            if (of.find(key) == of.end()) {
                of[key] = (int)e->batches.size();
                e->batches.emplace_back();
                e->batches.back().prec = h->prec;
                e->batches.back().kind = kind;
            }
            cb_ensemble::Batch &b = e->batches[of[key]];
            b.idx.push_back(i);
            b.ns.push_back(h->p.n_grids);
        }
        for (auto &b : e->batches)
            if (cudaStreamCreateWithFlags(&b.stream, cudaStreamNonBlocking) != cudaSuccess ||
                cudaMalloc(&b.dev, b.idx.size() * sizeof(Batch2Member)) != cudaSuccess) {
                cudaGetLastError();
                cb_ensemble_destroy(e);
                return fail(nullptr, CB_ENOMEM, "cb_ensemble_create: device allocation failed");
            }
        *out = e;
        return CB_OK;
    });
}

int cb_ensemble_member_plan(cb_ensemble *e, int m, int *cluster, int *threads) {
    return cb::guard(nullptr, [&]() -> int {
        if (!e || m < 0 || m >= (int)e->members.size() || !cluster || !threads)
            return fail(nullptr, CB_EINVAL, "cb_ensemble_member_plan: bad arguments");
        *cluster = *threads = 0;
        for (auto &b : e->batches)
            if (std::find(b.idx.begin(), b.idx.end(), m) != b.idx.end()) {
                const cb_handle *h = e->members[m];
                *cluster = size_class(h->prec, h->p.d, h->p.n_grids);
                *threads = batch2_threads(b.ns, b.prec, b.kind, b.next(LONG_INTERVAL));
            }
        return CB_OK;
    });
}

int cb_ensemble_destroy(cb_ensemble *e) {
    if (!e) return CB_EINVAL;
    for (auto &b : e->batches) {
        if (b.stream) cudaStreamSynchronize(b.stream);
        if (b.partials) cudaFreeAsync(b.partials, b.stream);
        cudaFree(b.dev);
        if (b.stream) cudaStreamDestroy(b.stream);
    }
    cudaFree(e->records);
    delete e;
    return CB_OK;
}

/* Advance every member nsteps steps. With sums_every > 0, the box averages of
 * every sums_every-th step are written to out[m * (nsteps / sums_every) + j]
 * (member m, event j); out may be NULL when sums_every == 0. */
int cb_ensemble_step(cb_ensemble *e, int nsteps, int sums_every, cb_sums *out) {
    return cb::guard(nullptr, [&]() -> int {
        if (!e || nsteps < 0 || sums_every < 0) return fail(nullptr, CB_EINVAL, "cb_ensemble_step: bad arguments");
        const int nev = sums_every > 0 ? nsteps / sums_every : 0;
        if (nev > 0 && !out) return fail(nullptr, CB_EINVAL, "cb_ensemble_step: out is NULL");
        const int count = (int)e->members.size();
        const size_t nrec = (size_t)count * nev;
        std::vector<DevState> rec(nrec);
        if (nrec > e->records_cap) {
            cudaFree(e->records);
            e->records = nullptr;
            e->records_cap = 0;
            if (cudaMalloc(&e->records, nrec * sizeof(DevState)) != cudaSuccess) {
                cudaGetLastError();
                return fail(nullptr, CB_ENOMEM, "cb_ensemble_step: device allocation of the records failed");
            }
            e->records_cap = nrec;
        }
        std::vector<double> t_start(count);
        for (int i = 0; i < count; ++i) t_start[i] = e->members[i]->t;
        cudaError_t err = cudaSuccess;
        /* first the members with streams of their own, which then step while the host gets
         * to the batches; records copied on the device */
        for (int i : e->own) {
            if (err != cudaSuccess) break;
            cb_handle *h = e->members[i];
            int done = 0, j = 0;
            while (done < nsteps) {
                const int kk = nev > 0 ? std::min(sums_every, nsteps - done) : nsteps - done;
                const bool line = nev > 0 && kk == sums_every && j < nev;
                int r = step_impl(h, kk, line ? CB_STEP_SUMS : 0, false);
                if (r != CB_OK) { err = cudaErrorLaunchFailure; break; }
                if (line) {
                    err = cudaMemcpyAsync(e->records + (size_t)i * nev + j, h->st, sizeof(DevState),
                                          cudaMemcpyDeviceToDevice, h->stream);
                    if (err != cudaSuccess) break;
                    ++j;
                }
                done += kk;
            }
        }
        for (auto &b : e->batches) {
            if (err != cudaSuccess) break;
            /* whatever the members still have queued on their own streams comes first */
            for (int i : b.idx)
                if (err == cudaSuccess && cudaStreamQuery(e->members[i]->stream) != cudaSuccess) {
                    cudaGetLastError();
                    err = cudaStreamSynchronize(e->members[i]->stream);
                }
            if (err == cudaSuccess) err = run_batch(e, b, nsteps, sums_every, nev);
        }
        /* every stream drains even after an error: the members' buffers must not be in use */
        for (auto &b : e->batches) {
            const cudaError_t s = cudaStreamSynchronize(b.stream);
            if (err == cudaSuccess) err = s;
        }
        for (int i : e->own) {
            const cudaError_t s = cudaStreamSynchronize(e->members[i]->stream);
            if (err == cudaSuccess) err = s;
        }
        if (err == cudaSuccess && nrec > 0)
            err = cudaMemcpy(rec.data(), e->records, nrec * sizeof(DevState), cudaMemcpyDeviceToHost);
        if (err != cudaSuccess) return cuda_fail(nullptr, err, "cb_ensemble_step");
        for (auto &b : e->batches)
            for (int i : b.idx) {
                cb_handle *h = e->members[i];
                if (b.launches & 1) {
                    h->cphi = 1 - h->cphi;
                    h->cpi = 1 - h->cpi;
                }
                for (int q = 0; q < nsteps; ++q) h->t += h->p.dt;   /* bubble.cpp:871, one addition per step */
                h->steps_done += nsteps;
                h->launches += b.launches;
            }
        for (int i = 0; i < count; ++i) {
            cb_handle *h = e->members[i];
            double t = t_start[i];
            for (int j = 0; j < nev; ++j) {
                for (int q = 0; q < sums_every; ++q) t += h->p.dt;
                cb_sums &o = out[(size_t)i * nev + j];
                std::memset(&o, 0, sizeof o);
                const int r = sums_from_record(h, rec[(size_t)i * nev + j], t, &o);
                if (r != CB_OK) return fail(nullptr, r, "cb_ensemble_step: " + h->err);
            }
        }
        return CB_OK;
    });
}

}  // extern "C"
