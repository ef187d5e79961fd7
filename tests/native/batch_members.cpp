/* A batch launch over more lattices than gridDim.y takes, one large lattice among
 * small ones, and its partial sums: what each member gets equals what it gets in a
 * launch of its own. Built and run by test_ensemble_batch_grid_gpu.py. */
#include <cstdio>
#include <cstring>
#include <vector>

#include "cb_handle.h"

namespace cb {
StepConst make_const(const cb_params *p);   /* cb_api.cpp */
}

using namespace cb;

namespace {

struct Lattices {
    std::vector<int> ns;
    std::vector<size_t> at;   /* a member's first element */
    size_t elems = 0;
    float *fields = nullptr;  /* phi, pi, phi', pi' of all members */
    DevState *st = nullptr, *rec = nullptr;
};

cb_params params(int n) {
    cb_params p;
    std::memset(&p, 0, sizeof p);
    p.d = 2;
    p.n_grids = n;
    p.L = n / 8.0;
    p.c = 3.0;
    p.dt = 0.0125;
    p.mpl = 200.0;
    p.delta_v = 1.0;
    p.precision = CB_FP32C;
    p.memorysave = 1;
    return p;
}

StepConst constants(int n) {
    const cb_params p = params(n);
    return make_const(&p);
}

bool ok(cudaError_t e, const char *what) {
    if (e != cudaSuccess) std::printf("%s: %s\n", what, cudaGetErrorString(e));
    return e == cudaSuccess;
}

bool make(Lattices &l, const std::vector<int> &ns) {
    l.ns = ns;
    for (int n : ns) {
        l.at.push_back(l.elems);
        l.elems += (size_t)n * n;
    }
    std::vector<float> f(4 * l.elems, 0.f);
    for (size_t i = 0; i < l.elems; ++i) {
        f[i] = 0.3f + (float)(i * 2654435761u % 1024) / 8192.f;
        f[l.elems + i] = (float)(i * 40503u % 1024) / 16384.f;
    }
    DevState s;
    std::memset(&s, 0, sizeof s);
    s.a = 1.0;
    s.kin_w = 0.5;
    s.vel_w = 1.0;
    s.adx = 0.125;
    s.inv_adx = 8.0;
    s.adx_pow2 = 1;
    std::vector<DevState> all(ns.size(), s);
    return ok(cudaMalloc(&l.fields, f.size() * sizeof(float)), "fields") &&
           ok(cudaMalloc(&l.st, all.size() * sizeof s), "states") && ok(cudaMalloc(&l.rec, all.size() * sizeof s), "records") &&
           ok(cudaMemcpy(l.fields, f.data(), f.size() * sizeof(float), cudaMemcpyHostToDevice), "upload") &&
           ok(cudaMemcpy(l.st, all.data(), all.size() * sizeof s, cudaMemcpyHostToDevice), "upload");
}

/* members [from, to): steps in one launch, the last with sums; fields and records of them */
bool run(Lattices &l, size_t from, size_t to, int steps, std::vector<float> &f, std::vector<DevState> &rec) {
    const std::vector<int> ns(l.ns.begin() + from, l.ns.begin() + to);
    const int kind = batch2_kind(constants(ns[0]), P_FP32);
    const std::vector<int> tiles = batch2_tiles(ns, P_FP32, kind, steps);
    if (tiles.size() != ns.size()) return std::printf("no plan\n"), false;
    std::vector<Batch2Member> m(ns.size());
    int rows = 0;
    for (size_t q = 0; q < ns.size(); ++q) {
        m[q].k = constants(ns[q]);
        for (int i = 0; i < 2; ++i) {
            m[q].phi[i] = l.fields + (size_t)(2 * i) * l.elems + l.at[from + q];
            m[q].pi[i] = l.fields + (size_t)(2 * i + 1) * l.elems + l.at[from + q];
        }
        m[q].st = l.st + from + q;
        m[q].records = l.rec + from + q;
        m[q].row = rows;
        rows += tiles[q];
    }
    /* exactly the rows the members' tiles need, and a guard behind them */
    constexpr int GUARD = 64;
    const size_t row_bytes = NSUM * sizeof(double);
    char *partials = nullptr;
    Batch2Member *dev = nullptr;
    std::vector<char> guard(GUARD * row_bytes);
    bool good = ok(cudaMalloc(&partials, (rows + GUARD) * row_bytes), "partials") &&
                ok(cudaMemset(partials, 0x5a, (rows + GUARD) * row_bytes), "partials") &&
                ok(cudaMalloc(&dev, m.size() * sizeof m[0]), "members") &&
                ok(cudaMemcpy(dev, m.data(), m.size() * sizeof m[0], cudaMemcpyHostToDevice), "members") &&
                ok(launch_step2_batch(P_FP32, kind, dev, ns, steps, 0, 0, (double *)partials, nullptr), "launch") &&
                ok(cudaMemcpy(guard.data(), partials + rows * row_bytes, guard.size(), cudaMemcpyDeviceToHost), "guard");
    for (char c : guard)
        if (good && c != 0x5a) good = false, std::printf("the guard behind the partial sums was written\n");
    const size_t elems = (to < l.at.size() ? l.at[to] : l.elems) - l.at[from];
    f.resize(2 * elems);
    rec.resize(ns.size());
    good = good && ok(cudaMemcpy(f.data(), l.fields + 2 * l.elems + l.at[from], elems * sizeof(float), cudaMemcpyDeviceToHost), "phi") &&
           ok(cudaMemcpy(f.data() + elems, l.fields + 3 * l.elems + l.at[from], elems * sizeof(float), cudaMemcpyDeviceToHost), "pi") &&
           ok(cudaMemcpy(rec.data(), l.rec + from, rec.size() * sizeof(DevState), cudaMemcpyDeviceToHost), "records");
    cudaFree(partials);
    cudaFree(dev);
    return good;
}

bool check(const std::vector<int> &ns, const std::vector<size_t> &which, int steps) {
    Lattices l;
    std::vector<float> all, one;
    std::vector<DevState> rall, rone;
    if (!make(l, ns) || !run(l, 0, ns.size(), steps, all, rall)) return false;
    for (size_t i : which) {
        if (!run(l, i, i + 1, steps, one, rone)) return false;
        const size_t e = (size_t)ns[i] * ns[i];
        if (std::memcmp(&all[l.at[i]], one.data(), e * sizeof(float)) != 0 ||
            std::memcmp(&all[l.elems + l.at[i]], one.data() + e, e * sizeof(float)) != 0)
            return std::printf("member %zu: fields differ\n", i), false;
        /* the same terms in double, in another order where the plan differs */
        const double a = rall[i].etot, b = rone[0].etot;
        if (!(a > 0.0) || a - b > 1e-12 * a || b - a > 1e-12 * a)
            return std::printf("member %zu: etot %.17g alone %.17g\n", i, a, b), false;
    }
    cudaFree(l.fields);
    cudaFree(l.st);
    cudaFree(l.rec);
    return true;
}

}  // namespace

int main() {
    std::vector<int> mixed(2001, 8);
    mixed[0] = 2048;
    const bool good = check(mixed, {0, 1, 2000}, 3) && check(std::vector<int>(66000, 8), {0, 65534, 65535, 65999}, 3);
    std::printf(good ? "ok\n" : "failed\n");
    return good ? 0 : 1;
}
