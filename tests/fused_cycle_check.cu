// A fused GMRES cycle whose blocks all finished, with the error word set: what a
// block leaves that gave up a bounded wait after block 0 had found the cycle
// converged.  The word is set from the host between two solves.  That solve must
// report a failure, and the next one must be the first one again, bit by bit.
#include "ctx.cuh"
#include "krylov.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

using namespace fvmb;

#define CHECK(cond)                                                                      \
    do {                                                                                 \
        if (!(cond)) { std::printf("line %d: %s (%s)\n", __LINE__, #cond, fvm_last_error()); return 1; } \
    } while (0)

int main() {
    fvm_problem p;
    CHECK(fvm_problem_richards3d(14, 12, 10, 14.0, 12.0, 10.0, 0.15, 1, 1.0, 10.0, 10.0, 2.0, 1e-5, &p) == 0);
    fvm_ctx* c = fvm_create(&p.mesh, &p.phys, 0);
    CHECK(c);
    const int N = p.mesh.n_nodes, m = 30;
    std::vector<double> hy(N), hw(N), first(N), again(N);
    for (int i = 0; i < N; ++i) {
        hy[i] = p.water_table - p.mesh.coords[3 * (size_t)i + 2] + 0.02 * std::sin(1.7 * i);
        hw[i] = 1.0 / (1e-6 * std::fabs(hy[i]) + 1e-6);
    }
    DevBuf<double> y, yp, w, F, x;
    y.upload(hy, c->stream);
    w.upload(hw, c->stream);
    yp.alloc(N);
    F.alloc(N);
    x.alloc(N);
    yp.zero(c->stream);
    CHECK(fvm_begin_step(c, 0.0, y.p, yp.p) == 0);
    CHECK(fvm_residual(c, 0.0, y.p, yp.p, F.p) == 0);
    CHECK(fvm_psetup(c, 0.0, 2e-3, 500.0, y.p, yp.p, F.p, w.p, 1) == 0);
    auto solve = [&](std::vector<double>& out, int& its) {
        double rn = 0.0;
        GmresCounters cnt;
        const int r = gmres_dev(c, 2e-3, y.p, yp.p, F.p, w.p, F.p, x.p, m, 5, 1, 1.0, &its, &rn, &cnt, 1);
        cudaMemcpy(out.data(), x.p, sizeof(double) * N, cudaMemcpyDeviceToHost);
        return r;
    };
    int its1 = 0, its2 = 0, its3 = 0;
    const long before = c->launches;
    CHECK(solve(first, its1) == 0 && its1 > 3);
    CHECK(c->launches - before < its1 + 10);   // (one launch for all steps)
    Krylov* K = c->kry[1];
    const int late = 3;
    CHECK(cudaMemcpy(K->err.p, &late, sizeof(int), cudaMemcpyHostToDevice) == cudaSuccess);
    CHECK(solve(again, its2) == 2);
    CHECK(solve(again, its3) == 0 && its3 == its1);
    CHECK(!std::memcmp(first.data(), again.data(), sizeof(double) * N));
    fvm_destroy(c);
    std::printf("ok\n");
    return 0;
}
