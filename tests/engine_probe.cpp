// Looks inside a batch engine for tests/test_gpu_engine_probe.py: what no call of
// the C ABI returns.  Linked with the library's own object files.
#include <algorithm>
#include <cstdint>
#include <functional>
#include <string>
#include <unordered_map>
#include <vector>

#define private public
#include "../state_estimation_with_cuda_gb300/csrc/engine/engine.h"
#undef private

using sle_gb300::Engine;
using sle_gb300::EngineConfig;
using sle_gb300::SolveRequest;

namespace {
SolveRequest request(int32_t max_iterations, double tol) {
    SolveRequest rq;
    rq.mode = sle_gb300::Mode::PRECISION;
    rq.max_iterations = max_iterations;
    rq.tolerance = tol;
    return rq;
}
}  // namespace

#define PROBE extern "C" __attribute__((visibility("default")))

PROBE Engine* probe_new(int32_t mixed, int32_t dataflow) {
    EngineConfig c;
    c.use_double_precision = mixed ? 0 : 1;
    c.dataflow = dataflow;
    return new Engine(c);
}
PROBE void probe_delete(Engine* e) { delete e; }
PROBE int32_t probe_add_grid(Engine* e, int32_t nb, const int32_t* type, const double* vset, int32_t nbr,
                             const int32_t* from, const int32_t* to, const double* r, const double* x, const double* b,
                             const double* tap, const double* shift, const int32_t* status, int32_t nm,
                             const int32_t* mtype, const int32_t* mloc, const int32_t* mend, const double* sigma,
                             const double* z) {
    int32_t id = -1;
    const int32_t rc = e->batch_add_grid(nb, type, vset, nbr, from, to, r, x, b, tap, shift, status, nm, mtype, mloc,
                                         mend, sigma, z, &id);
    return rc ? rc : id;
}
// Every grid, grid i from a flat start when flat[i]; the steps each took.
PROBE int32_t probe_solve(Engine* e, const uint8_t* flat, double tol, int32_t* steps) {
    const int32_t n = static_cast<int32_t>(e->grids().size());
    std::vector<int32_t> ids(n);
    for (int32_t i = 0; i < n; ++i) ids[i] = i;
    std::vector<Engine::GridResult> res(n);
    const int32_t rc = e->batch_solve(n, ids.data(), flat, request(20, tol), res.data());
    for (int32_t i = 0; i < n; ++i) steps[i] = res[i].iterations;
    return rc;
}
// Grid's part of the solution vector of the last step, in the plan's order.
PROBE int32_t probe_solution(Engine* e, int32_t grid, double* out) {
    int64_t s0 = 0;
    for (int32_t g = 0; g < grid; ++g) s0 += e->grid_plans_[g].n_state;
    const int32_t n = e->grid_plans_[grid].n_state;
    if (cudaStreamSynchronize(e->st_) != cudaSuccess) return -1;
    if (!e->mixed_) return cudaMemcpy(out, e->work_.sol + s0, sizeof(double) * n, cudaMemcpyDeviceToHost) ? -1 : 0;
    std::vector<float> x(n);
    if (cudaMemcpy(x.data(), e->work_.sol32 + s0, sizeof(float) * n, cudaMemcpyDeviceToHost)) return -1;
    std::copy(x.begin(), x.end(), out);
    return 0;
}
// One grid through stream mode.
PROBE int32_t probe_stream(Engine* e, int32_t grid, double tol) {
    int32_t rc = e->stream_begin(request(20, tol));
    if (rc == 0) rc = e->stream_activate(1, &grid, nullptr);
    std::vector<int32_t> done;
    std::vector<Engine::GridResult> res;
    while (rc == 0 && done.empty()) rc = e->stream_step(done, res);
    return rc;
}
PROBE int32_t probe_state(Engine* e, int32_t grid, double* v, double* th) { return e->batch_get_state(grid, v, th); }
// Do reads come from the host model (one copy of the whole batch's states)?
PROBE int32_t probe_reads_shared(Engine* e) { return (e->stale_ & Engine::DL_STATE) == 0; }
