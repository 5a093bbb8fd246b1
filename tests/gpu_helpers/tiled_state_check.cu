// Test harness: the FP32 engine with its members open: the kernels' error word set from the host (what no
// entry point can bring about without a fault), and which kernels a step takes.
#include <algorithm>
#include <condition_variable>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>
#include <cuda_runtime.h>
#define private public
#include "fv2d_tiled.cu"
#undef private

extern "C" {
// A batch of one solve, one iteration, the error word set to `bits`: the status of get_state, of norms
// and of synchronize, and get_state's message; -1 when the batch could not be made.
int batch_with_error(const fv2d_mesh_desc* d, const fv2d_case* cs, int bits, int* get, int* norms, int* sync, char* msg, int len) {
    std::unique_ptr<fv2d::TiledBatch> b(static_cast<fv2d::TiledBatch*>(fv2d::make_batch_fp32()));
    int sid = -1;
    if (b->init(d->num_cells + 64, d->num_faces + 64, 1) || b->add(d, cs, &sid) || b->step(1) || b->synchronize()) return -1;
    if (cudaMemcpy(b->core_.A_.err, &bits, 4, cudaMemcpyHostToDevice) != cudaSuccess) return -1;
    std::vector<double> q(4 * (size_t)d->num_cells);
    b->err_.clear();
    *get = b->get_state(sid, q.data());
    std::snprintf(msg, len, "%s", b->err_.c_str());
    int id = 0, it = 0, n = 0;
    double nr[4];
    *norms = b->norms(&id, nr, &it, 1, &n);
    *sync = b->synchronize();
    return 0;
}

static int path_of(const fv2d::TiledCore& c) {
    return c.iter_fn_ == (const void*)fv2d::k_titer<2> ? 2 : c.iter_fn_ == (const void*)fv2d::k_titer<3> ? 3 : c.first_ ? 1 : 0;
}
// What steps run, after one: 0 the general stage kernels, 1 the first-order ones, 2 and 3 whole iterations
// with two and three tiles per SM; -1 on an error.  For a single solve, and for a batch of a solve of each case.
int solver_path(const fv2d_mesh_desc* d, const fv2d_case* cs) {
    fv2d::TiledSolver s;
    std::string err;
    if (fv2d::build_mesh(d, cs, s.mesh_, err, s.side_block(d->num_cells)) || s.init(*cs) || s.step(1) || s.synchronize()) return -1;
    return path_of(s.core_);
}
int batch_path(const fv2d_mesh_desc* d, const fv2d_case* cases, int n) {
    fv2d::TiledBatch b;
    if (b.init((long long)n * (d->num_cells + 64), (long long)n * (d->num_faces + 64), n)) return -1;
    for (int i = 0, sid; i < n; i++)
        if (b.add(d, cases + i, &sid)) return -1;
    return b.step(1) || b.synchronize() ? -1 : path_of(b.core_);
}
}
