// Test harness: the FP32 engine's batch with its members open, for what no entry point can bring about
// without a fault: the kernels' error word set from the host.
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
}
