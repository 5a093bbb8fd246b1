// fv2d_residual_noalloc: first-order residual on caller-provided device arrays, with its per-face and
// per-cell scratch in fixed static device arrays, so the call allocates no memory at all.
//
// Who needs it: a caller whose device memory is entirely owned by another allocator (a host
// application that reserves the GPU's memory up front in its own pool, so a cudaMalloc from this
// library would fail or fragment that pool), or a latency-critical thread that must not call
// cudaMalloc/cudaFree because they can synchronise the whole device.  Such a caller passes its
// inputs and outputs as device pointers it already owns; the only extra memory is the static arrays
// below, which live with this library's device code on each GPU until the process exits.  With
// CUDA's lazy module loading (the default) that code and the arrays are placed on a device by the
// first call there, so that first call takes device memory and later calls take none: callers
// whose allocator reserves the GPU make one warm-up call per device before reserving, or set
// CUDA_MODULE_LOADING=EAGER.
//
// Built with -fmad=false, like the FP64 engine, so its arithmetic rounds like the rest of the FP64
// path.  The existing entry points and kernels are untouched.
#include <cuda_runtime.h>

#include <mutex>
#include <string>

#include "fv2d_gpu.h"
#include "fv2d_kernels.cuh"

namespace fv2d {
void set_global_error(const std::string& msg);   // fv2d_api.cu: the text fv2d_last_error(NULL) returns

namespace {

// Face scratch: the residual contribution (V*A - F*A) of every face, 4 doubles per face.
// FV2D_NOALLOC_MAX_FACES * 4 * 8 bytes = 8 MiB.
__device__ __align__(256) double g_noalloc_face_scratch[FV2D_NOALLOC_MAX_FACES * 4];
// Cell scratch (5.3 MiB): the primitives of every cell of a larger mesh (a cell has at least three faces and a face at
// most two cells, so 2/3 of the face limit holds every mesh; one with more cells goes without).
constexpr int kNoallocMaxCells = 2 * (FV2D_NOALLOC_MAX_FACES / 3) + 2;
__device__ __align__(256) double g_noalloc_cell_scratch[kNoallocMaxCells * 4];
// Faces from which the cells' primitives are worth their own launch (about 4 us): with / without, us a
// call: 8.1k faces 16.5 / 12.4, 23.9k 20.6 / 20.6, 48k 22.6 / 24.7, 259k 57.5 / 82.1.
constexpr int kNoallocPrimFaces = 24000;

constexpr int kMaxDevices = 64;
std::mutex g_mu;
double* g_scratch_addr[kMaxDevices][2] = {{nullptr, nullptr}};   // face scratch, cell scratch

// One-time set-up per device, with that device current: the device address of the scratch
// array.  In host code the symbol's name is only a host-side stand-in, never a device address.
// The address is cached per device ordinal for the life of the process; it belongs to the
// device's primary context, so a device reset after the first call is not supported.
int scratch_address(double** face, double** cell) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) { set_global_error(std::string("cudaGetDevice: ") + cudaGetErrorString(e)); return FV2D_ERR_NODEV; }
    if (dev < 0 || dev >= kMaxDevices) { set_global_error("device ordinal out of range"); return FV2D_ERR_NODEV; }
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_scratch_addr[dev][1]) {
        void *p = nullptr, *c = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_face_scratch);
        if (e == cudaSuccess) e = cudaGetSymbolAddress(&c, g_noalloc_cell_scratch);
        if (e != cudaSuccess || !p || !c) {
            set_global_error(std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
            return FV2D_ERR_CUDA;
        }
        g_scratch_addr[dev][0] = (double*)p;
        g_scratch_addr[dev][1] = (double*)c;
    }
    *face = g_scratch_addr[dev][0];
    *cell = g_scratch_addr[dev][1];
    return FV2D_OK;
}

__device__ __forceinline__ bool finite(double x) { return (__double2hiint(x) & 0x7FF00000) != 0x7FF00000; }

// Primitives and sound speed of a state (class_q.hpp:131-141, class_f.hpp:41-50).  Where an infinity, a zero
// or subnormal density or an overflow takes part, Divisor's corrections leave NaN (inf - inf): there
// the quotient is a * (1/b), IEEE's infinity, zero or NaN.  This entry has no non-physical flag, so such a state shows
// in its residual as with plain divisions.  One test for all three quotients (P/rho is not finite if u, v or P
// is not), a branch no warp enters otherwise: 57.4 us a call at 86k polygons and 12.35 at 120 to 7,000 quads
// with and without it, 15k faces 14.4 -> 15.4.  (IEEE divisions in the branch: 57.5 and 13.2; a range
// test of every operand and the plain flux beside the scaled one: 59.5 and 14.4.)
struct Prims {
    double u, v, P, c;
};
__device__ __forceinline__ Prims primitives(const double q[4], const Consts<double>& k, const Fp& fp) {
    Prims p;
    const Divisor r = prims_r(q, k, fp, p.u, p.v, p.P);
    double t = r.div(p.P, fp);
    if (!finite(t)) {
        if (!finite(p.u)) p.u = q[1] * r.y;
        if (!finite(p.v)) p.v = q[2] * r.y;
        p.P = (q[3] - (0.5 * q[0] * (p.u * p.u + p.v * p.v))) * k.gm1;
        t = p.P * r.y;
    }
    p.c = sqrt(k.gamma * t);
    return p;
}

// Cell pass: at first order a face's states are its cells' states, so the primitives are the cells'
// too, once per cell instead of once per face side (six times a polygon).
__global__ void __launch_bounds__(128)
k_noalloc_prims(int nc, const double* __restrict__ q, Prims* __restrict__ prims, Consts<double> k) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    const Fp fp;
    const double s[4] = {q[c], q[(size_t)nc + c], q[2 * (size_t)nc + c], q[3 * (size_t)nc + c]};
    const Prims o = primitives(s, k, fp);
    double2* w = reinterpret_cast<double2*>(prims + c);
    w[0] = make_double2(o.u, o.v);
    w[1] = make_double2(o.P, o.c);
}

// Face pass: first-order reconstruction (face states are the cell states), boundary ghosts,
// Rusanov flux (reconstruction.cpp:22-80, class_f.hpp:41-50, rusanov.cpp:20-36); writes the face's
// residual contribution (res.cpp:81-89) into the scratch.  First order carries no viscous flux
// (res.cpp:27-29), for EULER and NS alike.  CELL: the cells' primitives are in `prims`.
// FP64-pipe-bound (about 125 operations a face, 53 with the cells' primitives), in the exact scalings
// of the engine's face kernel.  86k polygons (259k faces), a call: 57.5 us (this pass 37, its FP64 pipe
// busy 77 %, the cell pass 10, the gather 16), 82 with per-face primitives, 98 with IEEE divisions and
// plain operators.
template <bool CELL>
__global__ void __launch_bounds__(128)
k_noalloc_face(int nf, const int* __restrict__ fc1, const int* __restrict__ fc2, const double* __restrict__ nx,
               const double* __restrict__ ny, const double* __restrict__ area, int nc, const double* __restrict__ q,
               const Prims* __restrict__ prims, double* __restrict__ scratch, Consts<double> k) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const Fp fp;
    const int c1 = fc1[f], c2 = fc2[f];
    const double fnx = nx[f], fny = ny[f], Ah = fp.mul(area[f], fp.half);
    double L[4], Rq[4];
#pragma unroll
    for (int j = 0; j < 4; j++) L[j] = q[(size_t)j * nc + c1];
    const Prims l = CELL ? prims[c1] : primitives(L, k, fp);
    Prims r;
    if (c2 >= 0) {
#pragma unroll
        for (int j = 0; j < 4; j++) Rq[j] = q[(size_t)j * nc + c2];
        if (CELL) r = prims[c2];
    } else if (c2 == -1) {
#pragma unroll
        for (int j = 0; j < 4; j++) Rq[j] = k.q_inf[j];
    } else if (c2 == -2) {
        const double vn = l.u * fnx + l.v * fny;
        cons(L[0], l.u - 2.0 * vn * fnx, l.v - 2.0 * vn * fny, l.P, k, Rq);
    } else if (c2 == -3) {
#pragma unroll
        for (int j = 0; j < 4; j++) Rq[j] = L[j];
    } else {
        cons(L[0], -l.u, -l.v, l.P, k, Rq);
    }
    if (!CELL || c2 < 0) r = primitives(Rq, k, fp);
    const double vn1 = fp.add(fp.mul(l.u, fnx), fp.mul(l.v, fny)), vn2 = fp.add(fp.mul(r.u, fnx), fp.mul(r.v, fny));
    const double t4 = fp.add(fabs(fp.add(vn1, vn2)), fp.add(l.c, r.c));   // 4 lambda
    const double X[4] = {
        fp.add(fp.mul(L[0], vn1), fp.mul(Rq[0], vn2)),
        fp.add(fp.add(fp.mul(fp.mul(L[0], l.u), vn1), fp.mul(l.P, fnx)), fp.add(fp.mul(fp.mul(Rq[0], r.u), vn2), fp.mul(r.P, fnx))),
        fp.add(fp.add(fp.mul(fp.mul(L[0], l.v), vn1), fp.mul(l.P, fny)), fp.add(fp.mul(fp.mul(Rq[0], r.v), vn2), fp.mul(r.P, fny))),
        fp.add(fp.mul(vn1, fp.add(L[3], l.P)), fp.mul(vn2, fp.add(Rq[3], r.P)))};
    double t[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const double F2 = __fma_rn(fp.mul(t4, fp.sub(Rq[j], L[j])), -fp.half, X[j]);   // twice the flux
        t[j] = zero_minus(fp.mul(F2, Ah));
    }
    double2* out = reinterpret_cast<double2*>(scratch + (size_t)4 * f);
    out[0] = make_double2(t[0], t[1]);
    out[1] = make_double2(t[2], t[3]);
}

// Cell pass: gather of the face contributions in the order the cell's face list gives (ascending
// face id reproduces the reference's scatter order, res.cpp:74-102), divided by the volume (:104-109);
// four lanes (one component each) per cell.
__global__ void __launch_bounds__(128)
k_noalloc_gather(int nc, const int* __restrict__ off, const int* __restrict__ inc, const double* __restrict__ vol,
                 const double* __restrict__ scratch, double* __restrict__ r) {
    // (not the thread's index over 4, which wraps from 2^30 cells on; cells without faces count too)
    const unsigned cell = blockIdx.x * (blockDim.x >> 2) + (threadIdx.x >> 2);
    if (cell >= (unsigned)nc) return;
    const int c = (int)cell, j = threadIdx.x & 3;
    const Fp fp;
    const int b = off[c], e = off[c + 1];
    const double v = vol[c];
    double acc = 0.0;
    for (int i0 = b; i0 < e; i0 += 4) {   // four incidences' loads in flight
        int iv[4];
        double t[4];
#pragma unroll
        for (int u = 0; u < 4; u++) iv[u] = i0 + u < e ? inc[i0 + u] : 0;
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (i0 + u < e) t[u] = scratch[(size_t)4 * (iv[u] >> 1) + j];
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (i0 + u < e) acc = fp.add(acc, neg_if(t[u], iv[u] & 1));   // side 1: acc -= t
    }
    r[(size_t)j * nc + c] = acc / v;
}

}  // namespace
}  // namespace fv2d

extern "C" int fv2d_residual_noalloc(const fv2d_noalloc_mesh* m, const fv2d_case* cs, const double* q, double* r,
                                     void* stream) {
    using namespace fv2d;
    if (!m || !cs || !q || !r) { set_global_error("null argument"); return FV2D_ERR_ARG; }
    if (!m->face_cell1 || !m->face_cell2 || !m->face_nx || !m->face_ny || !m->face_area || !m->cell_face_offsets ||
        !m->cell_faces || !m->cell_vol) { set_global_error("null mesh array"); return FV2D_ERR_ARG; }
    if (m->num_cells <= 0 || m->num_faces <= 0) { set_global_error("empty mesh"); return FV2D_ERR_ARG; }
    if (m->num_faces > FV2D_NOALLOC_MAX_FACES) {
        set_global_error("num_faces " + std::to_string(m->num_faces) + " exceeds the static scratch limit of " +
                         std::to_string(FV2D_NOALLOC_MAX_FACES) + " faces; use fv2d_create/fv2d_stage instead");
        return FV2D_ERR_ARG;
    }
    if (!(cs->gamma > 1) || !(cs->rho > 0) || !(cs->P > 0)) { set_global_error("gamma > 1, rho > 0, P > 0 required"); return FV2D_ERR_CASE; }
    if (cs->flux_solver != FV2D_RUSANOV) { set_global_error("flux_solver must be RUSANOV"); return FV2D_ERR_CASE; }
    double *scratch = nullptr, *cells = nullptr;
    int rc = scratch_address(&scratch, &cells);
    if (rc) return rc;
    Consts<double> k{};
    k.gamma = cs->gamma;
    k.gm1 = cs->gamma - 1;
    k.R = cs->R;
    k.q_inf[0] = cs->rho;
    k.q_inf[1] = cs->rho * cs->u;
    k.q_inf[2] = cs->rho * cs->v;
    k.q_inf[3] = (cs->P / (cs->gamma - 1)) + 0.5 * cs->rho * (cs->u * cs->u + cs->v * cs->v);
    cudaStream_t st = (cudaStream_t)stream;
    const int nf = m->num_faces, nc = m->num_cells;
    const bool cell = nf >= kNoallocPrimFaces && nc <= kNoallocMaxCells;
    Prims* prims = reinterpret_cast<Prims*>(cells);
    if (cell) k_noalloc_prims<<<(nc + 127) / 128, 128, 0, st>>>(nc, q, prims, k);
    auto* face = cell ? k_noalloc_face<true> : k_noalloc_face<false>;
    face<<<(nf + 127) / 128, 128, 0, st>>>(nf, m->face_cell1, m->face_cell2, m->face_nx, m->face_ny, m->face_area, nc, q, prims,
                                           scratch, k);
    k_noalloc_gather<<<(int)((4LL * nc + 127) / 128), 128, 0, st>>>(nc, m->cell_face_offsets, m->cell_faces, m->cell_vol, scratch, r);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { set_global_error(std::string("launch: ") + cudaGetErrorString(e)); return FV2D_ERR_CUDA; }
    return FV2D_OK;
}

