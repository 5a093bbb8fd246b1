// Device code of the FP32 engine: one fused kernel per SSP-RK3 stage over the tile layout of
// fv2d_tiles.h.  Each CTA takes tiles from a counter; per tile:
//   load    one thread issues bulk asynchronous copies (cp.async.bulk, the TMA engine) of the
//           tile's record block, csr block and core-cell states into shared memory on an mbarrier
//           (its halo list was copied, and its blocks prefetched into L2, during the previous
//           tile's last flux pass); every wait on an mbarrier is bounded and reports a timeout
//   gather  meanwhile, the states of the ring-1 and ring-2 cells (neighbours of the tile)
//   grad    LSQ gradient + squeeze limiter of every core and ring-1 cell (compute_gradient,
//           src/solver/cell_gradient.cpp:9-131; squeeze, src/solver/squeeze.cpp:9-155), each cell's
//           sums in ascending original face id; limited gradients stay in shared memory
//   flux    reconstruction + boundary ghosts (reconstruction.cpp:22-80), NS face terms (:86-164),
//           Rusanov flux (rusanov.cpp:20-36) of every face of a core cell; the face's contribution
//           V*A - F*A (res.cpp:81-89) overwrites its displacement row in shared memory
//   update  residual gather (res.cpp:74-109), time step (ssp_rk3.cpp:24-47) and the SSP-RK3 stage
//           (ssp_rk3.cpp:50-77) of the core cells, in the compensated delta form of the FP32 path;
//           on the last stage, per-warp spectral maxima and residual sums, folded into the solve's
//           maximum and the tile's norm partials at the next tile's top
// A face shared by two tiles is evaluated by both, with the same inputs and the same code, so both
// get the same value; every per-cell sum runs in a fixed order, so results do not depend on the
// tile schedule, and a solve gives the same bits alone and in a batch (both run these kernels).
// First-order solves have a smaller kernel per stage (k_tfirst); solves whose tiles all fit on the GPU at once
// run whole iterations in one launch (k_titer).  Both run the same passes.
#pragma once

#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

#include "fv2d_kernels.cuh"
#include "fv2d_tiles.h"

namespace fv2d {

struct __align__(16) TParams {   // per solve
    Consts<float> k;
    int order2, ns, squeeze, global_dt;
    int fresh, init_prims, pad0, pad1;
};
static_assert(sizeof(TParams) % 16 == 0, "TParams is copied in 16-byte pieces");

struct TArgs {
    const TileDesc* tiles;
    const int* ntiles;
    int* counter;              // [3] next tile of each stage kernel (kernel s zeroes stage s+1's)
    TParams* P;
    const uint32_t* rec;
    const uint16_t* csr;
    const int* halo;
    const int* qcell;
    Q4<float>* Q[3];           // stage inputs: Qn, Q1, Q2
    Q4<float>* G[3];           // limited gradient of each stage input (x, y per cell)
    Q4<float>* D;              // RK increment (delta form)
    Q4<float>* Qlo;            // compensation term of Qn
    Q4<float>* R;              // residual (null: not kept)
    float *dt, *S;
    const float *vol, *rvol;
    const float4* lsq;         // per cell: the LSQ inverse-moment terms (Ixx, Iyy, Ixy) rounded to FP32, 0
    float* smax;               // [solves] max spectral sum (GLOBAL dt; zeroed by the second stage)
    int nsmax;                 // entries of smax
    int* flags;                // [solves] non-physical state seen
    double* tpart;             // [tiles][4] residual sums of squares of the last stage (null: none)
    int* err;                  // 2: an mbarrier wait timed out; 4: a tile descriptor out of range; 8: a grid barrier timed out
    int store_r;               // keep R on stages 0 and 1 too
};

// Shared-memory plan of one CTA (bytes; every region 16-byte aligned).
constexpr int kSmRecWords = 5 * kTileRecs + 3 * kTileGeo;
constexpr int kSmRec = 4 * kSmRecWords;
constexpr int kSmCsr = ((2 * kTileCsr + 15) / 16) * 16;
constexpr int kSmHalo = 4 * kTileCells;
constexpr int kSmCq = 16 * kTileCells;
constexpr int kSmCg = 32 * kTileGrad;
constexpr int kSmTotal = kSmRec + kSmCsr + kSmHalo + kSmCq + kSmCg;
constexpr int kSmTotalMax = 226 * 1024;   // a CTA's limit (227 KB) less its static shared memory

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t mb, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mb), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t mb, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes) : "memory");
}
// Bounded wait for the mbarrier phase with the given parity: false after ~2^22 polls (each poll
// suspends the thread for a while, so this is far longer than any copy takes).
__device__ __forceinline__ bool mbar_wait(uint32_t mb, uint32_t parity) {
    for (int i = 0; i < (1 << 22); i++) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(mb), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// Bulk copy global -> shared (16-byte aligned addresses, size a multiple of 16), completing on mb.
__device__ __forceinline__ void tma_load(void* dst, const void* src, uint32_t bytes, uint32_t mb) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(mb)
                 : "memory");
}

__device__ __forceinline__ float fw(uint32_t w) { return __uint_as_float(w); }

// Asynchronous copy of a 16-byte aligned object (a tile descriptor, a solve's parameters) to shared
// memory; complete after cp.async.wait_all.
template <class T>
__device__ __forceinline__ void copy_async(T* dst, const T* src) {
    static_assert(sizeof(T) % 16 == 0, "16-byte pieces");
#pragma unroll
    for (int i = 0; i < (int)(sizeof(T) / 16); i++)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst) + 16 * i),
                     "l"(reinterpret_cast<const char*>(src) + 16 * i)
                     : "memory");
}


// Every operation of the passes below rounds as written here, so the kernels that share them get the
// same bits: a product is either rounded by itself (fm, which the compiler does not contract) or
// the exact operand of a fused multiply-add (ff).
__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return a + b; }
__device__ __forceinline__ float fs(float a, float b) { return a - b; }
__device__ __forceinline__ float ff(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// a*b + c*d with the first product exact
__device__ __forceinline__ float mm(float a, float b, float c, float d) { return ff(a, b, fm(c, d)); }

// Primitives of a conservative state; returns 1/rho for later quotients.
__device__ __forceinline__ void tprims(const float p[4], const Consts<float>& k, float& rho, float& u, float& v,
                                       float& P, float& y) {
    rho = p[0];
    y = 1.0f / rho;
    u = fm(p[1], y);
    v = fm(p[2], y);
    P = fm(ff(-fm(0.5f, rho), mm(u, u, v, v), p[3]), k.gm1);
}
// Conservative state of primitives.
__device__ __forceinline__ void tcons(float rho, float u, float v, float P, const Consts<float>& k, float q[4]) {
    q[0] = rho;
    q[1] = fm(rho, u);
    q[2] = fm(rho, v);
    q[3] = ff(fm(0.5f, rho), mm(u, u, v, v), P / k.gm1);
}
// The no-slip wall's ghost of state p (primitives rho, u, v): velocity negated, the energy rebuilt
// from the pressure with the kinetic energy's rounded value in both steps.
__device__ __forceinline__ void tghost_noslip(const float p[4], const Consts<float>& k, float q[4]) {
    const float rho = p[0], y = 1.0f / rho, u = fm(p[1], y), v = fm(p[2], y);
    const float ke = mm(u, u, v, v), h = fm(0.5f, rho), m = fm(h, ke);
    q[0] = rho;
    q[1] = fm(rho, -u);
    q[2] = fm(rho, -v);
    q[3] = ff(fm(fs(p[3], m), k.gm1), 1.0f / k.gm1, m);
}

// A tile's blocks in shared memory, as the passes read them.
struct TileView {
    const uint32_t* sl;               // records: the two cells' local slots
    const float4* d;                  // records: (d1x, d1y, d2x, d2y)
    const float *nx, *ny, *A;         // records [0, ngeo)
    const uint16_t* off;              // csr offsets (bit 15 of an end offset: the cell has a boundary face)
    const uint32_t* ent;              // csr entries
    const Q4<float>* cq;              // cell states
    const Q4<float> *cg, *cgy;        // limited gradients per core and ring-1 cell, x and y apart: a warp's
                                      // gathers of 16-byte rows meet fewer bank conflicts than of 32-byte pairs
                                      // (1M-cell NS cylinder 309.6 -> 304.0 us per iteration)
};

// Of a programmatic dependent launch: all writes of the kernels before are visible after it.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The limited LSQ gradient of one core or ring-1 cell (local slot gI).  ghost(r): the state of the
// cell that a no-slip face's gradient ghost reads; prev(): the cell's previous-stage state.  PAIRS: warps
// without boundary faces take two faces at a time, whose extremes cost one three-operand minimum or
// maximum each instead of two (the stage kernels, bound by issue: 1M-cell NS cylinder 304.0 ->
// 298.4 us per iteration, 600k quads 157.0 -> 155.9; the whole-iteration kernel, bound by latency, is faster without:
// 50k Euler polygons 19.46 against 19.69).
template <bool PAIRS, class Ghost, class Prev>
__device__ __forceinline__ void tile_gradient(const TileView& v, const Consts<float>& k, int gI, bool squeeze, bool lim_prev,
                                              bool init_prims, bool stage0, const float4& mom, const Q4<float>& gpx,
                                              const Q4<float>& gpy, Ghost ghost, Prev prev, Q4<float>& gx, Q4<float>& gy) {
    const Q4<float> qc = v.cq[gI];
    // LSQ sums (Q(c2) - Q(c1)) * (dxj, dyj) over the cell's faces and, for the squeeze limiter, the
    // extremes over the neighbours of Q(n) - Q(c) (= the bounds Qmax - Q, Qmin - Q of squeeze.cpp:
    // rounding is monotone, so the extreme difference is the difference of the extreme) and over the
    // faces of gprev . (face centre - centre), the previous face value's part that varies by face
    // (its base Qprev - Q is added after the loop, again exactly for the extremes)
    float sx[4] = {0.f, 0.f, 0.f, 0.f}, sy[4] = {0.f, 0.f, 0.f, 0.f};
    float dmin[4], dmax[4], tmin[4], tmax[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        dmin[j] = 0.f; dmax[j] = 0.f;
        tmin[j] = 3.0e38f; tmax[j] = -3.0e38f;
    }
    // bit 15 of the end offset: the cell has a boundary face; the others' loop has no boundary
    // branches
    const uint32_t o1 = v.off[gI + 1];
    const int e0 = v.off[gI] & 0x7FFF, e1 = (int)(o1 & 0x7FFFu);
    auto face_loop = [&](auto interior, int first) {
        constexpr bool INTERIOR = decltype(interior)::value;
        for (int e = first; e < e1; e++) {
            const uint32_t ent = v.ent[e];
            const int r = (int)((ent & 0xFFFFu) >> 1), side = (int)(ent & 1u);
            const int so = (int)(int16_t)(ent >> 16);   // the face's other cell (or BC code)
            const float4 dd = v.d[r];
            const float d1x = dd.x, d1y = dd.y, d2x = dd.z, d2y = dd.w;
            float d[4];
            if (INTERIOR || so >= 0) {
                const Q4<float> qn = v.cq[so];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    d[j] = fs(qn.p[j], qc.p[j]);
                    if (squeeze) { dmin[j] = fminf(dmin[j], d[j]); dmax[j] = fmaxf(dmax[j], d[j]); }
                }
            } else if (so == -1) {
#pragma unroll
                for (int j = 0; j < 4; j++) d[j] = fs(k.q_inf[j], qc.p[j]);
            } else if (so == -2 || so == -4) {
                float rho, u, vv, P, yr, gq[4];
                if (so == -2) {   // slip wall: the cell velocity reflected (cell_gradient.cpp:43-55)
                    if (init_prims) { rho = k.rho_inf; u = k.u_inf; vv = k.v_inf; P = k.P_inf; }
                    else tprims(qc.p, k, rho, u, vv, P, yr);
                    const float fnx = v.nx[r], fny = v.ny[r];
                    const float vn2 = fm(2.0f, mm(u, fnx, vv, fny));
                    tcons(rho, ff(-vn2, fnx, u), ff(-vn2, fny, vv), P, k, gq);
                } else if (stage0) {   // no-slip: cell `face id`'s state, velocity negated (:62-73)
                    if (init_prims) { rho = k.rho_inf; u = k.u_inf; vv = k.v_inf; P = k.P_inf; }
                    else { const Q4<float> qq = ghost(r); tprims(qq.p, k, rho, u, vv, P, yr); }
                    tcons(rho, -u, -vv, P, k, gq);
                } else {
                    const Q4<float> qq = ghost(r);
                    tghost_noslip(qq.p, k, gq);
                }
#pragma unroll
                for (int j = 0; j < 4; j++) d[j] = fs(gq[j], qc.p[j]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++) d[j] = 0.f;
            }
            // LSQ displacement c1 -> c2 (or ghost), times Q(c2) - Q(c1): for a c2-side cell the
            // difference above is Q(c1) - Q(c2), so the displacement's sign is flipped instead
            const float fx = side ? fs(d2x, d1x) : fs(d1x, d2x), fy = side ? fs(d2y, d1y) : fs(d1y, d2y);
            const float ox = side ? d2x : d1x, oy = side ? d2y : d1y;   // face centre - this cell
#pragma unroll
            for (int j = 0; j < 4; j++) {
                sx[j] = ff(d[j], fx, sx[j]);
                sy[j] = ff(d[j], fy, sy[j]);
                if (lim_prev) {
                    const float x = mm(gpx.p[j], ox, gpy.p[j], oy);
                    tmin[j] = fminf(tmin[j], x);
                    tmax[j] = fmaxf(tmax[j], x);
                }
            }
        }
    };
    // one loop per warp: the general one if any of its cells has a boundary face (a warp running
    // both would take the sum of the two)
    if (__any_sync(__activemask(), (o1 & 0x8000u) != 0)) face_loop(std::false_type{}, e0);
    else if (!PAIRS) face_loop(std::true_type{}, e0);
    else {
        int e = e0;
        for (; e + 1 < e1; e += 2) {
            const uint32_t ea = v.ent[e], eb = v.ent[e + 1];
            const float4 da = v.d[(ea & 0xFFFFu) >> 1], db = v.d[(eb & 0xFFFFu) >> 1];
            const Q4<float> qa = v.cq[(int)(int16_t)(ea >> 16)], qb = v.cq[(int)(int16_t)(eb >> 16)];
            const bool sa = ea & 1u, sb = eb & 1u;
            // as above: the face centre from this cell (o) and the displacement to the other's (f)
            const float oxa = sa ? da.z : da.x, oya = sa ? da.w : da.y, oxb = sb ? db.z : db.x, oyb = sb ? db.w : db.y;
            const float fxa = fs(oxa, sa ? da.x : da.z), fya = fs(oya, sa ? da.y : da.w);
            const float fxb = fs(oxb, sb ? db.x : db.z), fyb = fs(oyb, sb ? db.y : db.w);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float a = fs(qa.p[j], qc.p[j]), b = fs(qb.p[j], qc.p[j]);
                sx[j] = ff(b, fxb, ff(a, fxa, sx[j]));
                sy[j] = ff(b, fyb, ff(a, fya, sy[j]));
                if (squeeze) { dmin[j] = fminf(fminf(a, b), dmin[j]); dmax[j] = fmaxf(fmaxf(a, b), dmax[j]); }
                if (lim_prev) {
                    const float x = mm(gpx.p[j], oxa, gpy.p[j], oya), y = mm(gpx.p[j], oxb, gpy.p[j], oyb);
                    tmin[j] = fminf(fminf(x, y), tmin[j]);
                    tmax[j] = fmaxf(fmaxf(x, y), tmax[j]);
                }
            }
        }
        face_loop(std::true_type{}, e);
    }
    const float ixx = mom.x, iyy = mom.y, ixy = mom.z;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        gx.p[j] = mm(sx[j], iyy, -sy[j], ixy);
        gy.p[j] = mm(sy[j], ixx, -sx[j], ixy);
    }
    if (squeeze) {
        // squeeze (squeeze.cpp:68-141): phi = the smallest (bound - Q) / (face value - Q) over the
        // faces whose previous face value leaves [Qmin, Qmax]; as x -> (bound - Q) / x is monotone
        // on either side of zero, that is the quotient at the extreme t
        Q4<float> qp;
        if (lim_prev) qp = prev();
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float up = dmax[j], dn = dmin[j];
            // t = (previous face value) - Q: its base plus the extremes above; -101 is the fresh
            // face history's value
            const float base = lim_prev ? fs(qp.p[j], qc.p[j]) : fs(-101.0f, qc.p[j]);
            const float thi = lim_prev ? fa(base, tmax[j]) : base, tlo = lim_prev ? fa(base, tmin[j]) : base;
            float phi = 1.0f;
            if (thi > up) phi = fminf(phi, up / thi);
            if (tlo < dn) phi = fminf(phi, dn / tlo);
            gx.p[j] = fm(gx.p[j], phi);
            gy.p[j] = fm(gy.p[j], phi);
        }
    }
}

// Flux of one face of a core cell (record r): V*A - F*A to w_t[r] and, on an iteration's last
// stage, its spectral term to w_sp[r].  (w_t and w_sp may be the record's own displacement and
// normal-x rows: both are read before they are written.)  INTERIOR: the record joins two cells, so
// the boundary branches go and both sides' reconstructions can be scheduled together.
template <bool INTERIOR, bool FIRST = false>
__device__ __forceinline__ void tile_flux(const TileView& v, const Consts<float>& k, int r, bool order2, bool visc,
                                          bool init_prims, bool last, float4* w_t, float* w_sp) {
    const Q4<float>* cq = v.cq;
    const Q4<float>* cg = v.cg;
    const Q4<float>* cgy = v.cgy;
    const uint32_t sl = v.sl[r];
    const int s1 = (int)(sl & 0xFFFFu), s2 = (int)(int16_t)(sl >> 16);
    const float4 dd = FIRST ? make_float4(0.f, 0.f, 0.f, 0.f) : v.d[r];
    const float d1x = dd.x, d1y = dd.y, d2x = dd.z, d2y = dd.w;
    const float fnx = v.nx[r], fny = v.ny[r];
    const float mxf = -fny, myf = fnx;   // unit tangent p1 -> p2
    // face states; for NS also the face-average tangential derivative m.(grad Q1 + grad Q2)/2,
    // the difference Q2 - Q1 and c1's velocity, so the cell states and gradients die early
    float L[4], Rq[4], dm[4], dq[4];
    float cu = 0.f, cv = 0.f;
    {
        const Q4<float> q1 = cq[s1];
        Q4<float> g1x, g1y;
        if (order2) { g1x = cg[s1]; g1y = cgy[s1]; }
        else {
#pragma unroll
            for (int j = 0; j < 4; j++) { g1x.p[j] = 0.f; g1y.p[j] = 0.f; }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            L[j] = FIRST ? q1.p[j] : ff(g1y.p[j], d1y, ff(g1x.p[j], d1x, q1.p[j]));
            dm[j] = mm(g1y.p[j], myf, g1x.p[j], mxf);
            dq[j] = -q1.p[j];
        }
        if (!INTERIOR && visc && s2 == -4) {
            if (init_prims) { cu = k.u_inf; cv = k.v_inf; }
            else { const float yq = 1.0f / q1.p[0]; cu = fm(q1.p[1], yq); cv = fm(q1.p[2], yq); }
        }
    }
    float lrho, lu, lv, lP, ly;
    tprims(L, k, lrho, lu, lv, lP, ly);
    if (INTERIOR || s2 >= 0) {
        const Q4<float> q2 = cq[s2];
        Q4<float> g2x, g2y;
        if (order2) { g2x = cg[s2]; g2y = cgy[s2]; }
        else {
#pragma unroll
            for (int j = 0; j < 4; j++) { g2x.p[j] = 0.f; g2y.p[j] = 0.f; }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            Rq[j] = FIRST ? q2.p[j] : ff(g2y.p[j], d2y, ff(g2x.p[j], d2x, q2.p[j]));
            dm[j] = fm(0.5f, ff(g2y.p[j], myf, ff(g2x.p[j], mxf, dm[j])));
            dq[j] = fa(dq[j], q2.p[j]);
        }
    } else if (s2 == -1) {
#pragma unroll
        for (int j = 0; j < 4; j++) Rq[j] = k.q_inf[j];
    } else if (s2 == -2) {
        const float vn2 = fm(2.0f, mm(lu, fnx, lv, fny));
        tcons(lrho, ff(-vn2, fnx, lu), ff(-vn2, fny, lv), lP, k, Rq);
    } else if (s2 == -3) {
#pragma unroll
        for (int j = 0; j < 4; j++) Rq[j] = L[j];
    } else {
        tghost_noslip(L, k, Rq);
    }
    const float A = v.A[r];
    const float lc = sqrtf(fm(fm(k.gamma, lP), ly));
    float rrho, ru, rv, rP, ry;
    tprims(Rq, k, rrho, ru, rv, rP, ry);
    const float rc = sqrtf(fm(fm(k.gamma, rP), ry));
    const float vn1 = mm(lu, fnx, lv, fny), vn2 = mm(ru, fnx, rv, fny);
    const float vna = fm(0.5f, fa(vn1, vn2)), ca = fm(0.5f, fa(lc, rc));
    const float sp = fa(fabsf(vna), ca);
    const float lam = fm(0.5f, sp);
    float Fr[4];
    if (k.roe) {
#pragma unroll
        for (int j = 0; j < 4; j++) Fr[j] = -101.0f;
    } else {
        // F(L) + F(R)
        const float lE = fa(L[3], lP);
        const float rE = fa(Rq[3], rP);
        const float X[4] = {
            mm(lrho, vn1, rrho, vn2),
            fa(mm(fm(lrho, lu), vn1, lP, fnx), mm(fm(rrho, ru), vn2, rP, fnx)),
            fa(mm(fm(lrho, lv), vn1, lP, fny), mm(fm(rrho, rv), vn2, rP, fny)),
            mm(vn1, lE, vn2, rE)};
#pragma unroll
        for (int j = 0; j < 4; j++) Fr[j] = mm(0.5f, X[j], -lam, fs(Rq[j], L[j]));
    }
    float V[4] = {0.f, 0.f, 0.f, 0.f};
    if (visc) {   // first order never adds the viscous flux (res.cpp:27-29,50-53)
        float S[4];
#pragma unroll
        for (int j = 0; j < 4; j++) S[j] = fa(L[j], Rq[j]);
        const float arho = fm(0.5f, S[0]), ya = 1.0f / arho;
        const float au = fm(fm(0.5f, S[1]), ya), av = fm(fm(0.5f, S[2]), ya);
        const float ke = mm(au, au, av, av);
        const float aP = fm(mm(0.5f, S[3], -fm(0.5f, arho), ke), k.gm1);
        float ux = 0.f, uy = 0.f, vx = 0.f, vy = 0.f, Px = 0.f, Py = 0.f, rx = 0.f, rly = 0.f;
        bool have = true;
        if (INTERIOR || s2 >= 0) {
            // l: unit vector c1 -> c2 (the LSQ displacement d1 - d2)
            const float tx = fs(d1x, d2x), ty = fs(d1y, d2y);
            const float yd = rsqrtf(mm(tx, tx, ty, ty));
            const float lxf = fm(tx, yd), lyf = fm(ty, yd);
            float dl[4];
#pragma unroll
            for (int j = 0; j < 4; j++) dl[j] = ff(dq[j], yd, dm[j]);   // reconstruction.cpp:138-146: l for both terms
            rx = fm(dl[0], lxf);
            const float rxu = fm(rx, au), rxv = fm(rx, av);
            ux = mm(dl[1], lxf, -rxu, ya);
            vx = mm(dl[2], lxf, -rxv, ya);
            rly = fm(dl[0], lyf);
            const float ryu = fm(rly, au);
            uy = mm(dl[1], lyf, -ryu, ya);
            vy = mm(dl[2], lyf, -ryu, ya);   // reconstruction.cpp:155 uses u
            Px = fm(k.gm1, ff(-arho, mm(au, ux, av, vx), mm(dl[3], lxf, -fm(0.5f, rx), ke)));
            Py = fm(k.gm1, ff(-arho, mm(au, uy, av, vy), mm(dl[3], lyf, -fm(0.5f, rly), ke)));
        } else if (s2 == -4) {
            const float ydn = rsqrtf(mm(d1x, d1x, d1y, d1y));
            const float dudn = fm(-cu, ydn), dvdn = fm(-cv, ydn);
            ux = fm(dudn, fnx); uy = fm(dudn, fny);
            vx = fm(dvdn, fnx); vy = fm(dvdn, fny);
        } else if (s2 == -2) {
            have = false;   // SLIP_WALL with NS: tau and grad T stay zero (:104-106)
        }
        if (have) {
            const float div = fa(ux, vy), mu2 = fm(2.0f, k.mu), third = 1.0f / 3.0f;
            const float txx = fm(mu2, ff(-div, third, ux));
            const float tyy = fm(mu2, ff(-div, third, vy));
            const float txy = fm(k.mu, fa(uy, vx));
            const float yden = 1.0f / fm(fm(k.R, arho), arho);
            const float dTx = fm(mm(Px, arho, -rx, aP), yden);
            const float dTy = fm(mm(Py, arho, -rly, aP), yden);
            V[1] = mm(txy, fny, txx, fnx);
            V[2] = mm(txy, fnx, tyy, fny);
            V[3] = mm(fnx, ff(k.k, dTx, mm(av, txy, au, txx)), fny,
                      ff(k.k, dTy, mm(au, txy, av, tyy)));
        }
    }
    w_t[r] = make_float4(fm(fs(V[0], Fr[0]), A), fm(fs(V[1], Fr[1]), A), fm(fs(V[2], Fr[2]), A), fm(fs(V[3], Fr[3]), A));
    if (last) w_sp[r] = k.roe ? fm(fa(fabsf(k.vn0), k.c0), A) : fm(sp, A);
}

// Residual of core cell c (res.cpp:74-109): its faces' contributions in ascending original face id,
// over its volume (yv = 1/vol); on the last stage its spectral terms' sum too.  The side's sign enters
// as an exact factor of a multiply-add, which costs no operation of its own (300k first-order
// polygons 30.13 -> 29.63 us per iteration).
__device__ __forceinline__ void tile_residual(const TileView& v, int c, const float4* w_t, const float* w_sp, bool last,
                                              float yv, float r4[4], float& snext) {
#pragma unroll
    for (int j = 0; j < 4; j++) r4[j] = 0.f;
    const int e0 = v.off[c] & 0x7FFF, e1 = v.off[c + 1] & 0x7FFF;
    for (int e = e0; e < e1; e++) {
        const uint32_t ent = v.ent[e];
        const int r = (int)((ent & 0xFFFFu) >> 1);
        const float4 tv = w_t[r];
        const float sg = __uint_as_float((ent << 31) | 0x3F800000u);   // +1 or, on the face's second side, -1
        r4[0] = ff(tv.x, sg, r4[0]);
        r4[1] = ff(tv.y, sg, r4[1]);
        r4[2] = ff(tv.z, sg, r4[2]);
        r4[3] = ff(tv.w, sg, r4[3]);
        if (last) snext = fa(snext, w_sp[r]);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) r4[j] = fm(r4[j], yv);
}

// The SSP-RK3 stage (ssp_rk3.cpp:50-77) in the compensated delta form: dn the new increment (first
// two stages), out the new state, lo the base state's compensation (updated by the last stage).
__device__ __forceinline__ void stage_combine(int stage, float dtc, const float r4[4], const Q4<float>& qn,
                                              const Q4<float>& dprev, Q4<float>& lo, Q4<float>& dn, Q4<float>& out) {
    if (stage == 0) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            dn.p[j] = fm(dtc, r4[j]);
            out.p[j] = fa(qn.p[j], dn.p[j]);
        }
    } else if (stage == 1) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            dn.p[j] = mm(0.25f, dprev.p[j], fm(0.25f, dtc), r4[j]);
            out.p[j] = fa(qn.p[j], dn.p[j]);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float inc = mm(2.0f / 3.0f, dprev.p[j], fm(2.0f / 3.0f, dtc), r4[j]);
            float s, err;
            two_sum(qn.p[j], fa(lo.p[j], inc), s, err);
            out.p[j] = s;
            lo.p[j] = err;
        }
    }
}

template <int STAGE>
__global__ void __launch_bounds__(kTileCore, 3) k_tstage(TArgs a) {
    extern __shared__ __align__(128) unsigned char sm[];
    uint32_t* srec = reinterpret_cast<uint32_t*>(sm);
    uint16_t* scsr = reinterpret_cast<uint16_t*>(sm + kSmRec);
    int* shalo = reinterpret_cast<int*>(sm + kSmRec + kSmCsr);
    Q4<float>* cq = reinterpret_cast<Q4<float>*>(sm + kSmRec + kSmCsr + kSmHalo);
    Q4<float>* cg = reinterpret_cast<Q4<float>*>(sm + kSmRec + kSmCsr + kSmHalo + kSmCq);
    Q4<float>* cgy = cg + kTileGrad;
    __shared__ TileDesc td;
    __shared__ __align__(16) TileDesc tdn;   // the next tile this CTA takes
    __shared__ TParams tp, tpn;   // this tile's solve parameters, the next tile's
    __shared__ __align__(8) unsigned long long mbar, mbar_h;
    __shared__ int s_next, s_ctr[2];
    __shared__ float redf[kTileCore / 32];      // last stage: per-warp spectral maxima of a tile
    __shared__ float redw[4][kTileCore / 32];   // and per-warp residual sums of squares

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t mb = smem_u32(&mbar), mbh = smem_u32(&mbar_h);
    uint32_t parity = 0, parity_h = 0;
    const int ntiles = *a.ntiles;
    const Q4<float>* __restrict__ Qin = a.Q[STAGE];
    const Q4<float>* __restrict__ Qprev = a.Q[(STAGE + 2) % 3];
    const Q4<float>* __restrict__ Gprev = a.G[(STAGE + 2) % 3];
    Q4<float>* __restrict__ Gout = a.G[STAGE];

    // thread 0 takes each next tile while the current one is being processed: its index during
    // the halo gather (whose own loads cover the atomic's latency; a barrier waits for the
    // thread's outstanding accesses), its descriptor by an asynchronous copy to shared memory
    // issued in the gradient pass; in the last flux pass (the halo list is free by then) it checks
    // the descriptor and starts the copy of the next tile's halo list, so that the next tile's
    // ring states are gathered while its other blocks are copied.  The solve's parameters are
    // reloaded only when the solve changes.
    int next_t = 0, tp_sid = -1, tpn_sid = -1;
    // (last stage) a tile's per-warp spectral maxima and residual sums are folded by the last warp
    // at the top of the next tile, while its blocks are copied (or at the end): the tile's maximum
    // into its solve's by an atomic, the sums of squares over the warps in FP64, in warp order, into
    // the tile's partials (batches' norms).  No barrier waits for either.
    int red_t = -1, red_sid = 0;
    auto fold = [&]() {
        if (STAGE != 2 || red_t < 0 || warp != kTileCore / 32 - 1) return;
        if (a.tpart && lane < 4) {
            double sum = 0.0;
            for (int w = 0; w < kTileCore / 32; w++) sum += (double)redw[lane][w];
            a.tpart[4 * (size_t)red_t + lane] = sum;
        }
        if (lane == 0) {
            float bm = 0.f;
            for (int w = 0; w < kTileCore / 32; w++) bm = max2(bm, redf[w]);
            atomic_max_pos(a.smax + red_sid, bm);
        }
        red_t = -1;
    };
    // (thread 0) the next tile's fate in s_next: its index, -1 (none left) or -2 (an empty slot of
    // a removed solve, or a descriptor out of range: skipped); for a tile, the halo copy on mbar_h,
    // whose phase also publishes tdn to the threads that wait on it
    auto decide = [&]() {
        if (next_t >= ntiles) { s_next = -1; return; }
        const TileDesc& d = tdn;
        if (d.ncore == 0) { s_next = -2; return; }
        const bool ok = d.ncore > 0 && d.ncore <= kTileCore && d.ncore + d.n1 <= kTileGrad &&
                        d.ncore + d.n1 + d.n2 <= kTileCells && d.nr <= kTileRecs && d.ngeo <= kTileGeo &&
                        d.ncc >= 0 && d.ncc <= d.nint && d.nint <= d.nrc && d.nrc <= d.ngeo && d.ngeo <= d.nr && d.fpw >= 32 && d.fpw <= 1024 &&
                        (d.fpw & 31) == 0 && d.nrp >= d.nr && d.ngp >= d.ngeo &&
                        5 * d.nrp + 3 * d.ngp <= kSmRecWords && d.ncsr <= kTileCsr && d.noff <= d.ncsr &&
                        d.n1 + d.n2 <= d.nhalo && d.nhalo <= kTileCells && (d.nrp & 3) == 0 && (d.ngp & 3) == 0 &&
                        (d.ncsr & 7) == 0 && (d.nhalo & 3) == 0 && (d.rec & 3) == 0 && (d.csr & 7) == 0 && (d.halo & 3) == 0;
        if (!ok) { atomicOr(a.err, 4); s_next = -2; return; }
        // the earlier generic accesses of the halo list are complete (a barrier precedes every
        // call); order them before the async-proxy writes
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        const uint32_t bhal = 4u * (uint32_t)d.nhalo;
        mbar_expect_tx(mbh, bhal);
        if (bhal) tma_load(shalo, a.halo + d.halo, bhal, mbh);
        {   // the tile's other blocks into L2 now, so that the copies at its top come from L2
            const uint32_t brec = 4u * (uint32_t)(5 * d.nrp + 3 * d.ngp), bcsr = 2u * (uint32_t)d.ncsr,
                           bq = 16u * (uint32_t)d.ncore;
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.rec + d.rec), "r"(brec) : "memory");
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.csr + d.csr), "r"(bcsr) : "memory");
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(Qin + d.c0), "r"(bq) : "memory");
        }
        s_next = next_t;
    };
    // for the next kernel in the stream: the next stage's tile counter and, in the second stage
    // (which does not read them), the GLOBAL-dt maxima that the last stage accumulates; stages run
    // in order, and a restart mid-iteration zeroes the counters on the host
    if (blockIdx.x == 0 && tid == 0) a.counter[(STAGE + 1) % 3] = 0;
    if (STAGE == 1)
        for (int i = blockIdx.x * blockDim.x + tid; i < a.nsmax; i += gridDim.x * blockDim.x) a.smax[i] = 0.f;
    if (tid == 0) {
        mbar_init(mb, 1);
        mbar_init(mbh, 1);
        next_t = atomicAdd(a.counter + STAGE, 1);
        if (next_t < ntiles) tdn = a.tiles[next_t];
        decide();
    }
    __syncthreads();
    for (;;) {
        const int t = s_next;
        if (t == -1) {
            fold();
            break;
        }
        if (t == -2) {
            __syncthreads();   // every thread has read s_next
            if (tid == 0) {
                next_t = atomicAdd(a.counter + STAGE, 1);
                if (next_t < ntiles) tdn = a.tiles[next_t];
                decide();
            }
            __syncthreads();
            continue;
        }
        if (tid == 0) {
            td = tdn;
            if (td.sid != tp_sid) {
                tp = td.sid == tpn_sid ? tpn : a.P[td.sid];
                tp_sid = td.sid;
            }
            // the previous tile's generic accesses of this shared memory are complete (barrier at
            // the end of the loop); order them before the async-proxy writes
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            const TileDesc& d = td;
            const uint32_t brec = 4u * (uint32_t)(5 * d.nrp + 3 * d.ngp), bcsr = 2u * (uint32_t)d.ncsr,
                           bq = 16u * (uint32_t)d.ncore;
            mbar_expect_tx(mb, brec + bcsr + bq);
            tma_load(srec, a.rec + d.rec, brec, mb);
            tma_load(scsr, a.csr + d.csr, bcsr, mb);
            tma_load(cq, Qin + d.c0, bq, mb);
            // L2 prefetches (bulk, asynchronous) of the tile's rows that the gradient and update
            // passes read with plain loads later; rounded out to 16 bytes, inside the arena
            auto pf = [&](const void* p, size_t bytes) {
                const size_t lo = (size_t)p & ~(size_t)15, hi = ((size_t)p + bytes + 15) & ~(size_t)15;
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lo), "r"((uint32_t)(hi - lo)) : "memory");
            };
            const size_t n = (size_t)d.ncore;
            if (tp.order2 && tp.squeeze) { pf(Qprev + d.c0, 16 * n); pf(Gprev + 2 * (size_t)d.c0, 32 * n); }
            if (tp.order2) pf(a.lsq + d.c0, 16 * n);
            pf(a.rvol + d.c0, 4 * n);
            if (STAGE == 0) { pf(a.vol + d.c0, 4 * n); pf(a.S + d.c0, 4 * n); }
            else { pf(a.Q[0] + d.c0, 16 * n); pf(a.D + d.c0, 16 * n); pf(a.dt + d.c0, 4 * n); }
            if (STAGE == 2) pf(a.Qlo + d.c0, 16 * n);
        }
        fold();   // the previous tile's last-stage reductions
        // ---- gather: the ring-1 and ring-2 states (after the halo copy; tdn is this tile's
        // descriptor until thread 0 requests the next one, after the barrier below), while the
        // other blocks are copied
        bool ok = mbar_wait(mbh, parity_h);
        parity_h ^= 1u;
        if (ok) {
            const int nh = tdn.n1 + tdn.n2, o = tdn.ncore, cb = tdn.cbase;
            for (int i = tid; i < nh; i += blockDim.x) cq[o + i] = Qin[cb + shalo[i]];
        }
        if (tid == 0) next_t = atomicAdd(a.counter + STAGE, 1);
        ok = mbar_wait(mb, parity) && ok;
        parity ^= 1u;
        if (__syncthreads_or(!ok)) {
            if (tid == 0) atomicOr(a.err, 2);
            return;
        }

        const int ncore = td.ncore, n1 = td.n1, nrp = td.nrp, ngp = td.ngp;
        const int cbase = td.cbase, c0 = td.c0;
        const Consts<float>& k = tp.k;
        const bool order2 = tp.order2 != 0, ns = tp.ns != 0;
        const bool fresh = STAGE == 0 && tp.fresh != 0, init_prims = STAGE == 0 && tp.init_prims != 0;
        const bool squeeze = tp.squeeze != 0;
        const TileView tv{srec, reinterpret_cast<const float4*>(srec + nrp),
                          reinterpret_cast<const float*>(srec + 5 * nrp),
                          reinterpret_cast<const float*>(srec + 5 * nrp + ngp),
                          reinterpret_cast<const float*>(srec + 5 * nrp + 2 * ngp),
                          scsr, reinterpret_cast<const uint32_t*>(scsr + td.noff), cq, cg, cgy};

        // ---- grad: the limited LSQ gradient of one core or ring-1 cell (local slot gI)
        auto grad_cell = [&](int gI) {
            const int gid = gI < ncore ? c0 + gI : cbase + shalo[gI - ncore];
            const bool lim_prev = squeeze && !fresh;
            // requested first: used only after the loop over the cell's faces
            const float4 mom = a.lsq[gid];
            Q4<float> gpx, gpy;
            if (lim_prev) { gpx = Gprev[2 * (size_t)gid]; gpy = Gprev[2 * (size_t)gid + 1]; }
            Q4<float> gx, gy;
            tile_gradient<true>(tv, k, gI, squeeze, lim_prev, init_prims, STAGE == 0, mom, gpx, gpy,
                          [&](int r) { return Qin[cbase + a.qcell[td.rbase + r]]; }, [&] { return Qprev[gid]; }, gx, gy);
            cg[gI] = gx;
            cgy[gI] = gy;
            if (gI < ncore) { Gout[2 * (size_t)gid] = gx; Gout[2 * (size_t)gid + 1] = gy; }
        };

        // ---- flux of one face of a core cell (record r); V*A - F*A replaces its displacement row
        // and the spectral term its normal's x
        float4* w_t = reinterpret_cast<float4*>(srec + nrp);
        float* w_sp = reinterpret_cast<float*>(srec + 5 * nrp);
        const bool visc = ns && order2;
        auto flux_rec = [&](int r, auto interior) {
            tile_flux<decltype(interior)::value>(tv, k, r, order2, visc, init_prims, STAGE == 2, w_t, w_sp);
        };

        // ---- schedule: core-cell gradients; then the ring-1 gradients on the first warps while the
        // other warps take the fluxes of faces between two core cells (they need core gradients
        // only), which the first warps join when done; then every remaining flux.  Fluxes go to
        // whole warps, td.fpw records at a time (the batch's faces-per-warp tuning), from shared
        // counters.
        if (tid == 0) { s_ctr[0] = 0; s_ctr[1] = 0; }
        if (order2) {
            if (tid == 0 && next_t < ntiles) copy_async(&tdn, a.tiles + next_t);
            // the history flags act only on an iteration's first stage (STAGE 0); the second stage's
            // kernel, which does not read them, clears them for the next iteration: once per solve
            // (the tile of its first cell), in a phase long enough to cover the stores
            if (STAGE == 1 && tid == 0 && c0 == cbase) { a.P[td.sid].fresh = 0; a.P[td.sid].init_prims = 0; }
            if (tid < ncore) grad_cell(tid);
            __syncthreads();
            if (tid == 0 && next_t < ntiles) {   // the next tile's solve parameters, if they change
                asm volatile("cp.async.wait_all;" ::: "memory");
                if (tdn.sid != tp_sid) { copy_async(&tpn, a.P + tdn.sid); tpn_sid = tdn.sid; }
            }
            // the first warps take the ring-1 gradients, then join the others on core-core fluxes
            if (tid < n1) grad_cell(ncore + tid);
            {
                const int fpw = td.fpw, ncc = td.ncc;
                for (;;) {
                    int base = 0;
                    if (lane == 0) base = atomicAdd(&s_ctr[0], fpw);
                    base = __shfl_sync(0xffffffffu, base, 0);
                    if (base >= ncc) break;
                    for (int r = base + lane; r < min(base + fpw, ncc); r += 32) flux_rec(r, std::true_type{});
                }
            }
        } else {
            if (tid == 0 && next_t < ntiles) copy_async(&tdn, a.tiles + next_t);
            if (STAGE == 1 && tid == 0 && c0 == cbase) { a.P[td.sid].fresh = 0; a.P[td.sid].init_prims = 0; }
        }
        __syncthreads();
        if (tid == 0) {   // the next tile: its descriptor checked, its halo list copied (free now)
            if (next_t < ntiles) asm volatile("cp.async.wait_all;" ::: "memory");
            decide();
        }
        {
            const int start = min(s_ctr[0], td.ncc), nrc = td.nrc, fpw = td.fpw, nint = td.nint;
            for (;;) {
                int base = 0;
                if (lane == 0) base = start + atomicAdd(&s_ctr[1], fpw);
                base = __shfl_sync(0xffffffffu, base, 0);
                if (base >= nrc) break;
                for (int r = base + lane; r < min(base + fpw, nrc); r += 32) {
                    if (r < nint) flux_rec(r, std::true_type{});
                    else flux_rec(r, std::false_type{});
                }
            }
        }
        __syncthreads();

        // ---- update: residual gather, time step, SSP-RK3 stage of the core cells
        float snext = 0.f;
        float r2[4] = {0.f, 0.f, 0.f, 0.f};
        if (tid < ncore) {
            const int c = tid, gid = c0 + c;
            // the stage's cell data, requested before the gather
            const float yv = a.rvol[gid];
            float dtc = 0.f, sc = 0.f, vc = 0.f;
            if (STAGE == 0) { vc = a.vol[gid]; if (!tp.global_dt) sc = a.S[gid]; }
            else dtc = a.dt[gid];
            Q4<float> qn, dprev, lo;
            if (STAGE == 0) qn = cq[c];
            else { qn = a.Q[0][gid]; dprev = a.D[gid]; }
            if (STAGE == 2) lo = a.Qlo[gid];
            float r4[4];
            tile_residual(tv, c, w_t, w_sp, STAGE == 2, yv, r4, snext);
            if (a.R && (a.store_r || STAGE == 2)) { Q4<float> rr; for (int j = 0; j < 4; j++) rr.p[j] = r4[j]; a.R[gid] = rr; }
            if (STAGE == 0) {
                dtc = fm(k.two_cfl, vc) / (tp.global_dt ? a.smax[td.sid] : sc);
                a.dt[gid] = dtc;
            }
            Q4<float> out, dn;
            stage_combine(STAGE, dtc, r4, qn, dprev, lo, dn, out);
            if (STAGE == 0) {
                a.D[gid] = dn;
                a.Q[1][gid] = out;
            } else if (STAGE == 1) {
                a.D[gid] = dn;
                a.Q[2][gid] = out;
            } else {
                a.Q[0][gid] = out;
                a.Qlo[gid] = lo;
                a.S[gid] = snext;
#pragma unroll
                for (int j = 0; j < 4; j++) r2[j] = r4[j] * r4[j];
            }
            if (!positive(out.p[0]) || !positive(out.p[3])) atomicOr(a.flags + td.sid, 1);
        }
        if (STAGE == 2) {
            // per warp: the spectral maximum (GLOBAL dt of the next iteration) and, for a batch, the
            // residual sums of squares (its per-solve norms), squares and sums in FP32; the warps'
            // values are folded at the next tile's top (fold: fixed order, FP64 across warps; GB300's
            // FP64 unit is narrow, so only four lanes of one warp do FP64 arithmetic)
            float m = snext;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = max2(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (a.tpart) {
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) r2[j] += __shfl_xor_sync(0xffffffffu, r2[j], o);
            }
            if (lane == 0) {
                redf[warp] = m;
#pragma unroll
                for (int j = 0; j < 4; j++) redw[j][warp] = r2[j];
            }
            red_t = t;
            red_sid = td.sid;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------
// A stage of first-order solves (when every solve of the launch is one): the fluxes and the update,
// without what only gradients need.  Such a stage is bound by latency (the descriptor, the blocks' copies,
// the ring gather, each a round trip to L2) and has little arithmetic to hide it behind, so it takes
// more, smaller CTAs: a tile's slots, normals, areas and the core cells' csr rows are 40 KB where the
// general kernel's blocks and gradient rows are 73 KB, and with four CTAs of 64 registers on an SM instead
// of three one's copies run under another's fluxes.  One CTA per tile, no counter; each stage is launched while
// the one before it runs (programmatic launch, triggered when every CTA of that one has started) and has
// copied what no kernel writes when that ends.  A tile's RK data is requested with its states, before the fluxes.
// Against the general kernel: 300k Euler polygons 62.9 -> 29.4 us per iteration, 1M quads 137 -> 99
// (about 145 B per cell and stage: 4.4 TB/s), 130k NS cylinder 45.2 -> 19.5; the same bits.
// The choices, measured on 300k Euler polygons when the kernel took 31.7 (its records not yet ordered for the
// banks): three CTAs per SM 37.3, five with spills 35.7; no early trigger 34.8; with five CTAs also no early
// trigger 37.8, no programmatic launches 39.0.
struct TFirst {
    int flux;                  // records with fluxes of the largest tile, rounded up to 4
    int grad;                  // core and ring-1 cells of the largest tile
};
// Shared memory (bytes) of that plan: slots, normals and areas, contributions, csr, states.
__host__ __device__ constexpr int first_smem(int flux, int grad) {
    return 16 * flux + 16 * flux + 2 * (kTileCore + 8) + 8 * flux + 16 * grad;
}
static_assert(first_smem(kTileGeo, kTileGrad) <= 47 * 1024, "within the limit of a plain launch");

template <int STAGE>
__global__ void __launch_bounds__(kTileCore, 4) k_tfirst(TArgs a, TFirst f) {
    extern __shared__ __align__(128) unsigned char sm[];
    float4* w_t = reinterpret_cast<float4*>(sm);
    Q4<float>* cq = reinterpret_cast<Q4<float>*>(sm + 16 * f.flux);
    uint32_t* ssl = reinterpret_cast<uint32_t*>(sm + 16 * f.flux + 16 * f.grad);
    float* snx = reinterpret_cast<float*>(ssl + f.flux);
    float* sny = snx + f.flux;
    float* sA = sny + f.flux;
    uint32_t* sent = reinterpret_cast<uint32_t*>(sA + f.flux);
    uint16_t* soff = reinterpret_cast<uint16_t*>(sent + 2 * f.flux);
    __shared__ __align__(16) TileDesc td;
    __shared__ __align__(16) TParams tp;
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ float redf[kTileCore / 32];
    __shared__ float redw[4][kTileCore / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, t = blockIdx.x;
    const uint32_t mb = smem_u32(&mbar);
    if (t >= *a.ntiles) { pdl_wait(); return; }
    if (tid < (int)(sizeof(TileDesc) / 16))
        reinterpret_cast<int4*>(&td)[tid] = reinterpret_cast<const int4*>(a.tiles + t)[tid];
    if (tid == 0) mbar_init(mb, 1);
    __syncthreads();
    const TileDesc& d = td;
    const int nrc = d.nrc, nrc4 = (nrc + 3) & ~3, ncore = d.ncore, n1 = d.n1, ne4 = (nrc + d.ncc + 3) & ~3;
    const int nof = (ncore + 1 + 7) & ~7;
    if (ncore == 0) { pdl_wait(); return; }   // an empty slot of a removed solve
    const bool ok = ncore > 0 && ncore <= kTileCore && n1 >= 0 && ncore + n1 <= f.grad && nrc >= 0 && nrc4 <= f.flux &&
                    d.ncc >= 0 && d.ncc <= d.nint && d.nint <= nrc && nrc <= d.ngeo && d.ngeo <= d.nr && d.nrp >= nrc4 &&
                    d.ngp >= nrc4 && nof <= d.noff && d.noff + 2 * ne4 <= d.ncsr && n1 <= d.nhalo && (d.nrp & 3) == 0 &&
                    (d.ngp & 3) == 0 && (d.noff & 7) == 0 && (d.rec & 3) == 0 && (d.csr & 7) == 0;
    if (!ok) {
        if (tid == 0) atomicOr(a.err, 4);
        pdl_wait();
        return;
    }
    // what no kernel writes: the records, the csr rows and the halo ids
    if (tid == 0) {
        const uint32_t br = 4u * (uint32_t)nrc4, be = 4u * (uint32_t)ne4, bo = 2u * (uint32_t)nof;
        mbar_expect_tx(mb, 4 * br + be + bo);
        const uint32_t* rec = a.rec + d.rec;
        const uint16_t* csr = a.csr + d.csr;
        if (br) {
            tma_load(ssl, rec, br, mb);
            tma_load(snx, rec + 5 * d.nrp, br, mb);
            tma_load(sny, rec + 5 * d.nrp + d.ngp, br, mb);
            tma_load(sA, rec + 5 * d.nrp + 2 * d.ngp, br, mb);
            tma_load(sent, csr + d.noff, be, mb);
        }
        tma_load(soff, csr, bo, mb);
    }
    const int c0 = d.c0, cbase = d.cbase, gid = c0 + tid;
    const int hid = tid < n1 ? a.halo[d.halo + tid] : 0;
    float yv = 1.f, vc = 0.f;
    if (tid < ncore) {
        yv = a.rvol[gid];
        if (STAGE == 0) vc = a.vol[gid];
    }
    pdl_wait();   // from here on, what the stages before this one wrote
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const Q4<float>* Qin = a.Q[STAGE];   // not __restrict__: it changes while this kernel is resident
    if (tid >= kTileCore - (int)(sizeof(TParams) / 16))
        reinterpret_cast<int4*>(&tp)[tid - (kTileCore - (int)(sizeof(TParams) / 16))] =
            reinterpret_cast<const int4*>(a.P + d.sid)[tid - (kTileCore - (int)(sizeof(TParams) / 16))];
    Q4<float> qn, dprev, lo;
    float dtc = 0.f, sc = 0.f;
    if (tid < ncore) {
        const Q4<float> q = Qin[gid];
        cq[tid] = q;
        if (STAGE == 0) { qn = q; sc = a.S[gid]; }
        else { qn = a.Q[0][gid]; dprev = a.D[gid]; dtc = a.dt[gid]; }
        if (STAGE == 2) lo = a.Qlo[gid];
    }
    if (tid < n1) cq[ncore + tid] = Qin[cbase + hid];
    for (int i = tid + kTileCore; i < n1; i += kTileCore) cq[ncore + i] = Qin[cbase + a.halo[d.halo + i]];
    const bool arrived = mbar_wait(mb, 0);
    if (__syncthreads_or(!arrived)) {
        if (tid == 0) atomicOr(a.err, 2);
        return;
    }
    const Consts<float>& k = tp.k;
    const bool init_prims = STAGE == 0 && tp.init_prims != 0;
    float* w_sp = snx;   // the spectral term replaces the normal's x
    const TileView tv{ssl, nullptr, snx, sny, sA, soff, sent, cq, nullptr, nullptr};
    for (int r = tid; r < nrc; r += kTileCore) {
        if (r < d.nint) tile_flux<true, true>(tv, k, r, false, false, init_prims, STAGE == 2, w_t, w_sp);
        else tile_flux<false, true>(tv, k, r, false, false, init_prims, STAGE == 2, w_t, w_sp);
    }
    if (STAGE == 1 && tid == 0 && c0 == cbase) {
        // the solve's first tile: its GLOBAL-dt maximum (read in the first stage, accumulated in the
        // last) starts again; its history flags (read in the first stage) end
        a.smax[d.sid] = 0.f;
        a.P[d.sid].fresh = 0;
        a.P[d.sid].init_prims = 0;
    }
    __syncthreads();
    float snext = 0.f;
    float r2[4] = {0.f, 0.f, 0.f, 0.f};
    if (tid < ncore) {
        float r4[4];
        tile_residual(tv, tid, w_t, w_sp, STAGE == 2, yv, r4, snext);
        if (a.R && (a.store_r || STAGE == 2)) { Q4<float> rr; for (int j = 0; j < 4; j++) rr.p[j] = r4[j]; a.R[gid] = rr; }
        if (STAGE == 0) {
            dtc = fm(k.two_cfl, vc) / (tp.global_dt ? a.smax[d.sid] : sc);
            a.dt[gid] = dtc;
        }
        Q4<float> out, dn;
        stage_combine(STAGE, dtc, r4, qn, dprev, lo, dn, out);
        if (STAGE != 2) {
            a.D[gid] = dn;
            a.Q[STAGE + 1][gid] = out;
        } else {
            a.Q[0][gid] = out;
            a.Qlo[gid] = lo;
            a.S[gid] = snext;
#pragma unroll
            for (int j = 0; j < 4; j++) r2[j] = r4[j] * r4[j];
        }
        if (!positive(out.p[0]) || !positive(out.p[3])) atomicOr(a.flags + d.sid, 1);
    }
    if (STAGE == 2) {   // maxima and sums as the general kernel's: per warp, then over the warps in order
        float m = snext;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = max2(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (a.tpart) {
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) r2[j] += __shfl_xor_sync(0xffffffffu, r2[j], o);
        }
        if (lane == 0) {
            redf[warp] = m;
#pragma unroll
            for (int j = 0; j < 4; j++) redw[j][warp] = r2[j];
        }
        __syncthreads();
        if (a.tpart && tid < 4) {
            double sum = 0.0;
            for (int w = 0; w < kTileCore / 32; w++) sum += (double)redw[tid][w];
            a.tpart[4 * (size_t)t + tid] = sum;
        }
        if (tid == 32) {
            float bm = 0.f;
            for (int w = 0; w < kTileCore / 32; w++) bm = max2(bm, redf[w]);
            atomic_max_pos(a.smax + d.sid, bm);
        }
    }
}

// ------------------------------------------------------------------------------------------
// Whole iterations in one launch, for solves whose tiles all fit on the GPU at once (one tile per
// CTA, a cooperative launch): a tile's records, csr and halo list are copied to shared memory once
// per launch, its states and limited gradients stay there from stage to stage, its cells' RK data in
// registers; the tiles exchange only their new states, through L2, with one grid barrier per stage.
// Such a solve is bound by latency, not by any unit: with a stage kernel per stage it spends ~15 us a
// stage on the launch, the tile's block copies and a 256-cell tile's passes on a third of the SMs.
// Here a stage is the barrier and the ring gather (~1.5 us), one round of gradients and fluxes and
// the update: 12k-cell NS cylinder 45.1 -> 16.1 us per iteration, 50k Euler polygons 42.5 -> 19.2, 512
// quads 26.6 -> 11.7.  What the passes read every stage (LSQ moments, previous states) is kept in shared
// memory too, since the barrier's acquire empties L1 (the 12k-cell cylinder: 19.8 -> 16.7
// us when it was added, with a barrier that has no fences beyond its release and acquire).  MINB 2 has the
// registers to run without spills; MINB 3 (128 B of spills) takes the solves whose tiles do not fit two to
// an SM.  First-order solves alone do not come here (k_tfirst); in a batch with others they do.
struct TIter {
    int iterations;
    unsigned bar0;             // the barrier's value when the launch starts
    unsigned* bar;             // arrivals so far (monotone, wraps)
    int o_csr, o_halo, o_cq, o_cg, o_t, o_sp, o_qp, o_lsq;   // shared-memory regions (bytes; the record block is at 0)
    int max_rec, max_csr, max_halo, max_cells, max_grad, max_flux;   // and what they hold (TileLayout's maxima)
};

// A state from L2 (the SM's own L1 does not see other SMs' writes).
__device__ __forceinline__ Q4<float> ldcg_q(const Q4<float>* p) {
    const float4 x = __ldcg(reinterpret_cast<const float4*>(p));
    Q4<float> q;
    q.p[0] = x.x; q.p[1] = x.y; q.p[2] = x.z; q.p[3] = x.w;
    return q;
}

// Barrier over the grid of a cooperative launch (every CTA is resident): all writes of every CTA
// before it are visible after it.  Bounded: false (in every thread of the CTA) when the others have
// not arrived after 2^23 polls (seconds: far longer than any stage takes, with room for other
// kernels that hold some of the SMs when the grid is launched).
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned target) {
    __syncthreads();
    int bad = 0;
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        int polls = 0;
        for (;;) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if ((int)(v - target) >= 0) break;
            if (++polls > (1 << 23)) { bad = 1; break; }
        }
    }
    return !__syncthreads_or(bad);
}

template <int MINB>
__global__ void __launch_bounds__(kTileCore, MINB) k_titer(TArgs a, TIter it) {
    extern __shared__ __align__(128) unsigned char sm[];
    uint32_t* srec = reinterpret_cast<uint32_t*>(sm);
    uint16_t* scsr = reinterpret_cast<uint16_t*>(sm + it.o_csr);
    int* shalo = reinterpret_cast<int*>(sm + it.o_halo);
    Q4<float>* cq = reinterpret_cast<Q4<float>*>(sm + it.o_cq);
    Q4<float>* cg = reinterpret_cast<Q4<float>*>(sm + it.o_cg);
    Q4<float>* cgy = cg + it.max_grad;
    float4* w_t = reinterpret_cast<float4*>(sm + it.o_t);
    float* w_sp = reinterpret_cast<float*>(sm + it.o_sp);
    Q4<float>* sqp = reinterpret_cast<Q4<float>*>(sm + it.o_qp);      // previous stage's states
    float4* slsq = reinterpret_cast<float4*>(sm + it.o_lsq);          // LSQ moments
    __shared__ __align__(16) TileDesc td;
    __shared__ __align__(16) TParams tp;
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ float redw[4][kTileCore / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t mb = smem_u32(&mbar);
    const int t = blockIdx.x;
    if (tid == 0) {
        td = a.tiles[t];
        mbar_init(mb, 1);
    }
    __syncthreads();
    // an empty slot (a removed solve's) or a descriptor outside the plan only takes part in the barriers
    const TileDesc& d = td;
    const bool live = d.ncore > 0 && d.ncore <= kTileCore && d.n1 >= 0 && d.n2 >= 0 && d.ncore + d.n1 <= it.max_grad &&
                      d.ncore + d.n1 + d.n2 <= it.max_cells && d.nrc <= it.max_flux && d.nint >= 0 && d.nint <= d.nrc &&
                      d.nrc <= d.ngeo && d.ngeo <= d.nr && d.nrp >= d.nr && d.ngp >= d.ngeo &&
                      5 * d.nrp + 3 * d.ngp <= it.max_rec && d.ncsr <= it.max_csr && d.noff <= d.ncsr &&
                      d.n1 + d.n2 <= d.nhalo && d.nhalo <= it.max_halo && (d.nrp & 3) == 0 && (d.ngp & 3) == 0 &&
                      (d.ncsr & 7) == 0 && (d.nhalo & 3) == 0 && (d.rec & 3) == 0 && (d.csr & 7) == 0 && (d.halo & 3) == 0;
    if (!live && d.ncore != 0 && tid == 0) atomicOr(a.err, 4);
    if (live) {
        if (tid == 0) {
            tp = a.P[d.sid];
            const uint32_t brec = 4u * (uint32_t)(5 * d.nrp + 3 * d.ngp), bcsr = 2u * (uint32_t)d.ncsr,
                           bhal = 4u * (uint32_t)d.nhalo;
            mbar_expect_tx(mb, brec + bcsr + bhal);
            tma_load(srec, a.rec + d.rec, brec, mb);
            tma_load(scsr, a.csr + d.csr, bcsr, mb);
            if (bhal) tma_load(shalo, a.halo + d.halo, bhal, mb);
        }
        const bool ok = mbar_wait(mb, 0);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) atomicOr(a.err, 2);
            return;
        }
    }
    const int ncore = live ? d.ncore : 0, n1 = live ? d.n1 : 0, nh = live ? n1 + d.n2 : 0;
    const int cbase = d.cbase, c0 = d.c0, nrp = d.nrp, ngp = d.ngp, nrc = live ? d.nrc : 0, nint = d.nint, sid = d.sid;
    const Consts<float>& k = tp.k;
    const bool order2 = live && tp.order2 != 0, visc = order2 && tp.ns != 0, squeeze = tp.squeeze != 0;
    const TileView tv{srec, reinterpret_cast<const float4*>(srec + nrp), reinterpret_cast<const float*>(srec + 5 * nrp),
                      reinterpret_cast<const float*>(srec + 5 * nrp + ngp),
                      reinterpret_cast<const float*>(srec + 5 * nrp + 2 * ngp), scsr,
                      reinterpret_cast<const uint32_t*>(scsr + d.noff), cq, cg, cgy};
    // the core cells' RK data
    const int gid = c0 + tid;
    Q4<float> qn, lo, dinc;
    float dtc = 0.f, sc = 0.f, vc = 1.f, yv = 1.f;
#pragma unroll
    for (int j = 0; j < 4; j++) { qn.p[j] = 0.f; lo.p[j] = 0.f; dinc.p[j] = 0.f; }
    if (tid < ncore) {
        qn = a.Q[0][gid];
        cq[tid] = qn;
        lo = a.Qlo[gid];
        sc = a.S[gid];
        vc = a.vol[gid];
        yv = a.rvol[gid];
    }
    if (order2)
        for (int gI = tid; gI < ncore + n1; gI += blockDim.x) {
            const int g = gI < ncore ? c0 + gI : cbase + shalo[gI - ncore];
            slsq[gI] = a.lsq[g];
            if (squeeze) {
                sqp[gI] = a.Q[2][g];
                cg[gI] = a.G[2][2 * (size_t)g];
                cgy[gI] = a.G[2][2 * (size_t)g + 1];
            }
        }
    unsigned target = it.bar0;
    for (int i = 0; i < it.iterations; i++) {
        const bool final = i == it.iterations - 1;
#pragma unroll 1
        for (int s = 0; s < 3; s++) {
            const Q4<float>* Qin = s == 0 ? a.Q[0] : s == 1 ? a.Q[1] : a.Q[2];
            const bool begin = i == 0 && s == 0;      // the previous stage ran in an earlier launch
            const bool fresh = begin && tp.fresh != 0, init_prims = begin && tp.init_prims != 0;
            // ---- gather: the ring cells' states (ring 2 only for gradients)
            for (int h = tid; h < (order2 ? nh : n1); h += blockDim.x) cq[ncore + h] = ldcg_q(Qin + cbase + shalo[h]);
            const float smax = s == 0 && live && tp.global_dt ? __ldcg(a.smax + sid) : 0.f;
            __syncthreads();
            // ---- gradients
            if (order2) {
                Q4<float>* Gout = s == 0 ? a.G[0] : s == 1 ? a.G[1] : a.G[2];
                const bool lim_prev = squeeze && !fresh;
                for (int gI = tid; gI < ncore + n1; gI += blockDim.x) {
                    Q4<float> gpx, gpy, gx, gy;
                    if (lim_prev) { gpx = cg[gI]; gpy = cgy[gI]; }
                    tile_gradient<false>(tv, k, gI, squeeze, lim_prev, init_prims, s == 0, slsq[gI], gpx, gpy,
                                  [&](int r) { return ldcg_q(Qin + cbase + a.qcell[td.rbase + r]); }, [&] { return sqp[gI]; }, gx, gy);
                    cg[gI] = gx;
                    cgy[gI] = gy;
                    sqp[gI] = cq[gI];
                    if (final && gI < ncore) { Gout[2 * (size_t)(c0 + gI)] = gx; Gout[2 * (size_t)(c0 + gI) + 1] = gy; }
                }
                __syncthreads();
            }
            // ---- fluxes
            for (int r = tid; r < nrc; r += blockDim.x) {
                if (r < nint) tile_flux<true>(tv, k, r, order2, visc, init_prims, s == 2, w_t, w_sp);
                else tile_flux<false>(tv, k, r, order2, visc, init_prims, s == 2, w_t, w_sp);
            }
            __syncthreads();
            // ---- update
            float snext = 0.f;
            float r2[4] = {0.f, 0.f, 0.f, 0.f};
            if (tid < ncore) {
                float r4[4];
                tile_residual(tv, tid, w_t, w_sp, s == 2, yv, r4, snext);
                if (final && a.R && s == 2) { Q4<float> rr; for (int j = 0; j < 4; j++) rr.p[j] = r4[j]; a.R[gid] = rr; }
                if (s == 0) {
                    dtc = fm(k.two_cfl, vc) / (tp.global_dt ? smax : sc);
                    if (final) a.dt[gid] = dtc;
                }
                Q4<float> out, dn = dinc;
                stage_combine(s, dtc, r4, qn, dinc, lo, dn, out);
                dinc = dn;
                (s == 0 ? a.Q[1] : s == 1 ? a.Q[2] : a.Q[0])[gid] = out;
                cq[tid] = out;
                if (s == 2) {
                    qn = out;
                    sc = snext;
                    if (final) { a.Qlo[gid] = lo; a.S[gid] = sc; }
#pragma unroll
                    for (int j = 0; j < 4; j++) r2[j] = r4[j] * r4[j];
                }
                if (!positive(out.p[0]) || !positive(out.p[3])) atomicOr(a.flags + sid, 1);
            }
            if (s == 1 && tid == 0 && live && c0 == cbase) {
                // the solve's first tile: its GLOBAL-dt maximum (read in the first stage, accumulated in
                // the last) starts again; its history flags (read before the first barrier) end
                a.smax[sid] = 0.f;
                if (i == 0) { a.P[sid].fresh = 0; a.P[sid].init_prims = 0; }
            }
            if (s == 2 && live) {
                float m = snext;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) m = max2(m, __shfl_xor_sync(0xffffffffu, m, o));
                if (lane == 0 && 32 * warp < ncore) atomic_max_pos(a.smax + sid, m);
                if (a.tpart && final) {   // as the stage kernel: FP32 per warp, FP64 over the warps in order
#pragma unroll
                    for (int j = 0; j < 4; j++)
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) r2[j] += __shfl_xor_sync(0xffffffffu, r2[j], o);
                    if (lane == 0)
#pragma unroll
                        for (int j = 0; j < 4; j++) redw[j][warp] = r2[j];
                    __syncthreads();
                    if (tid < 4) {
                        double sum = 0.0;
                        for (int w = 0; w < kTileCore / 32; w++) sum += (double)redw[tid][w];
                        a.tpart[4 * (size_t)t + tid] = sum;
                    }
                }
            }
            if (final && s == 2) break;
            target += gridDim.x;
            if (!grid_barrier(it.bar, target)) {
                if (tid == 0) atomicOr(a.err, 8);
                return;
            }
        }
    }
}

// Initial spectral sums of a solve's tiles (the initial Vn_avg, c_avg of every face,
// class_q.hpp:61-62) in each cell's csr order, and their maximum.
__global__ void __launch_bounds__(kTileCore) k_tspec_init(const TileDesc* __restrict__ tiles, int first, int count,
                                                        const uint32_t* __restrict__ rec, const uint16_t* __restrict__ csr,
                                                        const TParams* __restrict__ P, float* __restrict__ S,
                                                        float* __restrict__ smax) {
    __shared__ float red[kTileCore / 32];
    for (int t = first + blockIdx.x; t < first + count; t += gridDim.x) {
        const TileDesc d = tiles[t];
        const Consts<float>& k = P[d.sid].k;
        float s = 0.f;
        if ((int)threadIdx.x < d.ncore) {
            const uint16_t* off = csr + d.csr;
            const uint16_t* ent = off + d.noff;
            const float* A = reinterpret_cast<const float*>(rec + d.rec + 5 * (size_t)d.nrp + 2 * (size_t)d.ngp);
            for (int e = off[threadIdx.x] & 0x7FFF; e < (off[threadIdx.x + 1] & 0x7FFF); e++) s += (fabsf(k.vn0) + k.c0) * A[ent[2 * e] >> 1];
            S[d.c0 + threadIdx.x] = s;
        }
        float m = s;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = max2(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
        __syncthreads();
        if (threadIdx.x == 0) {
            float bm = 0.f;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) bm = max2(bm, red[w]);
            atomic_max_pos(smax + d.sid, bm);
        }
        __syncthreads();
    }
}

// Per-solve residual sums of squares: solve s owns tiles [srange[2s], srange[2s] + srange[2s+1]);
// one block per solve slot adds their per-tile sums in a fixed order.
__global__ void __launch_bounds__(256) k_tres_norm(const int* __restrict__ srange, const double* __restrict__ tpart,
                                                   double* __restrict__ res2) {
    __shared__ double sh[4][256];
    const int s = blockIdx.x, first = srange[2 * s], n = srange[2 * s + 1];
    double acc[4] = {0, 0, 0, 0};
    for (int i = threadIdx.x; i < n; i += blockDim.x)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[j] += tpart[4 * (size_t)(first + i) + j];
#pragma unroll
    for (int j = 0; j < 4; j++) sh[j][threadIdx.x] = acc[j];
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h)
#pragma unroll
            for (int j = 0; j < 4; j++) sh[j][threadIdx.x] += sh[j][threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0)
#pragma unroll
        for (int j = 0; j < 4; j++) res2[4 * s + j] = sh[j][0];
}

}  // namespace fv2d
