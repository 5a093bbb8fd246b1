// Device kernels of the fv2d residual-and-update step, FP64 engine (and the state transfers and small
// helpers both precisions share, templated on the state type T).
//
// One RK stage = three launches:
//   k_gradient  (four lanes per cell)  LSQ gradient over the cell's faces + squeeze limiter, one
//                                      component per lane
//   k_face      (one thread per face;  reconstruction, boundary ghosts, NS face terms, Rusanov
//    k_face_pair: two lanes)           flux; writes the face's residual contribution
//   k_update    (four lanes per cell)  gathers the face contributions in ascending original face
//                                      id, divides by the volume, applies the SSP-RK3 stage, and
//                                      (last stage) the spectral sums for the next time step
// Every per-cell sum visits the cell's faces in ascending ORIGINAL face id, the order in which
// the reference's face loops scatter into the cell, so with FMA contraction off (-fmad=false) the
// results are bit-identical to the reference; no atomics touch the state.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace fv2d {

template <class T>
struct alignas(4 * sizeof(T)) Q4 {
    T p[4];
};

template <class T>
struct Consts {
    T gamma, gm1, R, mu, k;            // gm1 = gamma - 1, k = mu*Cp/Pr (class_flow.hpp:36-40)
    T q_inf[4];                        // freestream conservative state (class_flow.hpp:28-34)
    T rho_inf, u_inf, v_inf, P_inf;    // freestream primitives (initial Qbar primitives)
    T two_cfl;                         // 2*CFL
    T vn0, c0;                         // initial Vn_avg, c_avg (class_q.hpp:61-62)
    // flux_solver = ROE: the reference's res() calls no flux routine (res.cpp:62-69), so the
    // inviscid flux of every face is class_F::init's -101 (class_f.hpp:26-30) and Vn_avg, c_avg
    // (the time step's spectral terms) keep their initial values
    int roe;
};

// Face geometry, SoA, device order.
template <class T>
struct FaceGeo {
    const T *nx, *ny, *area, *c1dx, *c1dy, *c2dx, *c2dy, *dxj, *dyj, *mx, *my, *lx, *ly, *dist;
};

// Every mesh array a stage reads, device order (single solve) or arena order (batch).
template <class T>
struct DevMesh {
    const int *inc_off, *inc, *nbr, *fc1, *fc2, *qcell;
    const Q4<T>* igeo;   // per incidence (CSR order): dxj, dyj, offset of the face centre from the cell
    FaceGeo<T> g;
    const double *Ixx, *Iyy, *Ixy;
    const T* vol;
    // geometry-only reciprocals, computed once (k_reciprocals) with the same Recip<T>::of the kernels
    // would evaluate every stage: 1/|dist| per face (NS interior faces), 1/vol per cell
    const T *rdist, *rvol;
    // reconstructed face states of the last face pass, [2 nf]: 2f + side (the incidence code) holds
    // the state on cell c1's (side 0) or c2's (side 1) side of face f - exactly the stale face
    // values the next squeeze reads.  Null where no squeeze follows.
    Q4<T>* fval;
};

template <class T>
__device__ __forceinline__ Q4<T> ldq(const Q4<T>* a, int i) {
    return a[i];
}

// Programmatic dependent launch: a stage kernel loads what no kernel writes (the mesh), waits for the
// kernel before it and then lets the next one's CTAs start.  So at most two kernels are in flight, and
// a waiting kernel's SM reads nothing that the running one writes.  (The arrays that kernels write are
// not __restrict__ const: they change while a waiting kernel is resident, so its loads of them must not
// go by the read-only path.)
struct Prior {
    __device__ __forceinline__ void operator()() const {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
};
struct NoWait {
    __device__ __forceinline__ void operator()() const {}
};

// Ordered comparison a < b.  For doubles it runs on the integer pipe: a non-NaN double's bit
// pattern, with -0 folded onto +0 and the magnitude bits of negatives inverted, orders exactly as
// IEEE '<' (equal values, +0 and -0 included, give equal keys), and the compare and select issue on
// the integer ALU pipe instead of taking a DSETP slot on GB300's narrow FP64 pipe.  (NaN inputs,
// which only arise in states already flagged as non-physical, may order differently.)
__device__ __forceinline__ long long order_key(double x) {
    long long b = __double_as_longlong(x);
    b = (b == (long long)0x8000000000000000ULL) ? 0LL : b;
    return b ^ ((b >> 63) & 0x7FFFFFFFFFFFFFFFLL);
}
template <class T>
__device__ __forceinline__ bool less(T a, T b) { return a < b; }
template <>
__device__ __forceinline__ bool less<double>(double a, double b) { return order_key(a) < order_key(b); }

// std::min({a, b}) / std::max({a, b}) semantics (first argument wins ties)
template <class T>
__device__ __forceinline__ T min2(T a, T b) { return less(b, a) ? b : a; }
template <class T>
__device__ __forceinline__ T max2(T a, T b) { return less(a, b) ? b : a; }

// Division sharing one reciprocal between several quotients with the same denominator.
// FP64: y = RN(1/b) (__drcp_rn), then two of Markstein's residual corrections
// (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34(1), 1990): q0 = RN(a*y) is within 1.5 ulp of a/b, the first correction
// q1 = q0 + RN(a - b*q0)*y brings it within 1 ulp, and with that faithful q1 the residual
// a - b*q1 is exact and q2 = RN(q1 + (a - b*q1)*y) is the correctly rounded a/b.  Valid for
// normal operands whose quotient neither overflows nor underflows (all solver quantities); a zero
// numerator (checked on its bits, not with an FP64 compare) returns the exact signed zero a*y.
// Tested bit for bit against IEEE division.
template <class T>
struct Recip;
template <>
struct Recip<double> {
    static __device__ __forceinline__ double of(double b) { return __drcp_rn(b); }
    static __device__ __forceinline__ double div(double a, double b, double y) {
        const double q0 = a * y;
        if ((__double_as_longlong(a) << 1) == 0) return q0;   // a == +-0, tested on the integer pipe
        const double q1 = __fma_rn(__fma_rn(-b, q0, a), y, q0);
        return __fma_rn(__fma_rn(-b, q1, a), y, q1);
    }
};

// a/3: one residual correction suffices for this divisor (two are needed in general).
// y = RN(1/3) = 1/3 (1 - 2^-54), so a*y is within half an ulp of a/3 and q0 = RN(a*y) is faithful;
// r = a - 3 q0 is then exact (an integer multiple of ulp(q0), below 3 ulp), and q0 + r*y is within
// 2^-53 ulp of a/3.  a/3 lies at least ulp/6 from every rounding midpoint (a - 3m, m a midpoint,
// is a non-zero multiple of ulp/2), so RN(q0 + r*y) is the correctly rounded a/3.  Checked against
// IEEE division on the host (tests/cpu_helpers/div3_check.cpp).
__device__ __forceinline__ double div3(double a) {
    const double y = 1.0 / 3.0, q0 = a * y;
    if ((__double_as_longlong(a) << 1) == 0) return q0;   // a == +-0
    return __fma_rn(__fma_rn(-3.0, q0, a), y, q0);
}

// FP64 arithmetic as fused multiply-adds of vector registers.  GB300's FP64 pipe takes a warp's DFMA
// with three vector-register operands every 16 cycles per SM, but a DADD, a DMUL, or a DFMA with a
// constant, immediate or uniform-register operand only every 19 (measured with 1,000 operations per
// thread, 4 to 32 warps on an SM).  So sums and products go as a*1 + b and a*b + (-0), which round
// exactly as a + b and a*b do, signed zeros included: a*1 is exact, and adding -0 changes no value and
// no zero's sign.  The constants have to come from memory: from literals or kernel parameters the
// compiler rebuilds the slower forms.
// Together with the exact scalings of face_flux, on the 1M-cell NS cylinder: face kernel 2.20 -> 1.76 ms
// (FP64 pipe busy 95 % of the time); with the component lanes of the cell passes gradient 0.459 -> 0.431,
// update 0.141 -> 0.146 (below), 8.37 -> 6.99 ms per iteration.
// half: a factor of 1/2 enters through the multiply-add that uses it (x - m/2 = fma(m, -1/2, x), as
// m/2 is exact), so it costs no operation of its own.
__device__ double g_fp64_consts[4] = {1.0, -0.0, 0.5, 0.25};
struct Fp {
    double one, nz, half;
    __device__ __forceinline__ Fp() {
        one = g_fp64_consts[0];
        nz = g_fp64_consts[1];
        half = g_fp64_consts[2];
    }
    __device__ __forceinline__ double add(double a, double b) const { return __fma_rn(a, one, b); }
    __device__ __forceinline__ double sub(double a, double b) const { return __fma_rn(a, one, -b); }
    __device__ __forceinline__ double mul(double a, double b) const { return __fma_rn(a, b, nz); }
};

// Several quotients by one denominator b: y = RN(1/b) and yl the digits of 1/b after it, so that
// q0 = RN(a*y + RN(a*yl)) is a/b within 2^-50 ulp before its rounding, hence faithful; then the residual
// a - b*q0 is exact and q0 + (a - b*q0)*y rounds to the correctly rounded a/b (Markstein, as above:
// y correctly rounded, q0 faithful).  Four operations a quotient and two per denominator, against
// five for the two residual corrections of Recip.  Same operand range; a zero numerator gives the exact
// signed zero, or NaN over a zero.  Tested bit for bit against IEEE division.
struct Divisor {
    double b, y, yl;
    int z;   // high word of +0 / b: b's sign, over NaN's bits where b is a zero (a state of no density is then flagged)
    __device__ __forceinline__ Divisor(double b_, double y_, const Fp& f) {
        b = b_;
        y = y_;
        yl = f.mul(__fma_rn(-b_, y_, f.one), y_);
        const int hb = __double2hiint(b_);
        z = (hb & (int)0x80000000) | (((hb << 1) | __double2loint(b_)) == 0 ? 0x7FF80000 : 0);
    }
    __device__ __forceinline__ Divisor(double b_, const Fp& f) : Divisor(b_, Recip<double>::of(b_), f) {}
    __device__ __forceinline__ double div(double a, const Fp& f) const {
        const double q0 = __fma_rn(a, y, f.mul(a, yl));
        const double q = __fma_rn(__fma_rn(-b, q0, a), y, q0);
        const int ha = __double2hiint(a);
        const bool zero = ((ha << 1) | __double2loint(a)) == 0;
        return zero ? __hiloint2double((ha & (int)0x80000000) ^ z, 0) : q;
    }
};

// +0 - x, IEEE round to nearest, for a term (V A) that is identically +0 (V = +0, area A >= +0):
// -x, and +0 when x is a zero of either sign
__device__ __forceinline__ double zero_minus(double x) {
    const long long b = __double_as_longlong(x) ^ (long long)0x8000000000000000ULL;
    return (b << 1) == 0 ? 0.0 : __longlong_as_double(b);
}

// Primitives of one state (class_Q::updateflow, class_q.hpp:131-141; T, the temperature, is never read by the
// step and is not formed): rho's divisor is shared by u and v, and returned for P/rho.
__device__ __forceinline__ Divisor prims_r(const double p[4], const Consts<double>& k, const Fp& f, double& u, double& v,
                                           double& P) {
    const Divisor r(p[0], f);
    u = r.div(p[1], f);
    v = r.div(p[2], f);
    const double m = f.mul(p[0], f.add(f.mul(u, u), f.mul(v, v)));
    P = f.mul(__fma_rn(m, -f.half, p[3]), k.gm1);   // E - (0.5 rho (u^2 + v^2)), the product's half exact
    return r;
}

// class_flow::updateQ (class_flow.hpp:28-34)
template <class T>
__device__ __forceinline__ void cons(T rho, T u, T v, T P, const Consts<T>& k, T q[4]) {
    q[0] = rho;
    q[1] = rho * u;
    q[2] = rho * v;
    q[3] = (P / k.gm1) + T(0.5) * rho * (u * u + v * v);
}

// ------------------------------------------------------------------------------------------
// Gradient + squeeze limiter.  compute_gradient (src/solver/cell_gradient.cpp:9-131) and
// squeeze (src/solver/squeeze.cpp:9-155), restated as one gather per cell.
// The squeeze compares against the face values of the PREVIOUS stage (res.cpp:40 runs before the
// reconstruction at :48): those its face pass stored (DevMesh::fval), or the -101 sentinel the face
// states start with (class_q.hpp:73-76) on the first stage after initialisation.
// a[j] for a run-time j without indexing (which would put the array in local memory)
template <class T>
__device__ __forceinline__ T pick4(const T a[4], int j) {
    return j == 0 ? a[0] : j == 1 ? a[1] : j == 2 ? a[2] : a[3];
}

#ifndef FV2D_FP64_BLOCK
#define FV2D_FP64_BLOCK 128   // threads per block of the gradient and face kernels
#endif

// One component j of cell c's limited gradient: a thread per cell and component.  The components share
// only the mesh and, at walls, the ghost's primitives, so four lanes per cell do the same FP64 work
// as one, in a quarter of the chain (64 cycles an operation for a lone warp, whatever its active
// lanes) and with fewer registers.  With the limiter below: 8,192 quads 107 -> 67 us per iteration, 50k NS
// polygons 446 -> 395, 400k 2,854 -> 2,752 (update_lane's share included).
// The limiter takes the smallest of 1 and the factors (bound - Q) / (face value - Q) of the previous face
// values that leave the bounds (squeeze.cpp:68-141).  Rounded subtraction and division are monotone, so
// on either side the smallest factor is the one at the extreme face value: one division per
// violated side instead of one per violating face.  Where the bounds meet (the neighbourhood is uniform)
// every factor is a zero, -0 below and +0 above, and the reference keeps the last face's.
template <bool SQUEEZE, class Wait>
__device__ __forceinline__ void gradient_lane(int c, int j, const Fp& fp, const DevMesh<double>& m, const Q4<double>* Q,
                                              Q4<double>* Gout, const Consts<double>& k, int first_stage, int init_prims, Wait wait) {
    const int* __restrict__ inc = m.inc;
    const int* __restrict__ nbr = m.nbr;
    const double* Qd = reinterpret_cast<const double*>(Q);
    const double* fv = reinterpret_cast<const double*>(m.fval);
    const FaceGeo<double>& g = m.g;
    const int b = m.inc_off[c], e = m.inc_off[c + 1];
    double sx = 0.0, sy = 0.0;
    // software-pipelined: the ids of the incidence after next and the states of the next one are
    // requested before the current one is processed (every cell has at least 3 faces)
    int inc_n = inc[b], nb_n = nbr[b], inc_2 = inc[b + 1], nb_2 = nbr[b + 1];
    double2 ig_n = *reinterpret_cast<const double2*>(m.igeo + b);
    wait();
    const double qc = Qd[4 * (size_t)c + j];
    double qn_n = 0.0, qf_n = -101.0;   // -101: the face states before the first stage (class_q.hpp:73-76)
    auto states = [&] {
        if (nb_n >= 0) qn_n = Qd[4 * (size_t)nb_n + j];
        if (SQUEEZE && !first_stage) qf_n = fv[4 * (size_t)inc_n + j];
    };
    states();
    // the bounds start with the first face's states in the reference's order (squeeze.cpp: the c1
    // side's, then the c2 side's), which decides between +0 and -0
    double mn = qc, mx = qc, fmn = 0.0, fmx = 0.0;
    long long kc = 0, kmn = 0, kmx = 0, kfmn = 0, kfmx = 0;
    int last = 0;   // the last face value that differs from Q: below (-1) or above (1)
    if (SQUEEZE) {
        kc = order_key(qc);
        if (nb_n >= 0 && (inc_n & 1)) mn = mx = qn_n;
        kmn = kmx = order_key(mn);
        if (kc < kmn) { kmn = kc; mn = qc; }
        if (kmx < kc) { kmx = kc; mx = qc; }
        fmn = fmx = qf_n;
        kfmn = kfmx = order_key(qf_n);
    }
    for (int i = b; i < e; i++) {
        const int f = inc_n >> 1, side = inc_n & 1, nb = nb_n;
        const double2 ig = ig_n;
        const double qn = qn_n, qf = qf_n;
        if (i + 1 < e) {
            inc_n = inc_2;
            nb_n = nb_2;
            ig_n = *reinterpret_cast<const double2*>(m.igeo + i + 1);
            states();
            if (i + 2 < e) { inc_2 = inc[i + 2]; nb_2 = nbr[i + 2]; }
        }
        double d;
        if (nb >= 0) {
            d = side == 0 ? fp.sub(qn, qc) : fp.sub(qc, qn);   // reference orientation: c2 - c1
            if (SQUEEZE) {
                const long long kn = order_key(qn);
                if (kn < kmn) { kmn = kn; mn = qn; }
                if (kmx < kn) { kmx = kn; mx = qn; }
            }
        } else if (nb == -1) {
            d = fp.sub(pick4(k.q_inf, j), qc);
        } else if (nb == -2 || nb == -4) {
            double rho, u, v, P, gq[4];
            if (init_prims) { rho = k.rho_inf; u = k.u_inf; v = k.v_inf; P = k.P_inf; }
            else {
                const Q4<double> qq = Q[nb == -2 ? c : m.qcell[f]];
                rho = qq.p[0];
                prims_r(qq.p, k, fp, u, v, P);
            }
            if (nb == -2) {        // slip wall: reflect the cell velocity (cell_gradient.cpp:43-55)
                const double fnx = g.nx[f], fny = g.ny[f];
                const double vn = u * fnx + v * fny;
                cons(rho, u - 2.0 * vn * fnx, v - 2.0 * vn * fny, P, k, gq);
            } else {               // no-slip: state of cell `face id`, velocity negated (:62-73)
                cons(rho, -u, -v, P, k, gq);
            }
            d = fp.sub(pick4(gq, j), qc);
        } else {
            d = 0.0;
        }
        if (SQUEEZE) {
            const long long kf = order_key(qf);
            if (kf < kfmn) { kfmn = kf; fmn = qf; }
            if (kfmx < kf) { kfmx = kf; fmx = qf; }
            last = kf < kc ? -1 : kc < kf ? 1 : last;
        }
        sx = fp.add(sx, fp.mul(d, ig.x));
        sy = fp.add(sy, fp.mul(d, ig.y));
    }
    const double ixx = m.Ixx[c], iyy = m.Iyy[c], ixy = m.Ixy[c];
    double gx = fp.sub(fp.mul(sx, iyy), fp.mul(sy, ixy));
    double gy = fp.sub(fp.mul(sy, ixx), fp.mul(sx, ixy));
    if (SQUEEZE) {
        // the reference's starting values
        if (!(kmn < order_key(100000000000.0))) { mn = 100000000000.0; kmn = order_key(mn); }
        if (!(order_key(-100000000000.0) < kmx)) { mx = -100000000000.0; kmx = order_key(mx); }
        const bool below = kfmn < kmn, above = kmx < kfmx;
        double phi = 1.0;
        if (below || above) {   // one division for the violated side, a second where both are
            phi = fp.sub(below ? mn : mx, qc) / fp.sub(below ? fmn : fmx, qc);
            if (below && above) {
                const double up = fp.sub(mx, qc) / fp.sub(fmx, qc);
                const bool zeros = ((__double_as_longlong(phi) | __double_as_longlong(up)) << 1) == 0;
                phi = zeros ? (last < 0 ? phi : up) : min2(up, phi);
            }
            phi = min2(phi, 1.0);
        }
        gx = fp.mul(gx, phi);
        gy = fp.mul(gy, phi);
    }
    double* go = reinterpret_cast<double*>(Gout + 2 * (size_t)c);
    go[j] = gx;
    go[4 + j] = gy;
}

#ifndef FV2D_FP64_GMINB
#define FV2D_FP64_GMINB 6   // 6 x 128 threads at 80 registers: 400k-cell NS cylinder 2.75 ms per iteration, 2.81 with 8
                            // (64 registers, spills), 2.79 with 5
#endif
template <bool SQUEEZE>
__global__ void __launch_bounds__(FV2D_FP64_BLOCK, FV2D_FP64_GMINB)
k_gradient(int nc, DevMesh<double> m, const Q4<double>* Q, Q4<double>* Gout, Consts<double> k,
           int first_stage, int init_prims) {
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
    if (c >= nc) return;
    const Fp fp;
    gradient_lane<SQUEEZE>(c, threadIdx.x & 3, fp, m, Q, Gout, k, first_stage, init_prims, Prior());
}

#ifndef FV2D_FP64_FMINB
#define FV2D_FP64_FMINB 4   // 4 x 128 threads at up to 128 registers
#endif

// ------------------------------------------------------------------------------------------
// Face kernel: reconstruction + boundary ghosts (reconstruction.cpp:22-80), NS face terms
// (reconstruction.cpp:86-164, class_q.hpp:163-169, class_f.hpp:52-59), Rusanov flux
// (class_f.hpp:41-50, rusanov.cpp:20-36) and the face's residual contribution (res.cpp:81-89).
// Writes t = (V*A) - (F*A) per face and, on the last stage of an iteration, the spectral term
// (|Vn_avg| + c_avg)*A that the next time step sums (ssp_rk3.cpp:28-36).
// First order: q + 0 dx + 0 dy is q, but for a -0 that meets a +0 product.
__device__ __forceinline__ double first_order_state(double q, double dx, double dy) {
    const bool pos = (__double2hiint(dx) & __double2hiint(dy)) >= 0;
    return pos && __double_as_longlong(q) == (long long)0x8000000000000000ULL ? 0.0 : q;
}

// Powers of two travel through the formulas as exact scalings instead of operations: the average
// state's sums S = L + R stand for 2 (L + R)/2, the wave speed t = |vn1 + vn2| + (c1 + c2) for 4 lambda,
// the flux F2 for 2 F against half the area, the viscous flux V2 for 2 V (mu and k enter doubled), and
// the remaining halves ride on multiply-adds.  Every rounded intermediate is the reference's times a
// power of two, so the results are the same bits.  352 FP64 pipe slots for an NS face (356 on the last stage),
// 160 for an Euler face, those of the reciprocals and roots included.
template <bool ORDER2, bool NS, bool LAST, class Wait>
__device__ __forceinline__ void face_flux(int f, const Fp& fp, const DevMesh<double>& m, const Q4<double>* Q,
                                          const Q4<double>* G, Q4<double>* tout, double* sout, const Consts<double>& k,
                                          int init_prims, Wait wait) {
    const FaceGeo<double>& g = m.g;
    const int c1 = m.fc1[f], c2 = m.fc2[f];
    const double fnx = g.nx[f], fny = g.ny[f], A = g.area[f];
    const double d1x = g.c1dx[f], d1y = g.c1dy[f], d2x = g.c2dx[f], d2y = g.c2dy[f];
    wait();
    const Q4<double> q1 = ldq(Q, c1);
    Q4<double> g1x, g1y;
    if (ORDER2) { g1x = ldq(G, 2 * c1); g1y = ldq(G, 2 * c1 + 1); }
    // the right cell's loads are issued now, beside the left cell's (a boundary face, c2 < 0,
    // loads cell c1's row instead and never uses it), so the two gathers overlap
    const int c2l = c2 >= 0 ? c2 : c1;
    const Q4<double> q2 = ldq(Q, c2l);
    Q4<double> g2x, g2y;
    if (ORDER2) { g2x = ldq(G, 2 * c2l); g2y = ldq(G, 2 * c2l + 1); }
    double L[4], Rq[4];
#pragma unroll
    for (int j = 0; j < 4; j++)
        L[j] = ORDER2 ? fp.add(fp.add(q1.p[j], fp.mul(g1x.p[j], d1x)), fp.mul(g1y.p[j], d1y)) : first_order_state(q1.p[j], d1x, d1y);
    const double lrho = L[0];
    double lu, lv, lP;
    const Divisor ld = prims_r(L, k, fp, lu, lv, lP);
    const double lc = sqrt(k.gamma * ld.div(lP, fp));
    if (c2 >= 0) {
#pragma unroll
        for (int j = 0; j < 4; j++)
            Rq[j] = ORDER2 ? fp.add(fp.add(q2.p[j], fp.mul(g2x.p[j], d2x)), fp.mul(g2y.p[j], d2y)) : first_order_state(q2.p[j], d2x, d2y);
    } else if (c2 == -1) {
#pragma unroll
        for (int j = 0; j < 4; j++) Rq[j] = k.q_inf[j];
    } else if (c2 == -2) {
        const double vn = lu * fnx + lv * fny;
        cons(lrho, lu - 2.0 * vn * fnx, lv - 2.0 * vn * fny, lP, k, Rq);
    } else if (c2 == -3) {
#pragma unroll
        for (int j = 0; j < 4; j++) Rq[j] = L[j];
    } else {
        cons(lrho, -lu, -lv, lP, k, Rq);
    }
    if (m.fval) {   // the next squeeze's stale face values (BC faces: the c1 side only)
        Q4<double> lq, rq;
#pragma unroll
        for (int j = 0; j < 4; j++) { lq.p[j] = L[j]; rq.p[j] = Rq[j]; }
        m.fval[2 * f] = lq;
        if (c2 >= 0) m.fval[2 * f + 1] = rq;
    }
    const double rrho = Rq[0];
    double ru, rv, rP;
    const Divisor rd = prims_r(Rq, k, fp, ru, rv, rP);
    const double rc = sqrt(k.gamma * rd.div(rP, fp));

    // Rusanov: F2 = 2 Fr = (F1 + F2) - (t/2)(R - L), t = 4 lambda = 2 (|Vn_avg| + c_avg)
    const double vn1 = fp.add(fp.mul(lu, fnx), fp.mul(lv, fny)), vn2 = fp.add(fp.mul(ru, fnx), fp.mul(rv, fny));
    const double t4 = fp.add(fabs(fp.add(vn1, vn2)), fp.add(lc, rc));
    const double Ah = fp.mul(A, fp.half);
    double F2[4];
    if (k.roe) {
#pragma unroll
        for (int j = 0; j < 4; j++) F2[j] = -202.0;
    } else {
        const double X[4] = {
            fp.add(fp.mul(lrho, vn1), fp.mul(rrho, vn2)),
            fp.add(fp.add(fp.mul(fp.mul(lrho, lu), vn1), fp.mul(lP, fnx)), fp.add(fp.mul(fp.mul(rrho, ru), vn2), fp.mul(rP, fnx))),
            fp.add(fp.add(fp.mul(fp.mul(lrho, lv), vn1), fp.mul(lP, fny)), fp.add(fp.mul(fp.mul(rrho, rv), vn2), fp.mul(rP, fny))),
            fp.add(fp.mul(vn1, fp.add(L[3], lP)), fp.mul(vn2, fp.add(Rq[3], rP)))};
#pragma unroll
        for (int j = 0; j < 4; j++) F2[j] = __fma_rn(fp.mul(t4, fp.sub(Rq[j], L[j])), -fp.half, X[j]);
    }

    // viscous flux, V2 = 2 V (first order never adds it: res.cpp:27-29,50-53)
    double V2[4] = {0.0, 0.0, 0.0, 0.0};
    if (NS && ORDER2) {
        double S[4];   // twice the average state
#pragma unroll
        for (int j = 0; j < 4; j++) S[j] = fp.add(L[j], Rq[j]);
        const Divisor sd(S[0], fp);
        const double au = sd.div(S[1], fp), av = sd.div(S[2], fp);
        const double ke = fp.add(fp.mul(au, au), fp.mul(av, av));
        const double aP2 = fp.mul(__fma_rn(fp.mul(S[0], ke), -fp.half, S[3]), k.gm1);   // twice the pressure
        double ux = 0.0, uy = 0.0, vx = 0.0, vy = 0.0, Px = 0.0, Py = 0.0, rx = 0.0, ry = 0.0;
        bool have = true;
        if (c2 >= 0) {
            const double ad = fabs(g.dist[f]);
            const Divisor dd(ad, m.rdist[f], fp);   // 1/|dist| precomputed
            // unit tangent p1 -> p2 (readmesh.cpp:400-406) from the normal: mx = dx/|d| = -ny and
            // my = dy/|d| = nx, bit for bit (same |d| expression, sign-symmetric rounding)
            const double mxf = -fny, myf = fnx, lxf = g.lx[f], lyf = g.ly[f];
            double dQx[4], dQy[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const double dl = dd.div(fp.sub(q2.p[j], q1.p[j]), fp);
                const double dm2 = fp.add(fp.add(fp.add(fp.mul(g1x.p[j], mxf), fp.mul(g1y.p[j], myf)), fp.mul(g2x.p[j], mxf)),
                                          fp.mul(g2y.p[j], myf));   // twice the tangential derivative
                dQy[j] = __fma_rn(fp.mul(dm2, lyf), fp.half, fp.mul(dl, lyf));
                dQx[j] = __fma_rn(fp.mul(dm2, lxf), fp.half, fp.mul(dl, lxf));
            }
            // quotients by S0 = 2 rho are half of those by rho
            rx = dQx[0];
            ux = __fma_rn(sd.div(fp.mul(rx, au), fp), -2.0, dQx[1]);
            vx = __fma_rn(sd.div(fp.mul(rx, av), fp), -2.0, dQx[2]);
            ry = dQy[0];
            const double ryu = sd.div(fp.mul(ry, au), fp);
            uy = __fma_rn(ryu, -2.0, dQy[1]);
            vy = __fma_rn(ryu, -2.0, dQy[2]);   // reconstruction.cpp:155 uses u
            Px = fp.mul(k.gm1, __fma_rn(fp.mul(S[0], fp.add(fp.mul(au, ux), fp.mul(av, vx))), -fp.half,
                                        __fma_rn(fp.mul(rx, ke), -fp.half, dQx[3])));
            Py = fp.mul(k.gm1, __fma_rn(fp.mul(S[0], fp.add(fp.mul(au, uy), fp.mul(av, vy))), -fp.half,
                                        __fma_rn(fp.mul(ry, ke), -fp.half, dQy[3])));
        } else if (c2 == -4) {
            const double dn = fabs(sqrt(d1x * d1x + d1y * d1y));
            double cu, cv;
            if (init_prims) { cu = k.u_inf; cv = k.v_inf; }
            else { cu = q1.p[1] / q1.p[0]; cv = q1.p[2] / q1.p[0]; }
            const Divisor nd(dn, fp);
            const double dudn = nd.div(-cu, fp), dvdn = nd.div(-cv, fp);
            ux = dudn * fnx; uy = dudn * fny;
            vx = dvdn * fnx; vy = dvdn * fny;
        } else if (c2 == -2) {
            have = false;   // SLIP_WALL with NS: tau and grad T keep their initial zeros (:104-106)
        }
        double txx, txy, tyy, dTx, dTy;   // twice the stresses; half the temperature derivatives
        if (have) {
            const double third = div3(fp.add(ux, vy)), mu2 = 2.0 * k.mu, mu4 = 4.0 * k.mu;
            txx = fp.mul(mu4, fp.sub(ux, third));
            txy = fp.mul(mu2, fp.add(uy, vx));
            tyy = fp.mul(mu4, fp.sub(vy, third));
            const double den = fp.mul(fp.mul(k.R, S[0]), S[0]), yden = __drcp_rn(den);   // 4 R rho^2
            dTx = Recip<double>::div(fp.sub(fp.mul(Px, S[0]), fp.mul(rx, aP2)), den, yden);
            dTy = Recip<double>::div(fp.sub(fp.mul(Py, S[0]), fp.mul(ry, aP2)), den, yden);
        } else {
            txx = 0.0; txy = 0.0; tyy = 0.0; dTx = 0.0; dTy = 0.0;
        }
        const double k4 = 4.0 * k.k;
        V2[1] = fp.add(fp.mul(txx, fnx), fp.mul(txy, fny));
        V2[2] = fp.add(fp.mul(txy, fnx), fp.mul(tyy, fny));
        V2[3] = fp.add(fp.mul(fnx, fp.add(fp.add(fp.mul(au, txx), fp.mul(av, txy)), fp.mul(k4, dTx))),
                       fp.mul(fny, fp.add(fp.add(fp.mul(au, txy), fp.mul(av, tyy)), fp.mul(k4, dTy))));
    }
    Q4<double> t;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        // (V*A) - (F*A); V[0] is always +0, and all of V is +0 for Euler and first order
        if (j == 0 || !(NS && ORDER2)) t.p[j] = zero_minus(fp.mul(F2[j], Ah));
        else t.p[j] = fp.sub(fp.mul(V2[j], Ah), fp.mul(F2[j], Ah));
    }
    tout[f] = t;
    if (LAST) sout[f] = k.roe ? (fabs(k.vn0) + k.c0) * A : fp.mul(t4, Ah);
}

template <bool ORDER2, bool NS, bool LAST>
__global__ void __launch_bounds__(FV2D_FP64_BLOCK, FV2D_FP64_FMINB)
k_face(int nf, DevMesh<double> m, const Q4<double>* Q, const Q4<double>* G, Q4<double>* tout, double* sout, Consts<double> k,
       int init_prims) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const Fp fp;
    face_flux<ORDER2, NS, LAST>(f, fp, m, Q, G, tout, sout, k, init_prims, Prior());
}

// ------------------------------------------------------------------------------------------
// Spectral sums S_c = sum_f (|Vn_avg| + c_avg) A_f in ascending original face id
// (ssp_rk3.cpp:28-36).  s == nullptr: the initial Vn_avg, c_avg of every face (class_q.hpp:61-62).
template <class T>
__device__ __forceinline__ void atomic_max_pos(T* addr, T v);
template <>
__device__ __forceinline__ void atomic_max_pos<double>(double* addr, double v) {
    atomicMax(reinterpret_cast<unsigned long long*>(addr), (unsigned long long)__double_as_longlong(v));
}
template <>
__device__ __forceinline__ void atomic_max_pos<float>(float* addr, float v) {
    atomicMax(reinterpret_cast<unsigned int*>(addr), __float_as_uint(v));
}

template <class T>
__device__ __forceinline__ T block_max(T v) {
    __shared__ T red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max2(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        v = lane < (int)(blockDim.x >> 5) ? red[lane] : T(0);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = max2(v, __shfl_xor_sync(0xffffffffu, v, o));
    }
    return v;
}

template <class T>
__global__ void __launch_bounds__(256)
k_spectral_init(int nc, const int* __restrict__ inc_off, const int* __restrict__ inc, const T* __restrict__ area,
                T* __restrict__ S, T* __restrict__ smax, Consts<T> k) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    T s = T(0);
    if (c < nc) {
        for (int i = inc_off[c]; i < inc_off[c + 1]; i++) s += (fabs(k.vn0) + k.c0) * area[inc[i] >> 1];
        S[c] = s;
    }
    const T m = block_max(c < nc ? s : T(0));
    if (threadIdx.x == 0) atomic_max_pos(smax, m);
}

// ------------------------------------------------------------------------------------------
// Residual gather + SSP-RK3 stage (res.cpp:74-109, ssp_rk3.cpp:38-77).
// STAGE 0: dt from the spectral sums (GLOBAL: 2*CFL*vol/max S, LOCAL: 2*CFL*vol/S), Q1 = Qn+dt*R
// STAGE 1: Q2 = 0.75*Qn + 0.25*Q1 + 0.25*dt*R
// STAGE 2: Qn = 1/3*Qn + 2/3*Q2 + 2/3*dt*R, and the spectral sums for the next iteration.
// Non-physical results (rho <= 0, E <= 0, NaN) raise bit 0 of *flag; values are kept as computed.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    const float bp = s - a;
    e = (a - (s - bp)) + (b - bp);
}

constexpr int kUpdChunk = 4;   // incidences whose loads the residual gather issues together (4.6 % faster k_update)

// S_c = sum of the face spectral terms in CSR order, loads issued a chunk at a time
__device__ __forceinline__ double spectral_sum(const int* __restrict__ inc, const double* sface, int b, int e,
                                               const Fp& fp) {
    double s = 0.0;
    constexpr int U = kUpdChunk;
    for (int i0 = b; i0 < e; i0 += U) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u < e) v[u] = *(sface + (inc[i0 + u] >> 1));
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u < e) s = fp.add(s, v[u]);
    }
    return s;
}

// -x when s == 1, x when s == 0: a sign-bit flip on the integer pipe.  r - t == r + (-t) exactly in
// IEEE arithmetic (zeros included), so the residual gather adds the flipped contribution instead
// of branching between += and -= on the incidence's side (a warp's lanes disagree on it).
__device__ __forceinline__ double neg_if(double x, int s) {
    return __longlong_as_double(__double_as_longlong(x) ^ ((long long)s << 63));
}

// x > 0 (false for NaN).  FP64 on the integer pipe: 0 < bits <= bits(+inf).
template <class T>
__device__ __forceinline__ bool positive(T x) { return x > T(0); }
template <>
__device__ __forceinline__ bool positive<double>(double x) {
    return (unsigned long long)__double_as_longlong(x) - 1ull < 0x7ff0000000000000ull;
}

// What a cell's update reads of the mesh: its incidence range and first incidences, its volume.
struct UpdateMesh {
    int b = 0, e = 0, inc[kUpdChunk];
    double vol = 1.0, rvol = 1.0;   // rvol: 1/vol, precomputed
    __device__ __forceinline__ UpdateMesh(int c, const DevMesh<double>& m) {
        b = m.inc_off[c];
        e = m.inc_off[c + 1];
        vol = m.vol[c];
        rvol = m.rvol[c];
#pragma unroll
        for (int u = 0; u < kUpdChunk; u++) inc[u] = b + u < e ? m.inc[b + u] : 0;
    }
};

// One component j of cell c's update; returns its residual component.
template <int STAGE>
__device__ __forceinline__ double update_lane(int c, int j, const Fp& fp, const DevMesh<double>& m, const UpdateMesh& um,
                                              const Q4<double>* tface, Q4<double>* Qn, Q4<double>* Q1, Q4<double>* Q2,
                                              double dtc, Q4<double>* Rout, int* flag) {
    const double* t = reinterpret_cast<const double*>(tface);
    const size_t o = 4 * (size_t)c + j;
    const int b = um.b, e = um.e;
    const double qn = reinterpret_cast<const double*>(Qn)[o];
    const double qs = STAGE == 0 ? 0.0 : reinterpret_cast<const double*>(STAGE == 1 ? Q1 : Q2)[o];
    double r = 0.0;
    // chunks of kUpdChunk incidences: every record and face contribution of a chunk is requested
    // before the first is summed (more loads in flight per thread); the sums keep CSR order
    constexpr int U = kUpdChunk;
    for (int i0 = b; i0 < e; i0 += U) {
        int iv[U];
        double tv[U];
#pragma unroll
        for (int u = 0; u < U; u++) iv[u] = i0 == b ? um.inc[u] : i0 + u < e ? m.inc[i0 + u] : 0;
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u < e) tv[u] = t[4 * (size_t)(iv[u] >> 1) + j];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u < e) r = fp.add(r, neg_if(tv[u], iv[u] & 1));   // side 1: r -= t
    }
    {   // r / vol: two residual corrections from RN(r*y), as Recip (Divisor's digits would cost every lane more)
        const double q0 = fp.mul(r, um.rvol), q1 = __fma_rn(__fma_rn(-um.vol, q0, r), um.rvol, q0);
        r = (__double_as_longlong(r) << 1) == 0 ? q0 : __fma_rn(__fma_rn(-um.vol, q1, r), um.rvol, q1);
    }
    if (Rout) reinterpret_cast<double*>(Rout)[o] = r;
    const double dr = fp.mul(dtc, r);
    double out;
    if (STAGE == 0) {
        out = fp.add(qn, dr);
        reinterpret_cast<double*>(Q1)[o] = out;
    } else if (STAGE == 1) {   // 3/4 Qn + 1/4 Q1 + 1/4 dt R, the exact quarters on the multiply-adds
        out = __fma_rn(dr, 0.25, __fma_rn(qs, 0.25, fp.mul(0.75, qn)));
        reinterpret_cast<double*>(Q2)[o] = out;
    } else {
        out = fp.add(fp.add(fp.mul(1.0 / 3.0, qn), fp.mul(2.0 / 3.0, qs)), fp.mul(fp.mul(2.0 / 3.0, dtc), r));
        reinterpret_cast<double*>(Qn)[o] = out;
    }
    if ((j == 0 || j == 3) && !positive(out)) atomicOr(flag, 1);
    return r;
}

// Threads per block of the update kernel: four lanes (one component each) per cell; the block's first
// warp also holds one lane per cell for what a cell needs once: its time step in the first stage
// (one division) and its spectral sum in the last.  Large meshes, where the pipe and not the chain is the
// limit, pay for it: each lane repeats the incidence loop's and the division's overhead (66 -> 73 pipe
// slots per cell; 300k cells 43.3 -> 45.3 us, 1M 141 -> 146), against 20 us less in the gradient at 300k.
// The second stage, which does not read it, zeroes the spectral maximum that the last accumulates.
constexpr int kUpdBlock = 128, kUpdCells = kUpdBlock / 4;

template <int STAGE>
__global__ void __launch_bounds__(kUpdBlock)
k_update(int nc, DevMesh<double> m, const Q4<double>* tface, const double* sface, Q4<double>* Qn,
         Q4<double>* Q1, Q4<double>* Q2, double* dt, double* S, double* smax, Q4<double>* Rout, int* flag, Consts<double> k,
         int global_dt) {
    __shared__ double sdt[kUpdCells];
    const Fp fp;
    const int c0 = blockIdx.x * kUpdCells, c = c0 + (threadIdx.x >> 2), j = threadIdx.x & 3, cw = c0 + threadIdx.x;
    const UpdateMesh um(min(c, nc - 1), m);
    Prior()();
    if (STAGE == 0) {
        if (threadIdx.x < kUpdCells && cw < nc) {
            const double d = (k.two_cfl * m.vol[cw]) / (global_dt ? *smax : S[cw]);
            sdt[threadIdx.x] = d;
            dt[cw] = d;
        }
        __syncthreads();
    }
    if (STAGE == 1 && blockIdx.x == 0 && threadIdx.x == 0) *smax = 0.0;
    if (c < nc)
        update_lane<STAGE>(c, j, fp, m, um, tface, Qn, Q1, Q2, STAGE == 0 ? sdt[threadIdx.x >> 2] : dt[c], Rout, flag);
    if (STAGE == 2 && threadIdx.x < kUpdCells) {
        double s = 0.0;
        if (cw < nc) {
            s = spectral_sum(m.inc, sface, m.inc_off[cw], m.inc_off[cw + 1], fp);
            S[cw] = s;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s = max2(s, __shfl_xor_sync(0xffffffffu, s, o));
        if (threadIdx.x == 0) atomic_max_pos(smax, s);
    }
}

// Two lanes per face, for meshes small enough that every warp has its SM quarter's FP64 pipe to itself, so
// that the length of a lane's chain of operations is the pass's time: lane h = 0 takes cell c1's side, components 0
// and 1 of the flux and the x derivatives, lane h = 1 cell c2's side, components 2 and 3 and the y
// derivatives.  Every value is computed by the expression face_flux uses, so the bits are the same;
// 204 FP64 pipe slots a lane for an NS face against 352, 88 against 160 for an Euler face.  All 32 lanes
// call (act: the lane pair has a face).  (With programmatic launches: 512 Euler quads 58 -> 50 us per iteration, 2k NS
// polygons 80 -> 72; with two warps to a quarter the extra work loses, 8k NS polygons 118 -> 131.)
template <bool ORDER2, bool NS>
__device__ __forceinline__ void face_pair(int f, int h, bool act, const Fp& fp, const DevMesh<double>& m, const Q4<double>* Q,
                                          const Q4<double>* G, Q4<double>* tout, double* sout, const Consts<double>& k,
                                          int init_prims, bool last, Prior wait) {
    constexpr unsigned FULL = 0xffffffffu;
    auto other = [&](double x) { return __shfl_xor_sync(FULL, x, 1); };
    // the partner's value of this lane's components: send the partner's pair, keep one's own
    auto swap2 = [&](const double v[4], double& a, double& b) {
        a = other(h ? v[0] : v[2]);
        b = other(h ? v[1] : v[3]);
    };
    const FaceGeo<double>& g = m.g;
    const int ff = act ? f : 0;
    const int c1 = m.fc1[ff], c2 = m.fc2[ff];
    const bool inner = c2 >= 0;
    const int cell = h && inner ? c2 : c1;
    const double fnx = g.nx[ff], fny = g.ny[ff];
    const double dx = h ? g.c2dx[ff] : g.c1dx[ff], dy = h ? g.c2dy[ff] : g.c1dy[ff];
    const double A = g.area[ff];
    wait();
    const Q4<double> q = Q[cell];
    Q4<double> gx, gy;
    if (ORDER2) { gx = G[2 * (size_t)cell]; gy = G[2 * (size_t)cell + 1]; }
    double X[4];   // this side's face state
    if (ORDER2) {
#pragma unroll
        for (int j = 0; j < 4; j++) X[j] = fp.add(fp.add(q.p[j], fp.mul(gx.p[j], dx)), fp.mul(gy.p[j], dy));
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++) X[j] = first_order_state(q.p[j], dx, dy);
    }
    double u = 0.0, v = 0.0, P = 0.0, c = 0.0;
    auto side = [&] {
        const Divisor r = prims_r(X, k, fp, u, v, P);
        c = sqrt(k.gamma * r.div(P, fp));
    };
    if (!h || inner) side();
    if (__any_sync(FULL, !inner)) {   // boundary faces: lane 1's state is a ghost of lane 0's
        double L[4], lu, lv, lP;
#pragma unroll
        for (int j = 0; j < 4; j++) L[j] = other(X[j]);
        lu = other(u);
        lv = other(v);
        lP = other(P);
        if (h && !inner) {
            if (c2 == -1) {
#pragma unroll
                for (int j = 0; j < 4; j++) X[j] = k.q_inf[j];
            } else if (c2 == -2) {
                const double vn = lu * fnx + lv * fny;
                cons(L[0], lu - 2.0 * vn * fnx, lv - 2.0 * vn * fny, lP, k, X);
            } else if (c2 == -3) {
#pragma unroll
                for (int j = 0; j < 4; j++) X[j] = L[j];
            } else {
                cons(L[0], -lu, -lv, lP, k, X);
            }
            side();
        }
    }
    if (m.fval && act && (!h || inner)) {
        Q4<double> o;
#pragma unroll
        for (int j = 0; j < 4; j++) o.p[j] = X[j];
        m.fval[2 * (size_t)f + h] = o;
    }
    const double vn = fp.add(fp.mul(u, fnx), fp.mul(v, fny));
    const double t4 = fp.add(fabs(fp.add(vn, other(vn))), fp.add(c, other(c)));
    const double Ah = fp.mul(A, fp.half);
    // this lane's two components: states of both sides, 2 F
    double oX[2], F2[2];
    swap2(X, oX[0], oX[1]);
    const double myX[2] = {h ? X[2] : X[0], h ? X[3] : X[1]};
    {
        const double F[4] = {fp.mul(X[0], vn), fp.add(fp.mul(fp.mul(X[0], u), vn), fp.mul(P, fnx)),
                             fp.add(fp.mul(fp.mul(X[0], v), vn), fp.mul(P, fny)), fp.mul(vn, fp.add(X[3], P))};
        double oF[2];
        swap2(F, oF[0], oF[1]);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const double d = h ? fp.sub(myX[i], oX[i]) : fp.sub(oX[i], myX[i]);   // R - L
            F2[i] = k.roe ? -202.0 : __fma_rn(fp.mul(t4, d), -fp.half, fp.add(h ? F[2 + i] : F[i], oF[i]));
        }
    }
    double V2[2] = {0.0, 0.0};
    if (NS && ORDER2) {
        double S[4];   // twice the average state
        {
            const double a = fp.add(myX[0], oX[0]), b = fp.add(myX[1], oX[1]), oa = other(a), ob = other(b);
            S[0] = h ? oa : a; S[1] = h ? ob : b; S[2] = h ? a : oa; S[3] = h ? b : ob;
        }
        const Divisor sd(S[0], fp);
        const double mine = sd.div(h ? S[2] : S[1], fp), theirs = other(mine);
        const double au = h ? theirs : mine, av = h ? mine : theirs;
        const double ke = fp.add(fp.mul(au, au), fp.mul(av, av));
        const double aP2 = fp.mul(__fma_rn(fp.mul(S[0], ke), -fp.half, S[3]), k.gm1);   // twice the pressure
        const double nh = h ? fny : fnx;
        double U = 0.0, V = 0.0, dP = 0.0, r = 0.0;   // this direction's derivatives of u, v, P, rho
        {
            // differences and tangential derivatives of this lane's components, then of all four
            double oq[2], ogx[2], ogy[2], dl[4], dm2[4];
            swap2(q.p, oq[0], oq[1]);
            swap2(gx.p, ogx[0], ogx[1]);
            swap2(gy.p, ogy[0], ogy[1]);
            const Divisor dd(inner ? fabs(g.dist[ff]) : 1.0, inner ? m.rdist[ff] : 1.0, fp);
            const double mxf = -fny, myf = fnx, lh = inner ? (h ? g.ly[ff] : g.lx[ff]) : 0.0;
            double a[2], b[2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const double mq = h ? q.p[2 + i] : q.p[i], mgx = h ? gx.p[2 + i] : gx.p[i], mgy = h ? gy.p[2 + i] : gy.p[i];
                const double q1 = h ? oq[i] : mq, q2 = h ? mq : oq[i], g1x = h ? ogx[i] : mgx, g1y = h ? ogy[i] : mgy,
                             g2x = h ? mgx : ogx[i], g2y = h ? mgy : ogy[i];
                a[i] = dd.div(fp.sub(q2, q1), fp);
                b[i] = fp.add(fp.add(fp.add(fp.mul(g1x, mxf), fp.mul(g1y, myf)), fp.mul(g2x, mxf)), fp.mul(g2y, myf));
            }
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const double oa = other(a[i]), ob = other(b[i]);
                dl[i] = h ? oa : a[i]; dl[2 + i] = h ? a[i] : oa;
                dm2[i] = h ? ob : b[i]; dm2[2 + i] = h ? b[i] : ob;
            }
            if (inner) {
                double dQ[4];
#pragma unroll
                for (int j = 0; j < 4; j++) dQ[j] = __fma_rn(fp.mul(dm2[j], lh), fp.half, fp.mul(dl[j], lh));
                r = dQ[0];
                U = __fma_rn(sd.div(fp.mul(r, au), fp), -2.0, dQ[1]);
                V = __fma_rn(sd.div(fp.mul(r, h ? au : av), fp), -2.0, dQ[2]);   // reconstruction.cpp:155 uses u for y
                dP = fp.mul(k.gm1, __fma_rn(fp.mul(S[0], fp.add(fp.mul(au, U), fp.mul(av, V))), -fp.half,
                                            __fma_rn(fp.mul(r, ke), -fp.half, dQ[3])));
            } else if (c2 == -4) {
                const double d1x = g.c1dx[ff], d1y = g.c1dy[ff];
                const double dn = fabs(sqrt(d1x * d1x + d1y * d1y));
                double cu, cv;
                if (init_prims) { cu = k.u_inf; cv = k.v_inf; }
                else { cu = q.p[1] / q.p[0]; cv = q.p[2] / q.p[0]; }   // both lanes hold cell c1's state here
                const Divisor nd(dn, fp);
                U = nd.div(-cu, fp) * nh;
                V = nd.div(-cv, fp) * nh;
            }
        }
        const double oU = other(U), oV = other(V);
        const double ux = h ? oU : U, vx = h ? oV : V, uy = h ? U : oU, vy = h ? V : oV;
        double ta = 0.0, tb = 0.0, dT = 0.0;   // row h of twice the stress tensor; half this direction's dT
        if (c2 != -2) {   // SLIP_WALL with NS: tau and grad T keep their initial zeros (:104-106)
            const double third = div3(fp.add(ux, vy));
            const double diag = fp.mul(4.0 * k.mu, fp.sub(h ? vy : ux, third)), off = fp.mul(2.0 * k.mu, fp.add(uy, vx));
            ta = h ? off : diag;
            tb = h ? diag : off;
            const double den = fp.mul(fp.mul(k.R, S[0]), S[0]);   // 4 R rho^2
            dT = Recip<double>::div(fp.sub(fp.mul(dP, S[0]), fp.mul(r, aP2)), den, __drcp_rn(den));
        }
        const double row = fp.add(fp.mul(ta, fnx), fp.mul(tb, fny));
        const double heat = fp.mul(nh, fp.add(fp.add(fp.mul(au, ta), fp.mul(av, tb)), fp.mul(4.0 * k.k, dT)));
        const double oheat = other(heat);
        V2[0] = h ? row : 0.0;
        V2[1] = h ? fp.add(oheat, heat) : row;
    }
    if (!act) return;
    double t[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        if (!(NS && ORDER2)) t[i] = zero_minus(fp.mul(F2[i], Ah));
        else t[i] = !h && i == 0 ? zero_minus(fp.mul(F2[i], Ah)) : fp.sub(fp.mul(V2[i], Ah), fp.mul(F2[i], Ah));
    }
    *reinterpret_cast<double2*>(reinterpret_cast<double*>(tout + f) + 2 * h) = make_double2(t[0], t[1]);
    if (last && !h) sout[f] = k.roe ? (fabs(k.vn0) + k.c0) * A : fp.mul(t4, Ah);
}

template <bool ORDER2, bool NS, bool LAST>
__global__ void __launch_bounds__(FV2D_FP64_BLOCK, FV2D_FP64_FMINB)
k_face_pair(int nf, DevMesh<double> m, const Q4<double>* Q, const Q4<double>* G, Q4<double>* tout, double* sout, Consts<double> k,
            int init_prims) {
    const int f = (blockIdx.x * blockDim.x + threadIdx.x) >> 1;
    if ((f & ~15) >= nf) return;   // whole warps
    const Fp fp;
    face_pair<ORDER2, NS>(f, threadIdx.x & 1, f < nf, fp, m, Q, G, tout, sout, k, init_prims, LAST, Prior());
}

// Geometry-only reciprocals of a mesh (or of one solve's ranges in a batch arena): rdist = 1/|dist|
// (dist may be null: no NS faces) and rvol = 1/vol, with the kernels' own Recip<T>::of.
template <class T>
__global__ void k_reciprocals(int nf, const T* __restrict__ dist, T* __restrict__ rdist, int nc,
                              const T* __restrict__ vol, T* __restrict__ rvol) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < max(nf, nc); i += gridDim.x * blockDim.x) {
        if (i < nf && dist) rdist[i] = Recip<T>::of(fabs(dist[i]));
        if (i < nc) rvol[i] = Recip<T>::of(vol[i]);
    }
}

// ------------------------------------------------------------------------------------------
// Host-format <-> device-format state (SoA double in file numbering <-> AoS T in device order).
template <class T>
__global__ void k_state_in(int nc, const int* __restrict__ new2old, const double* __restrict__ q, Q4<T>* __restrict__ Q,
                           Q4<T>* __restrict__ Qlo) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    const int o = new2old[c];
    Q4<T> v, lo;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const double x = q[(size_t)j * nc + o];
        v.p[j] = (T)x;
        lo.p[j] = (T)(x - (double)v.p[j]);
    }
    Q[c] = v;
    if (Qlo) Qlo[c] = lo;
}

template <class T>
__global__ void k_state_out(int nc, int ncomp, const int* __restrict__ new2old, const Q4<T>* __restrict__ Q,
                            double* __restrict__ q, const Q4<T>* __restrict__ Qlo) {
    // ncomp = 4 (state; plus its compensation term when Qlo is given) or 8 (gradient pairs)
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    const int o = new2old[c];
    const int per = ncomp / 4;
    for (int h = 0; h < per; h++) {
        const Q4<T> v = Q[(size_t)per * c + h];
        Q4<T> lo;
        if (Qlo) lo = Qlo[c];
#pragma unroll
        // FP64 (no compensation term): the value itself - adding 0.0 would turn -0 into +0
        for (int j = 0; j < 4; j++) q[(size_t)(4 * h + j) * nc + o] = Qlo ? (double)v.p[j] + (double)lo.p[j] : (double)v.p[j];
    }
}

template <class T>
__global__ void k_scalar_out(int nc, const int* __restrict__ new2old, const T* __restrict__ a, double* __restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    out[new2old[c]] = (double)a[c];
}

// Sum of squares of the residual per variable, FP64, deterministic two-level reduction.
template <class T>
__global__ void __launch_bounds__(256) k_res_norm_partial(int nc, const Q4<T>* __restrict__ R, double* __restrict__ part) {
    __shared__ double sh[4][256];
    double acc[4] = {0, 0, 0, 0};
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += gridDim.x * blockDim.x) {
        const Q4<T> r = R[c];
#pragma unroll
        for (int j = 0; j < 4; j++) acc[j] += (double)r.p[j] * (double)r.p[j];
    }
#pragma unroll
    for (int j = 0; j < 4; j++) sh[j][threadIdx.x] = acc[j];
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s)
#pragma unroll
            for (int j = 0; j < 4; j++) sh[j][threadIdx.x] += sh[j][threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0)
#pragma unroll
        for (int j = 0; j < 4; j++) part[4 * blockIdx.x + j] = sh[j][0];
}

}  // namespace fv2d
