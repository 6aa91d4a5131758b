/*
 * Plain-FP64 flux pass for sm_100a: gradients, per-face fluxes, update_Q and
 * get_W, bit-identical to Shadowfax's CPU pass.
 *
 * This translation unit is compiled with -fmad=false (no a*b+c contraction)
 * and IEEE division / square root, and keeps the reference's expression
 * order, so each value is rounded exactly as the reference rounds it.  pow()
 * has the values of sfx_pow (sfx_pow.h), shared with the CPU oracle, because
 * glibc's and CUDA's pow differ in the last bit; it is evaluated by sfx_powq
 * (sfx_powq.h).
 *
 * Kernels (one step = three launches, four with the exact solver's face list):
 *   k_grad_cells one thread per cell and variable: VorCell::estimate_gradient
 *                (src/VorCell.cpp:464-530); k_gradients, one thread per
 *                cell, for meshes whose faces do not sit between their
 *                cells' positions and for caller-owned arrays
 *   k_faces      one thread per face: VorFace::calculate_flux
 *                (src/VorFace.cpp:670-1024) with the Exact or HLLC solver;
 *                writes the limited dQ of the left cell once per face
 *   k_apply      one thread per cell: the face contributions in
 *                ascending face order (the order of VorTessManager::hydro's
 *                loop, src/VorTessManager.cpp:205-209), Q -= dQ
 *                (GasParticle::update_Q, GasParticle.cpp:617-624), get_W.
 * No floating-point atomics: every cell sums its own faces in a fixed order,
 * so reruns are bitwise identical.
 */
#include <cuda_runtime.h>

#include "sfx_internal.h"
#include "sfx_limiter.h"
#include "sfx_wide.h"

/* sfx_pow for the arguments sfx_powq does not settle, out of line */
__host__ __device__ __noinline__ double sfx_pow_rare64(double x, double y);
#define SFX_POWQ_RARE sfx_pow_rare64
#include "sfx_powq.h"
__host__ __device__ __noinline__ double sfx_pow_rare64(double x, double y) {
    return sfx_pow(x, y);
}

namespace {

constexpr unsigned kRightBit = 0x80000000u;

__device__ __forceinline__ void report_face(sfx_dev_error* e, int f, int st) {
    unsigned long long key = ((unsigned long long)(unsigned)f << 8) | (unsigned)st;
    atomicMin(&e->face_key, key);
}

__device__ __forceinline__ void report_cell(sfx_dev_error* e, int i, int st) {
    unsigned long long key = ((unsigned long long)(unsigned)i << 8) | (unsigned)st;
    atomicMin(&e->cell_key, key);
}

__device__ __forceinline__ bool failed(const sfx_dev_error* e) {
    return (*(volatile const unsigned long long*)&e->face_key != ~0ull) ||
           (*(volatile const unsigned long long*)&e->cell_key != ~0ull);
}

/* a face lower than f has failed: f cannot change the record */
__device__ __forceinline__ bool below(const sfx_dev_error* e, int f) {
    return *(volatile const unsigned long long*)&e->face_key < (unsigned long long)(unsigned)f << 8;
}

/* ---------------- time derivative (Exact :892-934 / HLLC :415-450) ------- */
template <int D>
__device__ __forceinline__ void time_derivative(double gamma, const double* W,
                                                const double (*g)[D + 2],
                                                double* dW);

template <>
__device__ __forceinline__ void time_derivative<3>(double gamma, const double* W,
                                                   const double (*g)[5],
                                                   double* dW) {
    dW[0] = -W[0] * (g[0][1] + g[1][2] + g[2][3]) - W[1] * g[0][0] -
            W[2] * g[1][0] - W[3] * g[2][0];
    dW[1] = -W[1] * g[0][1] - W[2] * g[1][1] - W[3] * g[2][1] - g[0][4] / W[0];
    dW[2] = -W[1] * g[0][2] - W[2] * g[1][2] - W[3] * g[2][2] - g[1][4] / W[0];
    dW[3] = -W[1] * g[0][3] - W[2] * g[1][3] - W[3] * g[2][3] - g[2][4] / W[0];
    dW[4] = -gamma * W[4] * (g[0][1] + g[1][2] + g[2][3]) - W[1] * g[0][4] -
            W[2] * g[1][4] - W[3] * g[2][4];
}

template <>
__device__ __forceinline__ void time_derivative<2>(double gamma, const double* W,
                                                   const double (*g)[4],
                                                   double* dW) {
    dW[0] = -W[1] * g[0][0] - W[2] * g[1][0] - W[0] * (g[0][1] + g[1][2]);
    dW[1] = -W[1] * g[0][1] - W[2] * g[1][1] - g[0][3] / W[0];
    /* the reference uses d(vy)/dy in both terms (ExactRiemannSolver.cpp:920) */
    dW[2] = -W[1] * g[1][2] - W[2] * g[1][2] - g[1][3] / W[0];
    dW[3] = -gamma * W[3] * (g[0][1] + g[1][2]) - W[1] * g[0][3] - W[2] * g[1][3];
}

template <int D>
__device__ __forceinline__ double dot(const double* a, const double* b) {
    double s = a[0] * b[0] + a[1] * b[1];
    if(D == 3) s = s + a[2] * b[2];
    return s;
}

template <int D>
__device__ __forceinline__ double norm(const double* a) {
    return sqrt(dot<D>(a, a));
}

/* VorFace.hpp:174-196 */
template <int D>
__device__ __forceinline__ void reconstruct(double* W, const double (*g)[D + 2],
                                            const double* d) {
#pragma unroll
    for(int k = 0; k < D + 2; ++k) {
        double s = g[0][k] * d[0] + g[1][k] * d[1];
        if(D == 3) s = s + g[2][k] * d[2];
        W[k] = W[k] + s;
    }
}

/* VorFace.hpp:92-137 */
template <int D>
__device__ __forceinline__ double limit1(double phimid0, double phiL, double phiR, double w) {
    const double psi1 = 0.5, psi2 = 0.25;
    double delta1 = psi1 * fabs(phiL - phiR);
    double delta2 = psi2 * fabs(phiL - phiR);
    double phimin = fmin(phiL, phiR);
    double phimax = fmax(phiL, phiR);
    double phibar = phiL + w * (phiR - phiL);
    if(phiL == phiR) return phiL;
    /* only the bound the result uses (phi- when phiL < phiR, else phi+), with
     * the sign-preserving fallback where the shifted extreme changes sign:
     * the reference's values, without the other bound's divisions */
    const bool up = phiL < phiR;
    const double ext = up ? phimin : phimax;
    double bound = up ? ext - delta1 : ext + delta1;
    if(!(bound * ext > 0.)) bound = ext / (1. + delta1 / fabs(ext));
    if(up) return fmax(bound, fmin(phibar + delta2, phimid0));
    return fmin(bound, fmax(phibar - delta2, phimid0));
}

/* mirror a state across a reflective face: transform, flip the normal
 * velocity, invtransform (VorFace.cpp:417-542, VorCell.cpp:479-485) */
/* from r = left - right and its norm (right - left is -r exactly) */
template <int D>
__device__ __forceinline__ void mirror_across(double* W, const double* r, double rnorm);

template <>
__device__ __forceinline__ void mirror_across<3>(double* W, const double* r, double rnorm) {
    double n0 = -r[0], n1 = -r[1], n2 = -r[2];
    const double n3 = rnorm;
    n0 /= n3;
    n1 /= n3;
    n2 /= n3;
    double o0, o1, o3, p0, p1, p2;
    if(n0 != 0. || n1 != 0.) {
        o0 = -n1;
        o1 = n0;
        o3 = sqrt(o0 * o0 + o1 * o1);
        o0 /= o3;
        o1 /= o3;
        p0 = -n2 * o1;
        p1 = n2 * o0;
        p2 = o3;
    } else {
        o0 = 0.;
        o1 = 1.;
        p0 = -1.;
        p1 = 0.;
        p2 = 0.;
    }
    double v0 = W[1], v1 = W[2], v2 = W[3];
    double t1 = v0 * n0 + v1 * n1 + v2 * n2;
    double t2 = v0 * o0 + v1 * o1;
    double t3 = v0 * p0 + v1 * p1 + v2 * p2;
    t1 = -t1;
    W[1] = t1 * n0 + t2 * o0 + t3 * p0;
    W[2] = t1 * n1 + t2 * o1 + t3 * p1;
    W[3] = t1 * n2 + t3 * p2;
}

template <>
__device__ __forceinline__ void mirror_across<2>(double* W, const double* r, double rnorm) {
    const double d0 = r[0], d1 = r[1], d2 = rnorm;
    double cost = -d0 / d2;
    double sint = -d1 / d2;
    double W1 = W[1] * cost + W[2] * sint;
    double W2 = -W[1] * sint + W[2] * cost;
    W1 = -W1;
    W[1] = W1 * cost - W2 * sint;
    W[2] = W1 * sint + W2 * cost;
}

template <int D>
__device__ __forceinline__ void mirror_state(double* W, const double* left,
                                             const double* right) {
    double r[D];
#pragma unroll
    for(int l = 0; l < D; ++l) r[l] = left[l] - right[l];
    mirror_across<D>(W, r, norm<D>(r));
}

/* ------------------------------- records -------------------------------
 * A mesh's step reads three records laid out for it (a gather of one variable
 * at a time from field-major arrays touches a 32-byte sector per double):
 *   ws   [n][8]   the cell's W, then its mass Q[0]
 *   grec [n][20] (3D), [n][12] (2D): gradients [l][k], then dW/dt at W
 *   dQf  [F][6] (3D), [F][4] (2D): the limited dQ of the left cell
 * and two per face that hold what the reference forms from positions on
 * every step, in its operation order (the mesh is static between uploads):
 *   ggeo gradient: A, 1/|r|, |r|, c, r, midpoint (NaN for a face of zero
 *        area); c = mid - (x_L + x_R)/2 and r = x_L - x_R
 *   fgeo flux: {left, right or -1}, A, A/area_L, A/area_R, |d_L|/|c_LR|,
 *        |d_R|/|c_LR|, d_L, d_R, normal */
template <int D>
struct Rec {
    static constexpr int S = D + 2;
    static constexpr int ws = 8;
    static constexpr int grec = D == 3 ? 20 : 12;
    static constexpr int dq = D == 3 ? 6 : 4;
    static constexpr int ggeo = 12;
    static constexpr int fgeo = D == 3 ? 16 : 12;
    /* cells per warp of the kernels with one lane per cell and variable */
    static constexpr int cells = 32 / S;
};

/* N doubles of a record on a 32-byte (N % 4 == 0) or 16-byte boundary */
template <int N>
__device__ __forceinline__ void load_record(const double* p, double* out) {
    static_assert(N % 2 == 0, "whole 16-byte units");
#pragma unroll
    for(int i = 0; i < N; i += N % 4 ? 2 : 4) {
        if constexpr(N % 4 == 0) {
            sfx_load32(p + i, out + i);
        } else {
            const double2 v = __ldg(reinterpret_cast<const double2*>(p + i));
            out[i] = v.x;
            out[i + 1] = v.y;
        }
    }
}

template <int N>
__device__ __forceinline__ void store_record(double* p, const double* v) {
#pragma unroll
    for(int i = 0; i < N; i += N % 4 ? 2 : 4) {
        if constexpr(N % 4 == 0)
            sfx_store32(p + i, v + i);
        else
            *reinterpret_cast<double2*>(p + i) = make_double2(v[i], v[i + 1]);
    }
}

/* a length, or a difference of positions, for which sfx_div_by's products and
 * residuals stay far from underflow and overflow */
__device__ __forceinline__ bool plain_size(double x) {
    return x == 0. || (fabs(x) > 0x1p-200 && fabs(x) < 0x1p200);
}

template <int D>
__global__ void __launch_bounds__(128) k_face_records(sfx_dmesh m) {
    using R = Rec<D>;
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if(f >= m.n_faces) return;
    const int n = m.n_cells, F = m.n_faces;
    const int iL = m.left[f];
    const bool has_right = m.kind[f] != SFX_FACE_MIRROR;
    const int iR = has_right ? m.right[f] : 0;
    const double A = m.area[f];
    double mid[D], xL[D], xRi[D], cenL[D], r[D], c[D], dL[D], dR[D], dd[D], cd[D];
    bool plain = true;
#pragma unroll
    for(int l = 0; l < D; ++l) {
        mid[l] = m.mid[(size_t)l * F + f];
        xL[l] = m.pos[(size_t)l * n + iL];
        xRi[l] = m.rpos[(size_t)l * F + f];
        cenL[l] = m.cen[(size_t)l * n + iL];
        c[l] = mid[l] - 0.5 * (xL[l] + xRi[l]);
        r[l] = xL[l] - xRi[l];
        plain = plain && plain_size(c[l]) && plain_size(r[l]);
        dL[l] = mid[l] - cenL[l] + (xL[l] - xL[l]);
        dR[l] = 0.;
        cd[l] = 0.;
        if(has_right) {
            const double cenR = m.cen[(size_t)l * n + iR], xR = m.pos[(size_t)l * n + iR];
            dR[l] = mid[l] - cenR + (xR - xRi[l]);
            cd[l] = cenL[l] - cenR;
        }
        dd[l] = xL[l] - xRi[l];
    }
    const double rn = norm<D>(r);
    double g[R::ggeo];
    g[0] = A;
    g[1] = plain && plain_size(rn) && rn > 0. ? 1. / rn : 0.;
    g[2] = rn;
#pragma unroll
    for(int l = 0; l < D; ++l) {
        g[3 + l] = c[l];
        g[3 + D + l] = r[l];
        /* a NaN offset takes no part in the slope limiter */
        g[3 + 2 * D + l] = A == 0. ? __longlong_as_double(0x7ff8000000000000ll) : mid[l];
    }
    if(D == 2) {
        /* the midpoint to the record's third 32 bytes */
        g[8] = g[7];
        g[9] = A == 0. ? g[7] : mid[1];
        g[7] = g[10] = g[11] = 0.;
    }
    store_record<R::ggeo>(m.ggeo + (size_t)f * R::ggeo, g);
    const double cn = norm<D>(cd);
    const double dn = norm<D>(dd);
    double h[R::fgeo];
    h[0] = __hiloint2double(has_right ? iR : -1, iL);
    h[1] = A;
    h[2] = A / m.tarea[iL];
    h[3] = has_right ? A / m.tarea[iR] : 0.;
    h[4] = has_right ? sqrt(dot<D>(dL, dL)) / cn : 0.;
    h[5] = has_right ? sqrt(dot<D>(dR, dR)) / cn : 0.;
#pragma unroll
    for(int l = 0; l < D; ++l) {
        h[6 + l] = dL[l];
        h[6 + D + l] = dR[l];
        /* VorFace::get_normal (VorFace.cpp:553-571) */
        h[6 + 2 * D + l] = -dd[l] / dn;
    }
    if(D == 3) h[R::fgeo - 1] = 0.;
    /* planes of 32 bytes per face: consecutive threads read consecutive faces */
#pragma unroll
    for(int q = 0; q < R::fgeo; q += 4) store_record<4>(m.fgeo + (size_t)q * F + 4 * (size_t)f, h + q);
}

/* each CSR entry with its neighbour cell, so that the gradient kernels load
 * it beside the face id instead of after it */
__global__ void __launch_bounds__(256) k_csr_neighbours(sfx_dmesh m) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(j >= m.nnz) return;
    const unsigned e = (unsigned)m.idx[j];
    const int f = (int)(e & ~kRightBit);
    const int nb = e & kRightBit ? m.left[f] : (m.kind[f] == SFX_FACE_MIRROR ? -1 : m.right[f]);
    m.ent[j] = make_int2((int)e, nb);
}

/* rows of W and Q -> W, Q (field-major) and, where the mesh has records, ws */
template <int D>
__global__ void __launch_bounds__(128) k_load_rows(sfx_dmesh m, const double* W, const double* Q) {
    constexpr int S = D + 2;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= m.n_cells) return;
#pragma unroll
    for(int k = 0; k < S; ++k) {
        m.W[(size_t)k * m.n_cells + i] = W[(size_t)i * S + k];
        m.Q[(size_t)k * m.n_cells + i] = Q[(size_t)i * S + k];
    }
    if(!m.ws) return;
    double* w = m.ws + (size_t)i * Rec<D>::ws;
#pragma unroll
    for(int k = 0; k < S; ++k) w[k] = W[(size_t)i * S + k];
    w[S] = Q[(size_t)i * S];
}

/* ------------------------------ gradients ------------------------------ */
/* REC: the gradients and dW/dt go to the cell's record (field-major
 * gradients otherwise, for caller-owned arrays) */
template <int D, bool REC>
__global__ void __launch_bounds__(128) k_gradients(sfx_dmesh m, double gamma) {
    constexpr int S = D + 2;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(REC && i == 0) *m.listed_n = 0; /* a new step's list */
    if(i >= sfx_grad_cells(m) || failed(m.err)) return;
    /* local time steps: an inactive cell keeps its gradients (src/Simulation.cpp:414-420) */
    if(m.local && m.tstart[i] != m.t_now) return;
    const int n = m.n_cells, F = m.n_faces;
    double W[S], xi[D], Wmax[S], Wmin[S], delta[D][S];
#pragma unroll
    for(int k = 0; k < S; ++k) {
        W[k] = m.W[(size_t)k * n + i];
        Wmax[k] = W[k];
        Wmin[k] = W[k];
#pragma unroll
        for(int l = 0; l < D; ++l) delta[l][k] = 0.;
    }
#pragma unroll
    for(int l = 0; l < D; ++l) xi[l] = m.pos[(size_t)l * n + i];
    const int beg = m.off[i], end = m.off[i + 1];
    for(int j = end - 1; j >= beg; --j) {
        const unsigned e = (unsigned)m.idx[j];
        const int f = (int)(e & ~kRightBit);
        const double A = m.area[f];
        if(A == 0.) continue;
        double mid[D], xj[D], Wj[S];
#pragma unroll
        for(int l = 0; l < D; ++l) mid[l] = m.mid[(size_t)l * F + f];
        if(!(e & kRightBit)) {
#pragma unroll
            for(int l = 0; l < D; ++l) xj[l] = m.rpos[(size_t)l * F + f];
            if(m.kind[f] == SFX_FACE_MIRROR) {
#pragma unroll
                for(int k = 0; k < S; ++k) Wj[k] = W[k];
                mirror_state<D>(Wj, xi, xj);
            } else {
                const int r = m.right[f];
#pragma unroll
                for(int k = 0; k < S; ++k) Wj[k] = m.W[(size_t)k * n + r];
            }
        } else {
            const int jl = m.left[f];
#pragma unroll
            for(int l = 0; l < D; ++l) xj[l] = m.pos[(size_t)l * n + jl];
#pragma unroll
            for(int k = 0; k < S; ++k) Wj[k] = m.W[(size_t)k * n + jl];
        }
        double c[D], rij[D];
#pragma unroll
        for(int l = 0; l < D; ++l) {
            c[l] = mid[l] - 0.5 * (xi[l] + xj[l]);
            rij[l] = xi[l] - xj[l];
        }
        const double rnorm = norm<D>(rij);
#pragma unroll
        for(int l = 0; l < D; ++l) {
#pragma unroll
            for(int k = 0; k < S; ++k) {
                delta[l][k] = delta[l][k] +
                              A * ((Wj[k] - W[k]) * c[l] / rnorm -
                                   0.5 * (W[k] + Wj[k]) * rij[l] / rnorm);
            }
        }
#pragma unroll
        for(int k = 0; k < S; ++k) {
            Wmax[k] = (Wmax[k] < Wj[k]) ? Wj[k] : Wmax[k];
            Wmin[k] = (Wj[k] < Wmin[k]) ? Wj[k] : Wmin[k];
        }
    }
    const double V = m.vol[i];
#pragma unroll
    for(int l = 0; l < D; ++l)
#pragma unroll
        for(int k = 0; k < S; ++k) delta[l][k] = delta[l][k] / V;
    double cen[D], alpha[S];
#pragma unroll
    for(int l = 0; l < D; ++l) cen[l] = m.cen[(size_t)l * n + i];
#pragma unroll
    for(int k = 0; k < S; ++k) alpha[k] = 1.;
    for(int j = end - 1; j >= beg; --j) {
        const int f = (int)((unsigned)m.idx[j] & ~kRightBit);
        if(m.area[f] == 0.) continue;
        double d[D];
#pragma unroll
        for(int l = 0; l < D; ++l) d[l] = m.mid[(size_t)l * F + f] - cen[l];
#pragma unroll
        for(int k = 0; k < S; ++k) {
            double dp = delta[0][k] * d[0] + delta[1][k] * d[1];
            if(D == 3) dp = dp + delta[2][k] * d[2];
            double q1 = Wmax[k] - W[k];
            double q2 = Wmin[k] - W[k];
            if(dp != 0.) {
                q1 = q1 / dp;
                q2 = q2 / dp;
            } else {
                q1 = 1.;
                q2 = 1.;
            }
            const double mx = (q1 < q2) ? q2 : q1;
            alpha[k] = (mx < alpha[k]) ? mx : alpha[k];
        }
    }
    if constexpr(REC) {
        double out[Rec<D>::grec];
#pragma unroll
        for(int l = 0; l < D; ++l)
#pragma unroll
            for(int k = 0; k < S; ++k) {
                delta[l][k] = delta[l][k] * alpha[k];
                out[l * S + k] = delta[l][k];
            }
        time_derivative<D>(gamma, W, delta, out + D * S);
        store_record<Rec<D>::grec>(m.grec + (size_t)i * Rec<D>::grec, out);
    } else {
#pragma unroll
        for(int l = 0; l < D; ++l)
#pragma unroll
            for(int k = 0; k < S; ++k)
                m.grad[((size_t)l * S + k) * n + i] = delta[l][k] * alpha[k];
    }
}

/* 0, or a normal size between 2^-300 and 2^300: with plain_size lengths,
 * every dividend of the gradient is then 0 or between 2^-560 and 2^520 */
__device__ __forceinline__ bool plain_state(double x) {
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return h - 0x2d300000u < 0x25800000u || (h | (unsigned)__double2loint(x)) == 0u;
}

/* asynchronous copy of BYTES (8 or 16) bytes to shared memory, both aligned to them */
template <int BYTES>
__device__ __forceinline__ void copy_async(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                         (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "n"(BYTES)
                 : "memory");
}

/* One lane per (cell, primitive variable), Rec::cells whole cells per warp:
 * the variables are independent in both loops, so each lane adds the terms
 *   A ((W_j - W_i) c / |r| - (W_i + W_j) / 2 r / |r|)
 * in the cell's face order, as the reference rounds them; the right cell of a
 * face sees the same c and |r| and the opposite r (the mesh qualifies when
 * every local face's right position is its right cell's position, gshare).
 * Bound by FP64 issue and the latency of the gathers.  The 2 D divisions by
 * |r| use the face's stored reciprocal (sfx_div_by: 5 operations; a zero term's
 * sign cannot change a sum that starts at +0), the limiter's minimum over the
 * faces takes two divisions per cell (sfx_limiter_min), and the face's
 * geometry and the neighbour's state come through a shared-memory ring filled
 * kGradStages faces ahead (lane k of a cell copies 16 bytes of the geometry
 * and one variable): no registers hold loads in flight.  Both loops divided
 * per face before, the first one in a kernel of its own that wrote 128 bytes
 * per face: 220 -> 83 us (event-timed; 80 in a profile) on 65,537 cells in 3D,
 * 104 -> 63 us on 150,001 in 2D (109 and 68 us without the ring; 88 and 66
 * without the kept midpoints).  96 registers in 3D: 102 left four blocks per SM
 * instead of five (87 us), 80 spill (86).  Two faces per ring stage: 85.  Cells
 * sorted by face count so that a warp's lanes run equally long: 83 us where this
 * took 88, but the update in that order lost more than that to a lower L1 hit
 * rate. */
constexpr int kGradBlock = 128, kGradStages = 4;

template <int D>
struct GradSlot {
    static constexpr int S = D + 2;
    double2 geo[S];  /* A, 1/|r|, |r|, c, r */
    double W[S];     /* the neighbour's state */
    int2 ent;        /* CSR entry, neighbour (-1: mirror) */
    /* to 144 bytes (3D) and 112 (2D): a warp's cells on different banks */
    double pad[D == 3 ? 2 : 1];
};

template <int D>
__global__ void __launch_bounds__(kGradBlock, D == 3 ? 5 : 6) k_grad_cells(sfx_dmesh m, double gamma) {
    using R = Rec<D>;
    constexpr int S = R::S;
    static_assert(sizeof(GradSlot<D>) == (D == 3 ? 144 : 112), "slot layout");
    __shared__ __align__(16) GradSlot<D> ring[kGradBlock / 32][kGradStages][R::cells];
    /* the first kKept faces' midpoints, for the limiter's loop (one double of
     * padding: a warp's cells on different banks) */
    constexpr int kKept = D == 3 ? 24 : 12;
    __shared__ double kept[kGradBlock / 32][R::cells][kKept * D + 1];
    if(blockIdx.x == 0 && threadIdx.x == 0) *m.listed_n = 0; /* a new step's list */
    const int lane = threadIdx.x & 31;
    const int slot = lane / S, k = lane - slot * S;
    const int i = ((blockIdx.x * kGradBlock + threadIdx.x) >> 5) * R::cells + slot;
    /* local time steps: an inactive cell keeps its gradients (src/Simulation.cpp:414-420) */
    const bool live = slot < R::cells && i < sfx_grad_cells(m) && !failed(m.err) &&
                      !(m.local && m.tstart[i] != m.t_now);
    if(!__any_sync(0xffffffffu, live)) return;
    const int ic = live ? i : 0;
    const double* own = m.ws + (size_t)ic * R::ws;
    const double W = own[k];
    double delta[D];
    double Wmax = W, Wmin = W;
    bool plain = plain_state(W);
#pragma unroll
    for(int l = 0; l < D; ++l) delta[l] = 0.;
    const int beg = live ? m.off[ic] : 0, end = live ? m.off[ic + 1] : 0;
    const int count = end - beg;
    const int most = __reduce_max_sync(0xffffffffu, count);
    /* face `it` of the cell (from its last to its first) into its ring slot;
     * the CSR entry was loaded one call before */
    int2 next = make_int2(0, -1);
    if(count > 0) next = __ldg(m.ent + end - 1);
    GradSlot<D>(*mine)[R::cells] = ring[threadIdx.x >> 5];
    double* mids = kept[threadIdx.x >> 5][slot < R::cells ? slot : 0];
    auto fetch = [&](int it) {
        if(it < count) {
            const int2 v = next;
            if(it + 1 < count) next = __ldg(m.ent + end - 2 - it);
            GradSlot<D>& q = mine[it % kGradStages][slot];
            const double* rec = m.ggeo + (size_t)((unsigned)v.x & ~kRightBit) * R::ggeo;
            copy_async<16>(&q.geo[k], rec + 2 * k);
            if(k < D && it < kKept) copy_async<8>(mids + it * D + k, rec + (D == 3 ? 9 : 8) + k);
            copy_async<8>(&q.W[k], m.ws + (size_t)(v.y < 0 ? ic : v.y) * R::ws + k);
            if(k == 0) q.ent = v;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for(int it = 0; it < kGradStages - 1; ++it) fetch(it);
#pragma unroll 1
    for(int it = 0; it < most; ++it) {
        /* this lane's copies for face `it` have landed; then every lane's */
        asm volatile("cp.async.wait_group %0;" ::"n"(kGradStages - 2) : "memory");
        __syncwarp();
        /* the slot refilled here was read before the barrier above */
        fetch(it + kGradStages - 1);
        if(it >= count) continue;
        const GradSlot<D>& q = mine[it % kGradStages][slot];
        double g[2 * S];
#pragma unroll
        for(int t = 0; t < S; ++t) {
            g[2 * t] = q.geo[t].x;
            g[2 * t + 1] = q.geo[t].y;
        }
        double Wj = q.W[k];
        const double A = g[0], y = g[1], rn = g[2];
        if(A == 0.) continue;
        const int2 ent = q.ent;
        if(ent.y < 0) {
            double Wm[S], r[D];
#pragma unroll
            for(int t = 0; t < S; ++t) Wm[t] = own[t];
#pragma unroll
            for(int l = 0; l < D; ++l) r[l] = g[3 + D + l];
            mirror_across<D>(Wm, r, rn);
#pragma unroll
            for(int t = 1; t <= D; ++t)
                if(t == k) Wj = Wm[t];
        }
        const double dW = Wj - W;
        double sW = 0.5 * (W + Wj);
        if((unsigned)ent.x & kRightBit) sW = -sW; /* r changes sign */
        plain = plain && plain_state(Wj);
        if(plain && y != 0.) {
#pragma unroll
            for(int l = 0; l < D; ++l)
                delta[l] = delta[l] + A * (sfx_div_by(dW * g[3 + l], rn, y) -
                                           sfx_div_by(sW * g[3 + D + l], rn, y));
        } else {
#pragma unroll
            for(int l = 0; l < D; ++l)
                delta[l] = delta[l] + A * (dW * g[3 + l] / rn - sW * g[3 + D + l] / rn);
        }
        Wmax = (Wmax < Wj) ? Wj : Wmax;
        Wmin = (Wj < Wmin) ? Wj : Wmin;
    }
    const double V = m.vol[ic];
    double cen[D];
#pragma unroll
    for(int l = 0; l < D; ++l) {
        delta[l] = delta[l] / V;
        cen[l] = m.cen[(size_t)l * m.n_cells + ic];
    }
    const double a = Wmax - W, b = Wmin - W;
    /* the offsets' projections on the gradient: the extremes decide the limiter */
    auto offset = [&](int it) {
        double d[D];
        if(it < kKept) {
#pragma unroll
            for(int l = 0; l < D; ++l) d[l] = mids[it * D + l] - cen[l];
        } else {
            const unsigned f = (unsigned)__ldg(m.idx + end - 1 - it) & ~kRightBit;
            const double* rec = m.ggeo + (size_t)f * R::ggeo + (D == 3 ? 9 : 8);
#pragma unroll
            for(int l = 0; l < D; ++l) d[l] = __ldg(rec + l) - cen[l];
        }
        double dp = delta[0] * d[0] + delta[1] * d[1];
        if(D == 3) dp = dp + delta[D - 1] * d[D - 1];
        return dp;
    };
    /* every lane's copies have landed */
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    double dmax = 0., dmin = 0.;
    int first = 0;
    for(int it = 0; it < count; ++it) {
        const double dp = offset(it);
        if(dp > dmax) dmax = dp;
        if(dp < dmin) dmin = dp;
        if(first == 0) first = dp > 0. ? 1 : (dp < 0. ? -1 : 0);
    }
    double alpha = 1.;
    if(plain && dmax < 0x1p300 && dmin > -0x1p300) {
        alpha = sfx_limiter_min(a, b, dmax, dmin, first);
    } else {
        for(int it = 0; it < count; ++it) {
            const double dp = offset(it);
            /* a face of zero area (NaN offset) is skipped; other NaNs never
             * compare below alpha */
            const double mx = sfx_limiter_ratio(a, b, dp);
            alpha = (mx < alpha) ? mx : alpha;
        }
    }
    double g[D];
#pragma unroll
    for(int l = 0; l < D; ++l) g[l] = delta[l] * alpha;
    /* dW/dt at the cell's state (time_derivative), one variable per lane */
    const int base = slot * S;
    double Wc[S], diag[D], gp[D];
#pragma unroll
    for(int q = 0; q < S; ++q) Wc[q] = __shfl_sync(0xffffffffu, W, base + q);
#pragma unroll
    for(int l = 0; l < D; ++l) {
        diag[l] = __shfl_sync(0xffffffffu, g[l], base + 1 + l);
        gp[l] = __shfl_sync(0xffffffffu, g[l], base + S - 1);
    }
    if(!live) return;
    double dW;
    if(D == 3) {
        const double div = diag[0] + diag[1] + diag[D - 1];
        const double lead = k == 0 ? -Wc[0] * div : (k == S - 1 ? -gamma * Wc[S - 1] * div : 0.);
        if(k == 0 || k == S - 1)
            dW = lead - Wc[1] * g[0] - Wc[2] * g[1] - Wc[D] * g[D - 1];
        else
            dW = -Wc[1] * g[0] - Wc[2] * g[1] - Wc[D] * g[D - 1] -
                 (k == 1 ? gp[0] : (k == 2 ? gp[1] : gp[D - 1])) / Wc[0];
    } else {
        const double div = diag[0] + diag[1];
        if(k == 0)
            dW = -Wc[1] * g[0] - Wc[2] * g[1] - Wc[0] * div;
        else if(k == 1)
            dW = -Wc[1] * g[0] - Wc[2] * g[1] - gp[0] / Wc[0];
        else if(k == 2) /* d(vy)/dy in both terms (ExactRiemannSolver.cpp:920) */
            dW = -Wc[1] * g[1] - Wc[2] * g[1] - gp[1] / Wc[0];
        else
            dW = -gamma * Wc[S - 1] * div - Wc[1] * g[0] - Wc[2] * g[1];
    }
    double* out = m.grec + (size_t)i * R::grec;
#pragma unroll
    for(int l = 0; l < D; ++l) out[l * S + k] = g[l];
    out[D * S + k] = dW;
}

/* --------------------------- exact solver --------------------------- */
struct ExactOut {
    int status;
    int code;
};

template <int D>
__device__ __forceinline__ double sound(const sfx_solver_params& s, const double* W) {
    return W[0] != 0. ? sqrt(s.gamma * W[D + 1] / W[0]) : 0.;
}

/* The solver's powers, sfx_pow's values (sfx_powq.h) in two out-of-line parts:
 * ln x as a pair, and x^y from it.  The iteration takes several powers of one
 * ratio p / p_K (f, f', the sampling), which share the logarithm.  Out of line
 * because the solver has some twenty power sites: inlined, its code overran
 * the instruction cache (21.5 of 27 stall cycles per issue were instruction
 * fetch; 807,000 random-field faces took 6.1 ms, then 0.82 ms). */
struct LogPair {
    double x, h, l; /* h is NaN where x is not a positive normal number */
};

__device__ __noinline__ LogPair xlog(double x) {
    LogPair p;
    p.x = x;
    if(!sfx_powq_log(x, &p.h, &p.l)) p.h = __longlong_as_double(0x7ff8000000000000ll);
    return p;
}

__device__ __noinline__ double xexp(LogPair p, double y) {
    const double th = y * p.h;
    const double tl = sfx_fma(y, p.h, -th) + y * p.l;
    double r;
    return sfx_powq_exp(th, tl, y, &r) ? r : sfx_pow_rare64(p.x, y);
}

__device__ __forceinline__ double xpow(double x, double y) {
    return xexp(xlog(x), y);
}

/* f_K(p) and, on a rarefaction side, ln(p / p_K) and z_K = (p/p_K)^((g-1)/(2g)) */
template <int D>
__device__ __forceinline__ double fb(const sfx_solver_params& s, double p, const double* Wb,
                                     double a, double* z, LogPair* lr) {
    if(p > Wb[D + 1]) {
        double A = s.tdgp1 / Wb[0];
        double B = s.gm1dgp1 * Wb[D + 1];
        *z = 0.;
        return (p - Wb[D + 1]) * sqrt(A / (p + B));
    }
    *lr = xlog(p / Wb[D + 1]);
    *z = xexp(*lr, s.gm1d2g);
    return s.tdgm1 * a * (*z - 1.);
}

template <int D>
__device__ __forceinline__ double gbf(const sfx_solver_params& s, double p,
                                      const double* Wb) {
    double A = s.tdgp1 / Wb[0];
    double B = s.gm1dgp1 * Wb[D + 1];
    return sqrt(A / (p + B));
}

/* f_K'(p), with lr = ln(p / p_K) on a rarefaction side */
template <int D>
__device__ __forceinline__ double fprimeb(const sfx_solver_params& s, double p,
                                          const double* Wb, double a, const LogPair& lr) {
    if(p > Wb[D + 1]) {
        double A = s.tdgp1 / Wb[0];
        double B = s.gm1dgp1 * Wb[D + 1];
        return (1. - 0.5 * (p - Wb[D + 1]) / (B + p)) * sqrt(A / (p + B));
    }
    return 1. / (Wb[0] * a) * xexp(lr, -s.gp1d2g);
}

/* The last f(p) of the iteration, per side, with its power
 * sfx_pow(p / p_K, (g-1)/(2g)) and the ratio's logarithm on a rarefaction
 * side.  The reference evaluates f_K(p) again for the wave velocity and that
 * power again for the sampling at the same p (ExactRiemannSolver.cpp:207-265):
 * the kept values are the same operations on the same operands, so reusing
 * them changes no bit. */
struct FLast {
    double p, fL, fR, zL, zR;
    LogPair lL, lR;
};

template <int D>
__device__ __forceinline__ double ffl(const sfx_solver_params& s, double p, const double* WL,
                                      const double* WR, double vL, double vR, double aL,
                                      double aR, FLast& c) {
    c.p = p;
    c.fL = fb<D>(s, p, WL, aL, &c.zL, &c.lL);
    c.fR = fb<D>(s, p, WR, aR, &c.zR, &c.lR);
    return c.fL + c.fR + (vR - vL);
}

template <int D>
__device__ __forceinline__ double fprime(const sfx_solver_params& s, const double* WL,
                                         const double* WR, double aL, double aR,
                                         const FLast& c) {
    return fprimeb<D>(s, c.p, WL, aL, c.lL) + fprimeb<D>(s, c.p, WR, aR, c.lR);
}

/* ExactRiemannSolver.cpp:644-673 */
template <int D>
__device__ double guess_p(const sfx_solver_params& s, const double* WL,
                          const double* WR, double vL, double vR, double aL,
                          double aR) {
    const double pL = WL[D + 1], pR = WR[D + 1];
    double pguess;
    const double pmin = (pR < pL) ? pR : pL;
    const double pmax = (pL < pR) ? pR : pL;
    const double qmax = pmax / pmin;
    double ppv = 0.5 * (pL + pR) - 0.125 * (vR - vL) * (WL[0] + WR[0]) * (aL + aR);
    double fl = s.tol * 0.5 * (pL + pR);
    ppv = (fl < ppv) ? ppv : fl;
    if(qmax <= 2. && pmin <= ppv && ppv <= pmax) {
        pguess = ppv;
    } else if(ppv < pmin) {
        pguess = xpow((aL + aR - s.gm1d2 * (vR - vL)) /
                                 (aL / xpow(pL, s.gm1d2g) + aR / xpow(pR, s.gm1d2g)),
                         s.tgdgm1);
    } else {
        const double gL = gbf<D>(s, ppv, WL), gR = gbf<D>(s, ppv, WR);
        pguess = (gL * pL + gR * pR - vR + vL) / (gL + gR);
    }
    fl = s.tol * 0.5 * (pL + pR);
    return (fl < pguess) ? pguess : fl;
}

/* ExactRiemannSolver.cpp:462-546, capped at SFX_MAX_ITER steps.  The limits'
 * function values fa and fbv come from the caller, which has evaluated f at
 * both of them. */
template <int D>
__device__ double brent(const sfx_solver_params& s, double lowerLimit,
                        double upperLimit, double fa, double fbv, double errorTol,
                        const double* WL, const double* WR, double vL, double vR, double aL,
                        double aR, FLast& last, int& iters, bool& errexit, bool& noconv) {
    double a = lowerLimit, b = upperLimit, c = 0., d = 1e230;
    double fc = 0., sv = 0., fs = 0.;
    if(fa * fbv >= 0) {
        errexit = true;
        return (fa < fbv) ? a : b;
    }
    if(fabs(fa) < fabs(fbv)) {
        double t = a;
        a = b;
        b = t;
        t = fa;
        fa = fbv;
        fbv = t;
    }
    c = a;
    fc = fa;
    bool mflag = true;
    while(!(fbv == 0) && (fabs(a - b) > errorTol * (a + b) * 0.5)) {
        if(iters >= SFX_MAX_ITER) {
            noconv = true;
            break;
        }
        ++iters;
        if((fa != fc) && (fbv != fc))
            sv = a * fbv * fc / (fa - fbv) / (fa - fc) +
                 b * fa * fc / (fbv - fa) / (fbv - fc) +
                 c * fa * fbv / (fc - fa) / (fc - fbv);
        else
            sv = b - fbv * (b - a) / (fbv - fa);
        const double tmp2 = (3. * a + b) / 4.;
        if(!(((sv > tmp2) && (sv < b)) || ((sv < tmp2) && (sv > b))) ||
           (mflag && (fabs(sv - b) >= (fabs(b - c) / 2.))) ||
           (!mflag && (fabs(sv - b) >= (fabs(c - d) / 2.))) ||
           (mflag && (fabs(b - c) < errorTol * (b + c) * 0.5)) ||
           (!mflag && (fabs(c - d) < errorTol * (c + d) * 0.5))) {
            sv = (a + b) / 2.;
            mflag = true;
        } else {
            mflag = false;
        }
        fs = ffl<D>(s, sv, WL, WR, vL, vR, aL, aR, last);
        d = c;
        c = b;
        fc = fbv;
        if(fa * fs < 0.) {
            b = sv;
            fbv = fs;
        } else {
            a = sv;
            fa = fs;
        }
        if(fabs(fa) < fabs(fbv)) {
            double t = a;
            a = b;
            b = t;
            t = fa;
            fa = fbv;
            fbv = t;
        }
    }
    return b;
}

template <int D>
__device__ __forceinline__ bool bad_state(const double* sol) {
    bool bad = (sol[0] < 0.) || (sol[0] != sol[0]);
#pragma unroll
    for(int k = 0; k < D; ++k) bad |= (sol[1 + k] != sol[1 + k]);
    bad |= (sol[D + 1] < 0.) || (sol[D + 1] != sol[D + 1]);
    return bad;
}

/* rarefaction fan state next to vacuum or at the interface; shared shape of
 * ExactRiemannSolver.cpp:318-330 / 350-362 and HLLCRiemannSolver.cpp:59-71 */
template <int D>
__device__ __forceinline__ void fan_left(double g, const double* WL, double vL,
                                         double aL, double* sol, double* vhalf) {
    const LogPair base = xlog(2. / (g + 1.) + (g - 1.) / (g + 1.) / aL * vL);
    sol[0] = WL[0] * xexp(base, 2. / (g - 1.));
    *vhalf = 2. / (g + 1.) * (aL + 0.5 * (g - 1.) * vL) - vL;
    sol[D + 1] = WL[D + 1] * xexp(base, 2. * g / (g - 1.));
}

template <int D>
__device__ __forceinline__ void fan_right(double g, const double* WR, double vR,
                                          double aR, double* sol, double* vhalf) {
    const LogPair base = xlog(2. / (g + 1.) - (g - 1.) / (g + 1.) / aR * vR);
    sol[0] = WR[0] * xexp(base, 2. / (g - 1.));
    *vhalf = 2. / (g + 1.) * (-aR + 0.5 * (g - 1.) * vR) - vR;
    sol[D + 1] = WR[D + 1] * xexp(base, 2. * g / (g - 1.));
}

/* vacuum sampling shared by ExactRiemannSolver::solve_vacuum
 * (ExactRiemannSolver.cpp:304-446) and HLLCRiemannSolver::vacuum_flux's
 * first half (HLLCRiemannSolver.cpp:44-156); the conditions are written in
 * the two sources with the operands swapped but are the same predicates */
template <int D>
__device__ void vacuum_sample(double g, const double* WL, const double* WR,
                              double vL, double vR, double aL, double aR,
                              const double* n, double* sol, int* code) {
    constexpr int S = D + 2;
    double vhalf = 0.;
    if(WR[0] == 0.) {
#pragma unroll
        for(int k = 0; k < S; ++k) sol[k] = WL[k];
        if(vL < aL) {
            double SL = vL + 2. * aL / (g - 1.);
            if(SL > 0.) {
                fan_left<D>(g, WL, vL, aL, sol, &vhalf);
                *code = 2 | SFX_BRANCH_S_LFAN;
            } else {
#pragma unroll
                for(int k = 0; k < S; ++k) sol[k] = 0.;
                *code = 2 | SFX_BRANCH_S_VAC;
            }
        } else {
            *code = 2 | SFX_BRANCH_S_LUP;
        }
    } else if(WL[0] == 0.) {
#pragma unroll
        for(int k = 0; k < S; ++k) sol[k] = WR[k];
        if(-aR < vR) {
            double SR = vR - 2. * aR / (g - 1.);
            if(SR >= 0.) {
#pragma unroll
                for(int k = 0; k < S; ++k) sol[k] = 0.;
                *code = 3 | SFX_BRANCH_S_VAC;
            } else {
                fan_right<D>(g, WR, vR, aR, sol, &vhalf);
                *code = 3 | SFX_BRANCH_S_RFAN;
            }
        } else {
            *code = 3 | SFX_BRANCH_S_RUP;
        }
    } else {
        double SR = vR - 2. * aR / (g - 1.);
        double SL = vL + 2. * aL / (g - 1.);
        if(SR > 0. && SL < 0.) {
#pragma unroll
            for(int k = 0; k < S; ++k) sol[k] = 0.;
            *code = 4 | SFX_BRANCH_S_VAC;
        } else if(SL >= 0.) {
#pragma unroll
            for(int k = 0; k < S; ++k) sol[k] = WL[k];
            if(aL > vL) {
                fan_left<D>(g, WL, vL, aL, sol, &vhalf);
                *code = 4 | SFX_BRANCH_S_LFAN;
            } else {
                *code = 4 | SFX_BRANCH_S_LUP;
            }
        } else {
#pragma unroll
            for(int k = 0; k < S; ++k) sol[k] = WR[k];
            if(-aR < vR) {
                fan_right<D>(g, WR, vR, aR, sol, &vhalf);
                *code = 4 | SFX_BRANCH_S_RFAN;
            } else {
                *code = 4 | SFX_BRANCH_S_RUP;
            }
        }
    }
#pragma unroll
    for(int k = 0; k < D; ++k) sol[1 + k] = sol[1 + k] + vhalf * n[k];
}

/* ExactRiemannSolver::solve (ExactRiemannSolver.cpp:108-290).  WR becomes WL
 * for a reflective face, as in the reference. */
template <int D>
__device__ ExactOut exact_solve(const sfx_solver_params& s, double* WL, double* WR,
                                const double* n, bool reflective, double* sol) {
    constexpr int S = D + 2;
    ExactOut out{SFX_OK, 0};
    double vL = WL[1] * n[0] + WL[2] * n[1];
    double vR = WR[1] * n[0] + WR[2] * n[1];
    if(D == 3) {
        vL = vL + WL[3] * n[2];
        vR = vR + WR[3] * n[2];
    }
    if(reflective) {
#pragma unroll
        for(int k = 0; k < S; ++k) WR[k] = WL[k];
        vR = -vL;
    }
    const double aL = sound<D>(s, WL), aR = sound<D>(s, WR);
    const double g = s.gamma;
    if(WL[0] == 0. || WR[0] == 0.) {
        if(WR[0] == 0. && WL[0] == 0.) {
#pragma unroll
            for(int k = 0; k < S; ++k) sol[k] = 0.;
            out.code = 1;
            return out;
        }
        vacuum_sample<D>(g, WL, WR, vL, vR, aL, aR, n, sol, &out.code);
        if(bad_state<D>(sol)) out.status = SFX_ERR_RIEMANN;
        return out;
    }
    if(2. * aL / (g - 1.) + 2. * aR / (g - 1.) <= vR - vL) {
        vacuum_sample<D>(g, WL, WR, vL, vR, aL, aR, n, sol, &out.code);
        if(bad_state<D>(sol)) out.status = SFX_ERR_RIEMANN;
        return out;
    }
    const double tol = s.tol;
    double p = 0.;
    double pguess = guess_p<D>(s, WL, WR, vL, vR, aL, aR);
    FLast last;
    last.lL = last.lR = LogPair{0., 0., 0.};
    /* f(0): on both sides the rarefaction branch with sfx_pow(0, e) = +0
     * (e > 0), i.e. (2/(g-1) a_K) * (0 - 1) exactly */
    const double fp = WL[D + 1] > 0. && WR[D + 1] > 0.
                              ? s.tdgm1 * aL * (0. - 1.) + s.tdgm1 * aR * (0. - 1.) + (vR - vL)
                              : ffl<D>(s, p, WL, WR, vL, vR, aL, aR, last);
    double fpguess;
    int newton = 0, brent_it = 0, mode;
    bool errexit = false, noconv = false;
    /* The reference has one Newton loop per mode: below the cutoff it runs to
     * the tolerance with p kept non-negative; above it, only while f < 0 (and
     * not at all when f(0) and f(guess) differ in sign).  One loop here, and one
     * evaluation site. */
    const bool only_newton = fp < s.cutoff;
    for(;;) {
        fpguess = ffl<D>(s, pguess, WL, WR, vL, vR, aL, aR, last);
        if(newton == 0 && !(only_newton || fp * fpguess >= 0.)) break;
        if(!(fabs(p - pguess) > tol * 0.5 * (p + pguess) && (only_newton || fpguess < 0.))) break;
        if(newton >= SFX_MAX_ITER) {
            noconv = true;
            break;
        }
        ++newton;
        p = pguess;
        pguess = pguess - fpguess / fprime<D>(s, WL, WR, aL, aR, last);
        if(only_newton && pguess < 0.) pguess = 0.;
    }
    if(only_newton) {
        mode = 1 << 3;
        p = pguess;
    } else {
        mode = 2 << 3;
        if(!noconv && fabs(p - pguess) > tol * 0.5 * (p + pguess) && fpguess > 0.) {
            mode = 3 << 3;
            p = brent<D>(s, 0., pguess, fp, fpguess, tol, WL, WR, vL, vR, aL, aR, last, brent_it,
                         errexit, noconv);
        } else {
            p = pguess;
        }
    }
    if(last.p != p) ffl<D>(s, p, WL, WR, vL, vR, aL, aR, last);
    const double u = 0.5 * (vL + vR) + 0.5 * (last.fR - last.fL);
    double vhalf;
    int region;
    if(u < 0) {
#pragma unroll
        for(int k = 0; k < S; ++k) sol[k] = WR[k];
        const double pdpR = p / WR[D + 1];
        if(p > WR[D + 1]) {
            const double SR = vR + aR * sqrt(s.gp1d2g * pdpR + s.gm1d2g);
            if(SR > 0) {
                sol[0] = WR[0] * (pdpR + s.gm1dgp1) / (s.gm1dgp1 * pdpR + 1.);
                sol[D + 1] = p;
                vhalf = u - vR;
                region = SFX_BRANCH_S_RSHOCK_STAR;
            } else {
                vhalf = 0.;
                region = SFX_BRANCH_S_RUP_SHOCK;
            }
        } else {
            const double SHR = vR + aR;
            if(SHR > 0) {
                const double STR = u + aR * last.zR;
                if(STR <= 0) {
                    const LogPair base = xlog(s.tdgp1 - s.gm1dgp1 / aR * vR);
                    sol[0] = WR[0] * xexp(base, s.tdgm1);
                    vhalf = s.tdgp1 * (-aR + s.gm1d2 * vR) - vR;
                    sol[D + 1] = WR[D + 1] * xexp(base, s.tgdgm1);
                    region = SFX_BRANCH_S_RFAN;
                } else {
                    sol[0] = WR[0] * xexp(last.lR, s.ginv);
                    sol[D + 1] = p;
                    vhalf = u - vR;
                    region = SFX_BRANCH_S_RRARE_STAR;
                }
            } else {
                vhalf = 0.;
                region = SFX_BRANCH_S_RUP;
            }
        }
    } else {
#pragma unroll
        for(int k = 0; k < S; ++k) sol[k] = WL[k];
        const double pdpL = p / WL[D + 1];
        if(p > WL[D + 1]) {
            const double SL = vL - aL * sqrt(s.gp1d2g * pdpL + s.gm1d2g);
            if(SL < 0) {
                sol[0] = WL[0] * (pdpL + s.gm1dgp1) / (s.gm1dgp1 * pdpL + 1.);
                sol[D + 1] = p;
                vhalf = u - vL;
                region = SFX_BRANCH_S_LSHOCK_STAR;
            } else {
                vhalf = 0.;
                region = SFX_BRANCH_S_LUP_SHOCK;
            }
        } else {
            const double SHL = vL - aL;
            if(SHL < 0) {
                const double STL = u - aL * last.zL;
                if(STL > 0) {
                    const LogPair base = xlog(s.tdgp1 + s.gm1dgp1 / aL * vL);
                    sol[0] = WL[0] * xexp(base, s.tdgm1);
                    vhalf = s.tdgp1 * (aL + s.gm1d2 * vL) - vL;
                    sol[D + 1] = WL[D + 1] * xexp(base, s.tgdgm1);
                    region = SFX_BRANCH_S_LFAN;
                } else {
                    sol[0] = WL[0] * xexp(last.lL, s.ginv);
                    vhalf = u - vL;
                    sol[D + 1] = p;
                    region = SFX_BRANCH_S_LRARE_STAR;
                }
            } else {
                vhalf = 0.;
                region = SFX_BRANCH_S_LUP;
            }
        }
    }
#pragma unroll
    for(int k = 0; k < D; ++k) sol[1 + k] = sol[1 + k] + vhalf * n[k];
    out.code = mode | region | (min(newton, 127) << 9) | (min(brent_it, 127) << 16) |
               (errexit ? (1 << 23) : 0);
    if(noconv)
        out.status = SFX_ERR_NOCONV;
    else if(bad_state<D>(sol))
        out.status = SFX_ERR_RIEMANN;
    return out;
}

/* ExactRiemannSolver::get_flux (:815-836) contracted with the normal
 * (solve_for_flux :858-880) */
template <int D>
__device__ __forceinline__ void exact_flux_from_half(double gamma, const double* Wh,
                                                     const double* v, const double* n,
                                                     double* flux) {
    constexpr int S = D + 2;
    double F[D][S];
#pragma unroll
    for(int idx = 0; idx < D; ++idx) {
#pragma unroll
        for(int k = 0; k < S; ++k) F[idx][k] = 0.;
        if(Wh[0] == 0.) continue;
        const double un = Wh[1 + idx] - v[idx];
        F[idx][0] = Wh[0] * un;
        F[idx][1] = Wh[0] * un * Wh[1];
        F[idx][2] = Wh[0] * un * Wh[2];
        if(D == 3) F[idx][3] = Wh[0] * un * Wh[3];
        double v2 = Wh[1] * Wh[1] + Wh[2] * Wh[2];
        if(D == 3) v2 = v2 + Wh[3] * Wh[3];
        const double e = 0.5 * Wh[0] * v2 + Wh[D + 1] / (gamma - 1.);
        F[idx][1 + idx] = F[idx][1 + idx] + Wh[D + 1];
        F[idx][D + 1] = un * e + Wh[D + 1] * Wh[1 + idx];
    }
#pragma unroll
    for(int k = 0; k < S; ++k) {
        double s = F[0][k] * n[0] + F[1][k] * n[1];
        if(D == 3) s = s + F[2][k] * n[2];
        flux[k] = s;
    }
}

/* ----------------------------- HLLC solver ----------------------------- */
template <int D>
__device__ __forceinline__ void hllc_deboost(const double* v, double* flux) {
    flux[1] = flux[1] + v[0] * flux[0];
    flux[2] = flux[2] + v[1] * flux[0];
    if(D == 3) {
        flux[3] = flux[3] + v[2] * flux[0];
        const double nrm2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
        flux[4] = flux[4] + (v[0] * flux[1] + v[1] * flux[2] + v[2] * flux[3] +
                             0.5 * nrm2 * flux[0]);
    } else {
        const double nrm2 = v[0] * v[0] + v[1] * v[1];
        flux[D + 1] = flux[D + 1] + (v[0] * flux[1] + v[1] * flux[2] + 0.5 * nrm2 * flux[0]);
    }
}

/* HLLCRiemannSolver::solve_for_flux (HLLCRiemannSolver.cpp:258-403) */
template <int D>
__device__ int hllc_flux(const sfx_solver_params& s, double* WL, double* WR,
                         const double* n, const double* v, bool reflective,
                         double* flux) {
    constexpr int S = D + 2;
    const double g = s.gamma;
    int code = SFX_BRANCH_HLLC;
#pragma unroll
    for(int k = 0; k < S; ++k) flux[k] = 0.;
    if(WL[0] == 0. && (reflective || WR[0] == 0.)) return code | 1;
    double uL = WL[1] * n[0] + WL[2] * n[1];
    double uR = WR[1] * n[0] + WR[2] * n[1];
    if(D == 3) {
        uL = uL + WL[3] * n[2];
        uR = uR + WR[3] * n[2];
    }
    if(reflective) {
#pragma unroll
        for(int k = 0; k < S; ++k) WR[k] = WL[k];
        uR = -uL;
    }
    const double aL = sqrt(g * WL[D + 1] / WL[0]);
    const double aR = sqrt(g * WR[D + 1] / WR[0]);
    if(WL[0] == 0. || WR[0] == 0. || 2. * aL / (g - 1.) + 2. * aR / (g - 1.) <= uR - uL) {
        double sol[S];
        int vc = 0;
        vacuum_sample<D>(g, WL, WR, uL, uR, aL, aR, n, sol, &vc);
        code |= vc;
        if(sol[0] == 0.) return code;
        double vsol = sol[1] * n[0] + sol[2] * n[1];
        double v2 = sol[1] * sol[1] + sol[2] * sol[2];
        if(D == 3) {
            vsol = vsol + sol[3] * n[2];
            v2 = v2 + sol[3] * sol[3];
        }
        flux[0] = sol[0] * vsol;
        flux[1] = sol[0] * sol[1] * vsol + sol[D + 1] * n[0];
        flux[2] = sol[0] * sol[2] * vsol + sol[D + 1] * n[1];
        if(D == 3) flux[3] = sol[0] * sol[3] * vsol + sol[D + 1] * n[2];
        const double e = sol[D + 1] / (g - 1.) / sol[0] + 0.5 * v2;
        flux[D + 1] = sol[0] * e * vsol + sol[D + 1] * vsol;
        hllc_deboost<D>(v, flux);
        return code;
    }
    const double rhobar = 0.5 * (WL[0] + WR[0]);
    const double abar = 0.5 * (aL + aR);
    const double pPVRS = 0.5 * (WL[D + 1] + WR[D + 1]) - 0.5 * (uR - uL) * rhobar * abar;
    const double pstar = (0. < pPVRS) ? pPVRS : 0.;
    double qL = 1., qR = 1.;
    if(pstar > WL[D + 1]) qL = sqrt(1. + 0.5 * (g + 1.) / g * (pstar / WL[D + 1] - 1.));
    if(pstar > WR[D + 1]) qR = sqrt(1. + 0.5 * (g + 1.) / g * (pstar / WR[D + 1] - 1.));
    const double SL = uL - aL * qL;
    const double SR = uR + aR * qR;
    const double Sstar = (WR[D + 1] - WL[D + 1] + WL[0] * uL * (SL - uL) -
                          WR[0] * uR * (SR - uR)) /
                         (WL[0] * (SL - uL) - WR[0] * (SR - uR));
    const bool left = Sstar >= 0.;
    const double* Wk = left ? WL : WR;
    const double uk = left ? uL : uR;
    const double Sk = left ? SL : SR;
    flux[0] = Wk[0] * uk;
    flux[1] = Wk[0] * Wk[1] * uk + Wk[D + 1] * n[0];
    flux[2] = Wk[0] * Wk[2] * uk + Wk[D + 1] * n[1];
    double v2 = Wk[1] * Wk[1] + Wk[2] * Wk[2];
    if(D == 3) {
        flux[3] = Wk[0] * Wk[3] * uk + Wk[D + 1] * n[2];
        v2 = v2 + Wk[3] * Wk[3];
    }
    const double ek = Wk[D + 1] / (g - 1.) / Wk[0] + 0.5 * v2;
    flux[D + 1] = Wk[0] * ek * uk + Wk[D + 1] * uk;
    const bool star = left ? (SL < 0.) : (SR > 0.);
    if(star) {
        double U[S];
        U[0] = 1.;
        U[1] = Wk[1] + (Sstar - uk) * n[0];
        U[2] = Wk[2] + (Sstar - uk) * n[1];
        if(D == 3) U[3] = Wk[3] + (Sstar - uk) * n[2];
        U[D + 1] = ek + (Sstar - uk) * (Sstar + Wk[D + 1] / (Wk[0] * (Sk - uk)));
        const double fac = Wk[0] * (Sk - uk) / (Sk - Sstar);
#pragma unroll
        for(int k = 0; k < S; ++k) U[k] = U[k] * fac;
        flux[0] = flux[0] + Sk * (U[0] - Wk[0]);
        flux[1] = flux[1] + Sk * (U[1] - Wk[0] * Wk[1]);
        flux[2] = flux[2] + Sk * (U[2] - Wk[0] * Wk[2]);
        if(D == 3) flux[3] = flux[3] + Sk * (U[3] - Wk[0] * Wk[3]);
        flux[D + 1] = flux[D + 1] + Sk * (U[D + 1] - Wk[0] * ek);
    }
    code |= left ? (star ? SFX_BRANCH_HLLC_LSTAR : SFX_BRANCH_HLLC_L)
                 : (star ? SFX_BRANCH_HLLC_RSTAR : SFX_BRANCH_HLLC_R);
    hllc_deboost<D>(v, flux);
    return code;
}

/* -------------------------------- faces -------------------------------- */

/* MUSCL-Hancock prediction + reconstruction + pairwise limiter + positivity
 * fallbacks for one side (VorFace.cpp:715-759 right, 762-804 left); dW0 is
 * dW/dt at Wt, w = |d| / |centroid difference| */
template <int D>
__device__ __forceinline__ void predict_side(double dt, double* Wt, const double* Wself,
                                             const double* Wother, const double (*g)[D + 2],
                                             const double* dW0, const double* d, bool do_limit,
                                             double w) {
    constexpr int S = D + 2;
    double dW[S];
#pragma unroll
    for(int k = 0; k < S; ++k) dW[k] = 0.5 * dt * dW0[k];
    reconstruct<D>(Wt, g, d);
    if(do_limit) {
#pragma unroll
        for(int k = 0; k < S; ++k) Wt[k] = limit1<D>(Wt[k], Wself[k], Wother[k], w);
    }
    if(Wt[0] < 0. || Wt[D + 1] < 0.) {
#pragma unroll
        for(int k = 0; k < S; ++k) Wt[k] = Wself[k];
    }
#pragma unroll
    for(int k = 0; k < S; ++k) Wt[k] = Wt[k] + dW[k];
    if(Wt[0] < 0. || Wt[D + 1] < 0.) {
#pragma unroll
        for(int k = 0; k < S; ++k) Wt[k] = Wt[k] - dW[k];
    }
}

/* what a face's flux needs of the mesh */
template <int D>
struct FaceGeom {
    int iL, iR; /* iR = -1: mirror */
    double A, facL, facR, wL, wR, dL[D], dR[D], n[D];
};

/* from positions, as the reference forms it (caller-owned arrays) */
template <int D>
__device__ __forceinline__ void face_geom(const sfx_dmesh& m, int f, FaceGeom<D>& q) {
    const int n = m.n_cells, F = m.n_faces;
    const int iL = q.iL, iR = q.iR < 0 ? 0 : q.iR;
    const bool has_right = q.iR >= 0;
    double dd[D], cd[D];
#pragma unroll
    for(int l = 0; l < D; ++l) {
        const double mid = m.mid[(size_t)l * F + f];
        const double xL = m.pos[(size_t)l * n + iL];
        const double xRi = m.rpos[(size_t)l * F + f];
        const double cenL = m.cen[(size_t)l * n + iL];
        q.dL[l] = mid - cenL + (xL - xL);
        q.dR[l] = 0.;
        cd[l] = 0.;
        if(has_right) {
            const double cenR = m.cen[(size_t)l * n + iR], xR = m.pos[(size_t)l * n + iR];
            q.dR[l] = mid - cenR + (xR - xRi);
            cd[l] = cenL - cenR;
        }
        dd[l] = xL - xRi;
    }
    const double r = norm<D>(cd);
    q.wL = has_right ? sqrt(dot<D>(q.dL, q.dL)) / r : 0.;
    q.wR = has_right ? sqrt(dot<D>(q.dR, q.dR)) / r : 0.;
    q.facL = q.A / m.tarea[iL];
    q.facR = has_right ? q.A / m.tarea[iR] : 0.;
    /* VorFace::get_normal (VorFace.cpp:553-571) */
    const double dn = norm<D>(dd);
#pragma unroll
    for(int l = 0; l < D; ++l) q.n[l] = -dd[l] / dn;
}

/* kFaceArrays: field-major arrays (caller-owned, or of a mesh without records).  kFaceRecords: a mesh's
 * records, dW/dt from the cell's (a static mesh with one step).
 * kFaceMoving: records, face velocities and local time steps, dW/dt formed
 * here (at the boosted state; a cell in the middle of its step keeps its
 * gradients).
 * What a face needs of its two cells is one gather of 2 + 5 (2D: 2 + 3)
 * 32-byte loads per side and its own geometry planes of 32 bytes that
 * consecutive threads read consecutively; from field-major arrays it was 28
 * (20) scattered doubles per side and the geometry's square roots and
 * divisions on every step.  HLLC: 101 -> 55 us on 65,537 cells (500,000 faces)
 * in 3D, 71 -> 44 us on 150,001 in 2D (67 and 51 with 16-byte loads); bound by
 * FP64 latency at 16 warps per SM (118 registers; 5 or 6 blocks of 128 per SM
 * took the same time). */
constexpr int kFaceArrays = 0, kFaceRecords = 1, kFaceMoving = 2;

/* a face's Riemann problem and what its dQ needs: predicted states, normal,
 * face velocity, dt A, and the over-flux limits (VorFace.cpp:837-866) */
template <int D>
struct FaceProblem {
    double WL[D + 2], WR[D + 2], n[D], v[D];
    double dtA, limL, limR;
    bool has_right;
};

template <int D, bool REC>
__device__ __forceinline__ void store_dQ(const sfx_dmesh& m, int f, const double* v) {
    constexpr int S = D + 2;
    if(REC) {
        double t[Rec<D>::dq];
#pragma unroll
        for(int k = 0; k < Rec<D>::dq; ++k) t[k] = k < S ? v[k < S ? k : 0] : 0.;
        store_record<Rec<D>::dq>(m.dQf + (size_t)f * Rec<D>::dq, t);
    } else {
#pragma unroll
        for(int k = 0; k < S; ++k) m.dQf[(size_t)k * m.n_faces + f] = v[k];
    }
}

/* The MUSCL-Hancock half of calculate_flux (VorFace.cpp:670-838); false:
 * nothing to solve (zero area, no active cell), dQ is zero */
template <int D, int MODE>
__device__ __forceinline__ bool face_problem(const sfx_dmesh& m, const sfx_solver_params& sp,
                                             double dt, int f, int write_branch,
                                             FaceProblem<D>& q) {
    using R = Rec<D>;
    constexpr int S = D + 2;
    constexpr bool REC = MODE != kFaceArrays;
    const int n = m.n_cells, F = m.n_faces;
    auto skip = [&]() {
        double z[S];
#pragma unroll
        for(int k = 0; k < S; ++k) z[k] = 0.;
        store_dQ<D, REC>(m, f, z);
        if(write_branch) m.branch[f] = SFX_BRANCH_SKIPPED;
    };
    FaceGeom<D> g;
    if(REC) {
        double h[R::fgeo];
#pragma unroll
        for(int k = 0; k < R::fgeo; k += 4)
            load_record<4>(m.fgeo + (size_t)k * F + 4 * (size_t)f, h + k);
        g.iL = __double2loint(h[0]);
        g.iR = __double2hiint(h[0]);
        g.A = h[1];
        g.facL = h[2];
        g.facR = h[3];
        g.wL = h[4];
        g.wR = h[5];
#pragma unroll
        for(int l = 0; l < D; ++l) {
            g.dL[l] = h[6 + l];
            g.dR[l] = h[6 + D + l];
            g.n[l] = h[6 + 2 * D + l];
        }
    } else {
        g.A = m.area[f];
        g.iL = m.left[f];
        g.iR = m.kind[f] == SFX_FACE_MIRROR ? -1 : m.right[f];
    }
    if(g.A == 0.) {
        skip();
        return false;
    }
    const int iL = g.iL;
    const bool has_right = g.iR >= 0;
    const int iR = has_right ? g.iR : 0;
    /* local time steps (VorFace.cpp:672-697): a face is computed when its
     * left cell is active, or (with a right cell) either cell is; its time
     * step is the shorter of the two cells' steps; the limits' timefac is that
     * over the longer one (dt / dt with one global step) */
    double dtmax = dt;
    if(MODE != kFaceRecords && m.local) {
        const bool aL = m.tstart[iL] == m.t_now;
        const bool aR = has_right && m.tstart[iR] == m.t_now;
        if(!aL && !aR) {
            skip();
            return false;
        }
        dt = sfx_realtime(m.t_total, m.tend[iL] - m.tstart[iL]);
        dtmax = dt;
        if(has_right) {
            const double dtR = sfx_realtime(m.t_total, m.tend[iR] - m.tstart[iR]);
            dt = fmin(dt, dtR);
            dtmax = fmax(dtmax, dtR);
        }
    }
    if(!REC) face_geom<D>(m, f, g);
    q.has_right = has_right;
#pragma unroll
    for(int l = 0; l < D; ++l) {
        q.n[l] = g.n[l];
        q.v[l] = MODE != kFaceRecords && m.vel ? m.vel[(size_t)l * F + f] : 0.;
    }
    double WRrec[S], Wt[S];
    double QLm, QRm = 0.;
    auto load_state = [&](int i, double* W, double& Qm) {
        if(REC) {
            double t[8];
            load_record<8>(m.ws + (size_t)i * R::ws, t);
#pragma unroll
            for(int k = 0; k < S; ++k) W[k] = t[k];
            Qm = t[S];
        } else {
#pragma unroll
            for(int k = 0; k < S; ++k) W[k] = m.W[(size_t)k * n + i];
            Qm = m.Q[i];
        }
    };
    double* WL = q.WL;
    double* WR = q.WR;
    load_state(iL, WL, QLm);
#pragma unroll
    for(int k = 0; k < S; ++k) {
        WR[k] = 0.;
        WRrec[k] = 0.;
    }
    if(has_right) load_state(iR, WR, QRm);
    if(MODE != kFaceRecords) {
#pragma unroll
        for(int l = 0; l < D; ++l) {
            WL[1 + l] = WL[1 + l] - q.v[l];
            WR[1 + l] = WR[1 + l] - q.v[l];
        }
    }
    /* gradients of cell i, and dW/dt at its (boosted) state W */
    auto load_slopes = [&](int i, const double* W, double (*gr)[S], double* dW0) {
        if(REC) {
            double t[R::grec];
            load_record<R::grec>(m.grec + (size_t)i * R::grec, t);
#pragma unroll
            for(int l = 0; l < D; ++l)
#pragma unroll
                for(int k = 0; k < S; ++k) gr[l][k] = t[l * S + k];
#pragma unroll
            for(int k = 0; k < S; ++k) dW0[k] = t[D * S + k];
        } else {
#pragma unroll
            for(int l = 0; l < D; ++l)
#pragma unroll
                for(int k = 0; k < S; ++k) gr[l][k] = m.grad[((size_t)l * S + k) * n + i];
        }
        if(MODE != kFaceRecords) time_derivative<D>(sp.gamma, W, gr, dW0);
    };
    if(has_right) {
        double gr[D][S], dW0[S];
        load_slopes(iR, WR, gr, dW0);
#pragma unroll
        for(int k = 0; k < S; ++k) Wt[k] = WR[k];
        predict_side<D>(dt, Wt, WR, WL, gr, dW0, g.dR, true, g.wR);
#pragma unroll
        for(int k = 0; k < S; ++k) WRrec[k] = Wt[k];
    }
    {
        double gr[D][S], dW0[S];
        load_slopes(iL, WL, gr, dW0);
#pragma unroll
        for(int k = 0; k < S; ++k) Wt[k] = WL[k];
        predict_side<D>(dt, Wt, WL, WR, gr, dW0, g.dL, has_right, g.wL);
    }
    if(WL[0] != 0.) {
#pragma unroll
        for(int k = 0; k < S; ++k) WL[k] = Wt[k];
    }
    if(WR[0] != 0.) {
#pragma unroll
        for(int k = 0; k < S; ++k) WR[k] = WRrec[k];
    }
    double timefac = 1.;
    if(MODE != kFaceRecords && has_right) timefac = dt / dtmax;
    q.dtA = dt * g.A;
    q.limL = g.facL * timefac * QLm;
    q.limR = g.facR * timefac * QRm;
    return true;
}

/* dt A flux with the over-flux limiter into the face's dQ; its branch code and
 * status */
template <int D, bool REC>
__device__ __forceinline__ void face_dQ(const sfx_dmesh& m, int f, const double* flux,
                                        double dtA, double limL, double limR, bool has_right,
                                        int code, int status, int write_branch) {
    constexpr int S = D + 2;
    double dQL[S], dQR[S];
#pragma unroll
    for(int k = 0; k < S; ++k) {
        dQL[k] = dtA * flux[k];
        dQR[k] = -dtA * flux[k];
    }
    if(dQL[0] > limL) {
        const double corfac = fabs(limL / dQL[0]);
#pragma unroll
        for(int k = 0; k < S; ++k) dQL[k] = dQL[k] * corfac;
#pragma unroll
        for(int k = 0; k < S; ++k) dQR[k] = -1. * dQL[k];
        code |= SFX_BRANCH_LIMIT_L;
    }
    if(has_right) {
        if(dQR[0] > limR) {
            const double corfac = fabs(limR / dQR[0]);
#pragma unroll
            for(int k = 0; k < S; ++k) dQR[k] = dQR[k] * corfac;
#pragma unroll
            for(int k = 0; k < S; ++k) dQL[k] = -1. * dQR[k];
            code |= SFX_BRANCH_LIMIT_R;
        }
    }
    store_dQ<D, REC>(m, f, dQL);
    if(write_branch) m.branch[f] = code;
    if(status == SFX_OK && flux[0] != flux[0]) status = SFX_ERR_NAN_FLUX;
    if(status != SFX_OK) report_face(m.err, f, status);
}

/* the exact solver's half state and flux in a face's frame */
template <int D>
__device__ __forceinline__ ExactOut exact_face(const sfx_solver_params& sp, double* WL,
                                               double* WR, const double* n, const double* v,
                                               bool has_right, double* flux) {
    double half[D + 2];
    const ExactOut eo = exact_solve<D>(sp, WL, WR, n, !has_right, half);
#pragma unroll
    for(int l = 0; l < D; ++l) half[1 + l] = half[1 + l] + v[l];
    exact_flux_from_half<D>(sp.gamma, half, v, n, flux);
    return eo;
}

/* one thread per face: HLLC, and both solvers on caller-owned arrays */
template <int D, int SOLVER, int MODE>
__global__ void __launch_bounds__(128) k_faces(sfx_dmesh m, sfx_solver_params sp,
                                               double dt, int write_branch) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if(f >= sfx_flux_faces(m) || failed(m.err)) return;
    FaceProblem<D> q;
    if(!face_problem<D, MODE>(m, sp, dt, f, write_branch, q)) return;
    double flux[D + 2];
    int status = SFX_OK, code;
    if(SOLVER == SFX_SOLVER_EXACT) {
        const ExactOut eo = exact_face<D>(sp, q.WL, q.WR, q.n, q.v, q.has_right, flux);
        status = eo.status;
        code = eo.code;
    } else {
        code = hllc_flux<D>(sp, q.WL, q.WR, q.n, q.v, !q.has_right, flux);
    }
    face_dQ<D, MODE != kFaceArrays>(m, f, flux, q.dtA, q.limL, q.limR, q.has_right, code,
                                    status, write_branch);
}

/* ------------------- exact solver: faces sorted by wave pattern -------------------
 * The iteration's cost depends on the face: which side is a shock and which a
 * rarefaction (different code on each side, and powers on a rarefaction), and
 * whether f(0) lies under the cutoff (Newton alone, a few steps) or not (5% of
 * a random field's faces; 2% then take Brent's method, about 30 evaluations).
 * One thread per face ran 9.5 of 32 lanes.  So a block sorts its faces by
 * wave pattern through shared memory and its threads solve them in that order;
 * faces with f(0) above the cutoff go to a list that k_faces_listed solves,
 * full warps of them (they would leave every block a warp of six running ten
 * times as long as the others).  The keys are formed in FP32: they decide
 * which thread solves a face and nothing else.  807,000 random-field faces in
 * 3D: 735 -> 254 us and 86 us for the list's 5%; bound by FP64 latency (16 warps
 * per SM at 128 registers).  The two rarefactions' powers interleaved, inline,
 * for more independent operations: 297 us (registers and code). */
constexpr int kExactBlock = 256, kKeys = 8, kKeyListed = 8, kKeyNone = 9;

template <int D>
__device__ __forceinline__ int wave_key(const sfx_solver_params& s, const FaceProblem<D>& q) {
    const float rL = (float)q.WL[0], pL = (float)q.WL[D + 1];
    const float rR = q.has_right ? (float)q.WR[0] : rL;
    const float pR = q.has_right ? (float)q.WR[D + 1] : pL;
    float vL = 0.f, vR = 0.f;
#pragma unroll
    for(int l = 0; l < D; ++l) {
        vL += (float)q.WL[1 + l] * (float)q.n[l];
        vR += (float)q.WR[1 + l] * (float)q.n[l];
    }
    if(!q.has_right) vR = -vL;
    const float g = (float)s.gamma, tdgm1 = (float)s.tdgm1, e = (float)s.gm1d2g;
    const float aL = sqrtf(__fdividef(g * pL, rL)), aR = sqrtf(__fdividef(g * pR, rR));
    const float dv = vR - vL;
    const float f0 = dv - tdgm1 * (aL + aR);
    if(!(f0 < 0.f)) return kKeys - 1; /* vacuum (or no number): no iteration */
    if(f0 >= (float)s.cutoff) return kKeyListed;
    const bool lowL = pL <= pR;
    const float pmin = lowL ? pL : pR, pmax = lowL ? pR : pL;
    /* f(p_min): the lower side contributes 0, the other one rarefies;
     * f(p_max): the lower side is a shock, the other one contributes 0 */
    const float fmin = tdgm1 * (lowL ? aR : aL) *
                               (exp2f(e * __log2f(__fdividef(pmin, pmax))) - 1.f) +
                       dv;
    const float A = __fdividef((float)s.tdgp1, lowL ? rL : rR);
    const float fmax = (pmax - pmin) * sqrtf(__fdividef(A, pmax + (float)s.gm1dgp1 * pmin)) + dv;
    /* the guess: a linear one for similar pressures, otherwise with powers or
     * square roots (ExactRiemannSolver.cpp:644-673) */
    const float ppv = 0.5f * (pL + pR) - 0.125f * dv * (rL + rR) * (aL + aR);
    const int linear = pmax <= 2.f * pmin && pmin <= ppv && ppv <= pmax;
    if(fmin >= 0.f) return 0 + linear;
    if(fmax <= 0.f) return 2 + linear;
    return (lowL ? 4 : 5);
}

template <int D, int MODE>
__global__ void __launch_bounds__(kExactBlock, 2)
        k_faces_exact(sfx_dmesh m, sfx_solver_params sp, double dt, int write_branch, int list) {
    constexpr int S = D + 2, NW = kExactBlock / 32;
    constexpr bool MOVING = MODE == kFaceMoving;
    __shared__ double sW[2 * S][kExactBlock], sn[D][kExactBlock];
    __shared__ double sv[MOVING ? D : 1][kExactBlock]; /* one unused row when static */
    __shared__ double sA[kExactBlock], sL[kExactBlock], sR[kExactBlock];
    __shared__ int sf[kExactBlock]; /* face, bit 31: no right cell */
    __shared__ int sbase[kKeys][NW];
    __shared__ int stotal;
    const int f = blockIdx.x * kExactBlock + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    FaceProblem<D> q;
    int key = kKeyNone;
    if(f < sfx_flux_faces(m) && !failed(m.err) &&
       face_problem<D, MODE>(m, sp, dt, f, write_branch, q))
        key = wave_key<D>(sp, q);
    if(!list && key == kKeyListed) key = kKeys - 2;
    /* the list: one atomic per warp; each face enters it at most once a step */
    const unsigned listed = __ballot_sync(0xffffffffu, key == kKeyListed);
    if(listed) {
        int at = 0;
        if(lane == 0) at = atomicAdd(m.listed_n, __popc(listed));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(listed & ((1u << lane) - 1u));
        if(key == kKeyListed) {
            if(at < m.n_faces)
                m.listed[at] = f;
            else
                report_face(m.err, f, SFX_ERR_INVALID);
        }
    }
    /* counting sort by key */
    unsigned mine = 0;
#pragma unroll
    for(int c = 0; c < kKeys; ++c) {
        const unsigned b = __ballot_sync(0xffffffffu, key == c);
        if(lane == c) sbase[c][warp] = __popc(b);
        if(key == c) mine = b;
    }
    __syncthreads();
    if(warp == 0) {
        /* exclusive scan in (key, warp) order, two entries per lane */
        static_assert(kKeys * NW == 64, "two counts per lane");
        int* t = &sbase[0][0];
        const int a = t[2 * lane], b = t[2 * lane + 1];
        int x = a + b;
#pragma unroll
        for(int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if(lane >= o) x += y;
        }
        t[2 * lane] = x - a - b;
        t[2 * lane + 1] = x - b;
        if(lane == 31) stotal = x;
    }
    __syncthreads();
    if(key < kKeys) {
        const int at = sbase[key][warp] + __popc(mine & ((1u << lane) - 1u));
#pragma unroll
        for(int k = 0; k < S; ++k) {
            sW[k][at] = q.WL[k];
            sW[S + k][at] = q.WR[k];
        }
#pragma unroll
        for(int l = 0; l < D; ++l) {
            sn[l][at] = q.n[l];
            if(MOVING) sv[MOVING ? l : 0][at] = q.v[l];
        }
        sA[at] = q.dtA;
        sL[at] = q.limL;
        sR[at] = q.limR;
        sf[at] = f | (q.has_right ? 0 : (int)kRightBit);
    }
    __syncthreads();
    const int t = threadIdx.x;
    if(t >= stotal) return;
    const bool has_right = sf[t] >= 0;
    double WL[S], WR[S], n[D], v[D], flux[S];
#pragma unroll
    for(int k = 0; k < S; ++k) {
        WL[k] = sW[k][t];
        WR[k] = sW[S + k][t];
    }
#pragma unroll
    for(int l = 0; l < D; ++l) {
        n[l] = sn[l][t];
        v[l] = MOVING ? sv[MOVING ? l : 0][t] : 0.;
    }
    const ExactOut eo = exact_face<D>(sp, WL, WR, n, v, has_right, flux);
    face_dQ<D, true>(m, (int)((unsigned)sf[t] & ~kRightBit), flux, sA[t], sL[t], sR[t], has_right,
                     eo.code, eo.status, write_branch);
}

/* The listed faces, one per thread; nothing to do when there are none.  A
 * failure of this step's other faces does not end it: the record names the
 * lowest failing face, and that one may be listed (after a failure of an
 * earlier step or phase the list is empty). */
constexpr int kListedBlock = 128, kListedBlocks = 4 * kSfxSMs;
/* one wave of blocks waits for its longest face whichever way it is sorted, and a
 * second launch would add to that: the list from two blocks on every SM */
constexpr int kListFrom = 2 * kSfxSMs * kExactBlock;

template <int D, int MODE>
__global__ void __launch_bounds__(kListedBlock)
        k_faces_listed(sfx_dmesh m, sfx_solver_params sp, double dt, int write_branch) {
    const int count = min(*(volatile const int*)m.listed_n, m.n_faces);
    for(int j = blockIdx.x * kListedBlock + threadIdx.x; j < count;
        j += kListedBlocks * kListedBlock) {
        const int f = m.listed[j];
        if(below(m.err, f)) continue;
        FaceProblem<D> q;
        if(!face_problem<D, MODE>(m, sp, dt, f, write_branch, q)) continue;
        double flux[D + 2];
        const ExactOut eo = exact_face<D>(sp, q.WL, q.WR, q.n, q.v, q.has_right, flux);
        face_dQ<D, true>(m, f, flux, q.dtA, q.limL, q.limR, q.has_right, eo.code, eo.status,
                         write_branch);
    }
}

/* ------------------------------ update ------------------------------ */

/* One thread per cell: the cell's faces in ascending face order (aidx), the
 * order in which the reference's face loop adds them (a face of zero area, or
 * between two inactive cells, holds zeros, which change no sum), then Q and
 * get_W.  Bound by the latency of the dQ gathers: a face's dQ is one record, a
 * 32-byte load in 2D and three of 16 bytes in 3D (field-major dQ touches a
 * 32-byte sector per double), U faces' loads in flight.  65,537 cells 3D 33 -> 23 us, 150,001
 * cells 2D 20.5 -> 19.1 us (event-timed); one lane per cell and variable took
 * 23 and 24 us. */
constexpr int kApplyBlock = 128;

template <int D, bool REC>
__global__ void __launch_bounds__(kApplyBlock) k_apply(sfx_dmesh m, double gamma) {
    using R = Rec<D>;
    constexpr int S = R::S;
    const int i = blockIdx.x * kApplyBlock + threadIdx.x;
    if(i >= sfx_update_cells(m) || failed(m.err)) return;
    const int n = m.n_cells;
    double dQ[S];
#pragma unroll
    for(int k = 0; k < S; ++k) dQ[k] = 0.;
    const int beg = m.off[i], end = m.off[i + 1];
    constexpr int U = 3; /* faces in flight */
    for(int j = beg; j < end; j += U) {
        unsigned e[U];
        double v[U][R::dq];
#pragma unroll
        for(int t = 0; t < U; ++t) e[t] = (unsigned)__ldg(m.aidx + (j + t < end ? j + t : j));
#pragma unroll
        for(int t = 0; t < U; ++t) {
            const size_t f = e[t] & ~kRightBit;
            if constexpr(REC) {
                load_record<R::dq>(m.dQf + f * R::dq, v[t]);
            } else {
#pragma unroll
                for(int k = 0; k < S; ++k) v[t][k] = __ldg(m.dQf + (size_t)k * m.n_faces + f);
            }
        }
#pragma unroll
        for(int t = 0; t < U; ++t)
            if(t == 0 || j + t < end) {
#pragma unroll
                for(int k = 0; k < S; ++k)
                    dQ[k] = dQ[k] + (e[t] & kRightBit ? -1. * v[t][k] : v[t][k]);
            }
    }
    double Q[S], W[S];
#pragma unroll
    for(int k = 0; k < S; ++k) Q[k] = m.Q[(size_t)k * n + i] - dQ[k];
    if(Q[0] < 0. || Q[D + 1] < 0.) {
        report_cell(m.err, i, SFX_ERR_NEG_STATE);
        return;
    }
    double* ws = REC ? m.ws + (size_t)i * R::ws : nullptr;
    if(m.local && m.tend[i] != m.t_next) {
        /* local time steps: a cell in the middle of its step takes the flux
         * of its active neighbours into Q; its W waits for the end of its
         * step (src/Simulation.cpp:791-836) */
#pragma unroll
        for(int k = 0; k < S; ++k) m.Q[(size_t)k * n + i] = Q[k];
        if(REC) ws[S] = Q[0];
        return;
    }
    /* get_W (ExactRiemannSolver.cpp:716-766 == HLLCRiemannSolver.cpp:495-535
     * on the hydro fields); may rewrite Q[D+1] (pressure floor) */
    const double V = m.vol[i];
#pragma unroll
    for(int k = 0; k < S; ++k) W[k] = 0.;
    if(Q[0] != 0.) {
        W[0] = Q[0] / V;
        W[1] = Q[1] / Q[0];
        W[2] = Q[2] / Q[0];
        double p2 = Q[1] * Q[1] + Q[2] * Q[2];
        if(D == 3) {
            W[D] = Q[D] / Q[0];
            p2 = p2 + Q[D] * Q[D];
        }
        W[D + 1] = (gamma - 1.) * (Q[D + 1] - 0.5 * p2 / Q[0]) / V;
        if(W[D + 1] < 1.e-30) {
            W[D + 1] = 1.e-30;
            Q[D + 1] = 0.5 * p2 / Q[0] + W[D + 1] * V / (gamma - 1.);
        }
        if(W[0] < 1.e-30) {
#pragma unroll
            for(int k = 0; k < S; ++k) W[k] = 0.;
        }
    }
    double t[8];
#pragma unroll
    for(int k = 0; k < 8; ++k) t[k] = 0.;
#pragma unroll
    for(int k = 0; k < S; ++k) {
        m.Q[(size_t)k * n + i] = Q[k];
        m.W[(size_t)k * n + i] = W[k];
        t[k] = W[k];
    }
    t[S] = Q[0];
    if(REC) store_record<8>(ws, t);
}

/* Host arrays are rows of one cell or face, device arrays field-major: the
 * transposes run here, on the copied rows, at memory speed.  On the host they,
 * and the temporaries they went through, took longer than the copies over the
 * bus: two 15 MB states out 8.0 -> 2.9 ms, one in 3.0 -> 1.1 ms. */
__global__ void __launch_bounds__(256) k_from_rows(const double* rows, int64_t n, int w,
                                                   double* out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    for(int k = 0; k < w; ++k) out[k * n + i] = rows[i * w + k];
}

__global__ void __launch_bounds__(256) k_to_rows(const double* in, int64_t n, int w,
                                                 double* rows) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    for(int k = 0; k < w; ++k) rows[i * w + k] = in[k * n + i];
}

/* rows [count][w] from (IN: to) an array with element (i, k) at a[i * rs + k * cs] */
template <bool IN>
__global__ void __launch_bounds__(256) k_strided_rows(double* a, int64_t rs, int64_t cs,
                                                      int64_t count, int w, double* rows) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(t >= count * w) return;
    const int64_t i = t / w, k = t - i * w;
    if(IN)
        a[i * rs + k * cs] = rows[t];
    else
        rows[t] = a[i * rs + k * cs];
}

/* Q = get_Q(V, W): ExactRiemannSolver.cpp:776-804 / HLLCRiemannSolver.cpp:471-483 */
template <int D>
__global__ void k_init_Q(sfx_dmesh m, double gamma, int kind, const double* rows) {
    constexpr int S = D + 2;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= m.n_cells) return;
    const int n = m.n_cells;
    double W[S], Q[S];
#pragma unroll
    for(int k = 0; k < S; ++k) W[k] = rows ? rows[(size_t)i * S + k] : m.W[(size_t)k * n + i];
    if(rows) {
#pragma unroll
        for(int k = 0; k < S; ++k) m.W[(size_t)k * n + i] = W[k];
    }
    const double V = m.vol[i];
    Q[0] = W[0] * V;
    Q[1] = Q[0] * W[1];
    Q[2] = Q[0] * W[2];
    double v2 = W[1] * W[1] + W[2] * W[2];
    if(D == 3) {
        Q[3] = Q[0] * W[3];
        v2 = v2 + W[3] * W[3];
    }
    if(kind == SFX_SOLVER_EXACT) {
        Q[D + 1] = (0.5 * W[0] * v2 + W[D + 1] / (gamma - 1.)) * V;
        if(Q[0] < 0. || Q[D + 1] < 0.) report_cell(m.err, i, SFX_ERR_NEG_STATE);
    } else {
        Q[D + 1] = V * W[D + 1] / (gamma - 1.) + 0.5 * Q[0] * v2;
    }
#pragma unroll
    for(int k = 0; k < S; ++k) m.Q[(size_t)k * n + i] = Q[k];
    if(m.ws) {
        double* w = m.ws + (size_t)i * Rec<D>::ws;
#pragma unroll
        for(int k = 0; k < S; ++k) w[k] = W[k];
        w[S] = Q[0];
    }
}

/* deterministic totals: fixed 1024 blocks over fixed ranges, fixed tree */
constexpr int kTotBlocks = 1024;
constexpr int kTotThreads = 256;

/* sum of field blockIdx.y over this block's cells of [0, count) of Q [S][n] */
__global__ void k_totals_partial(const double* Q, int n, int count, double* part) {
    __shared__ double sh[kTotThreads];
    const int per = (count + kTotBlocks - 1) / kTotBlocks;
    const int b0 = blockIdx.x * per;
    const int b1 = min(count, b0 + per);
    const int k = blockIdx.y;
    double acc = 0.;
    for(int i = b0 + threadIdx.x; i < b1; i += kTotThreads) acc = acc + Q[(size_t)k * n + i];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for(int w = kTotThreads / 2; w > 0; w >>= 1) {
        if(threadIdx.x < w) sh[threadIdx.x] = sh[threadIdx.x] + sh[threadIdx.x + w];
        __syncthreads();
    }
    if(threadIdx.x == 0) part[k * kTotBlocks + blockIdx.x] = sh[0];
}

/* one block per field */
__global__ void k_totals_final(double* part, int S, const sfx_dev_error* err) {
    __shared__ double sh[kTotBlocks];
    const int k = blockIdx.x;
    for(int t = threadIdx.x; t < kTotBlocks; t += blockDim.x) sh[t] = part[k * kTotBlocks + t];
    __syncthreads();
    for(int w = kTotBlocks / 2; w > 0; w >>= 1) {
        for(int t = threadIdx.x; t < w; t += blockDim.x) sh[t] = sh[t] + sh[t + w];
        __syncthreads();
    }
    if(threadIdx.x != 0) return;
    part[S * kTotBlocks + k] = sh[0];
    /* the error record beside them: one copy to the host for both */
    if(k == 0) {
        part[S * kTotBlocks + S] = __longlong_as_double((long long)err->face_key);
        part[S * kTotBlocks + S + 1] = __longlong_as_double((long long)err->cell_key);
    }
}

template <int D, int SOLVER>
__global__ void k_riemann(sfx_solver_params sp, int n, const double* WLa,
                          const double* WRa, const double* na, int reflective,
                          double* half, double* flux, int32_t* code) {
    constexpr int S = D + 2;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if(t >= n) return;
    double L[S], R[S], nn[D], v[D], fl[S];
#pragma unroll
    for(int l = 0; l < D; ++l) {
        nn[l] = na[(size_t)t * D + l];
        v[l] = 0.;
    }
    int c, st = SFX_OK;
    if(SOLVER == SFX_SOLVER_EXACT) {
#pragma unroll
        for(int k = 0; k < S; ++k) {
            L[k] = WLa[(size_t)t * S + k];
            R[k] = WRa[(size_t)t * S + k];
        }
        double h[S];
        ExactOut eo = exact_solve<D>(sp, L, R, nn, reflective != 0, h);
        if(half) {
#pragma unroll
            for(int k = 0; k < S; ++k) half[(size_t)t * S + k] = h[k];
        }
        st = eo.status;
        c = eo.code;
#pragma unroll
        for(int l = 0; l < D; ++l) h[1 + l] = h[1 + l] + v[l];
        exact_flux_from_half<D>(sp.gamma, h, v, nn, fl);
    } else {
#pragma unroll
        for(int k = 0; k < S; ++k) {
            L[k] = WLa[(size_t)t * S + k];
            R[k] = WRa[(size_t)t * S + k];
        }
        c = hllc_flux<D>(sp, L, R, nn, v, reflective != 0, fl);
    }
#pragma unroll
    for(int k = 0; k < S; ++k) flux[(size_t)t * S + k] = fl[k];
    code[t] = st ? -st : c;
}

/* halo records of a split mesh: [count][S + 1], the cell's W then its mass
 * Q[0] (the only Q field the face kernel reads of a cell it does not
 * update); an index outside the mesh is skipped, never dereferenced */
__global__ void k_pack_cells(sfx_dmesh m, const int32_t* idx, int count, double* out) {
    const int S = m.S, R = S + 1;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if(t >= (long long)count * R) return;
    const int j = (int)(t / R), q = (int)(t % R);
    const int c = idx[j];
    if(c < 0 || c >= m.n_cells) return;
    out[t] = q < S ? m.W[(size_t)q * m.n_cells + c] : m.Q[c];
}

__global__ void k_unpack_cells(sfx_dmesh m, const int32_t* idx, int count, const double* in) {
    const int S = m.S, R = S + 1;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if(t >= (long long)count * R) return;
    const int j = (int)(t / R), q = (int)(t % R);
    const int c = idx[j];
    if(c < 0 || c >= m.n_cells) return;
    if(q < S)
        m.W[(size_t)q * m.n_cells + c] = in[t];
    else
        m.Q[c] = in[t];
    if(m.ws) m.ws[(size_t)c * Rec<3>::ws + q] = in[t]; /* W, then the mass: the same stride in 2D */
}

inline int grid_for(long long n, int block) {
    return (int)((n + block - 1) / block);
}

inline int cuda_status(cudaError_t e) {
    return e == cudaSuccess ? SFX_OK : SFX_ERR_CUDA;
}

/* --------------------------- moving generators ---------------------------
 * One step of a moving mesh (a build of the reference without -DSTATIC):
 * every generator gets the velocity of VorCell::get_velocity
 * (src/VorCell.cpp:966-1008: the fluid velocity plus a term that steers the
 * generator towards its cell's centroid, at the sound speed when the offset
 * exceeds 1/4 of the cell radius, ramped in between; suppressed linearly
 * below density 1e-10), without the fluid velocity when a reflective unit
 * box would be left within dt (src/Simulation.cpp:366-398, RectangularBox::
 * inside); every face the velocity of VorFace::set_v
 * (src/VorFace.cpp:586-660: the mean of its generators' velocities plus the
 * part that keeps the face between them; a 3D mirror face does not move, a
 * 2D mirror generator moves as the mirror image of its cell's generator);
 * after the update the generators drift, x + dt v (Particle::drift,
 * src/utilities/Particle.cpp:281-283).  Same IEEE operations in the same
 * order as the reference, cube roots by sfx_cbrt. */
constexpr double kPi = 3.14159265358979323846;

template <int D>
__global__ void __launch_bounds__(128) k_gen_velocity(sfx_dmesh m, double gamma, double dt,
                                                      int periodic) {
    constexpr int S = D + 2;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= m.n_cells) return;
    /* local time steps: only the cells starting a step set their velocity
     * (the first kick of src/Simulation.cpp:366-398) */
    if(m.local && m.tstart[i] != m.t_now) return;
    const int n = m.n_cells;
    double W[S];
#pragma unroll
    for(int k = 0; k < S; ++k) W[k] = m.W[(size_t)k * n + i];
    double vel[D];
#pragma unroll
    for(int l = 0; l < D; ++l) vel[l] = 0.;
    if(W[0] != 0.) {
        double d[D];
#pragma unroll
        for(int l = 0; l < D; ++l) d[l] = m.cen[(size_t)l * n + i] - m.pos[(size_t)l * n + i];
        double Ri = m.vol[i];
        /* GasParticle::get_soundspeed: the solver's sqrt(gamma p / rho) */
        const double csnd = sqrt(gamma * W[D + 1] / W[0]);
        if(D == 3)
            Ri = sfx_cbrt(3. * Ri / 4. / kPi);
        else
            Ri = sqrt(Ri / kPi);
        const double dn = norm<D>(d);
        const double check = 4. * dn / Ri;
        if(check > 0.9) {
            double fac;
            if(check < 1.1)
                fac = csnd / dn * (dn - 0.9 * 0.25 * Ri) / (0.2 * 0.25 * Ri);
            else
                fac = csnd / dn;
#pragma unroll
            for(int l = 0; l < D; ++l) vel[l] = fac * d[l];
        }
    }
    double v[D];
#pragma unroll
    for(int l = 0; l < D; ++l) v[l] = W[1 + l] + vel[l];
    if(W[0] < 1.e-10) {
        const double fac = W[0] * 1.e10;
#pragma unroll
        for(int l = 0; l < D; ++l) v[l] = fac * v[l];
    }
    if(!periodic) {
        /* with local time steps, the cell's own step
         * (get_realtime_interval(end - start)) */
        const double dti = m.local ? sfx_realtime_interval(m.t_total, m.tend[i] - m.tstart[i]) : dt;
        bool inside = true;
#pragma unroll
        for(int l = 0; l < D; ++l) {
            const double nx = m.pos[(size_t)l * n + i] + dti * v[l];
            if(fabs(0.5 - nx) > 0.5) inside = false;
        }
        if(!inside) {
#pragma unroll
            for(int l = 0; l < D; ++l) v[l] -= W[1 + l];
        }
    }
#pragma unroll
    for(int l = 0; l < D; ++l) m.vgen[(size_t)l * n + i] = v[l];
}

template <int D>
__global__ void __launch_bounds__(128) k_face_velocity(sfx_dmesh m) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if(f >= m.n_faces) return;
    const int n = m.n_cells, F = m.n_faces;
    const int iL = m.left[f];
    const int kind = m.kind[f];
    double xl[D], xr[D], mid[D], vl[D], vr[D];
#pragma unroll
    for(int l = 0; l < D; ++l) {
        xl[l] = m.pos[(size_t)l * n + iL];
        xr[l] = m.rpos[(size_t)l * F + f];
        mid[l] = m.mid[(size_t)l * F + f];
        vl[l] = m.vgen[(size_t)l * n + iL];
    }
    if(kind != SFX_FACE_MIRROR) {
        const int iR = m.right[f];
#pragma unroll
        for(int l = 0; l < D; ++l) vr[l] = m.vgen[(size_t)l * n + iR];
    } else if(D == 3) {
#pragma unroll
        for(int l = 0; l < D; ++l) m.vel[(size_t)l * F + f] = 0.;
        return;
    } else {
        double Wd[4] = {0., vl[0], vl[1], 0.};
        mirror_state<2>(Wd, xl, xr);
        vr[0] = Wd[1];
        vr[1] = Wd[2];
    }
    double rRL[D];
#pragma unroll
    for(int l = 0; l < D; ++l) rRL[l] = xr[l] - xl[l];
    double r2 = rRL[0] * rRL[0] + rRL[1] * rRL[1];
    if(D == 3) r2 = r2 + rRL[2] * rRL[2];
    double fac = (vl[0] - vr[0]) * (mid[0] - 0.5 * (xl[0] + xr[0]));
#pragma unroll
    for(int l = 1; l < D; ++l) fac += (vl[l] - vr[l]) * (mid[l] - 0.5 * (xl[l] + xr[l]));
    fac /= r2;
#pragma unroll
    for(int l = 0; l < D; ++l) m.vel[(size_t)l * F + f] = 0.5 * (vl[l] + vr[l]) + fac * rRL[l];
}

template <int D>
__global__ void __launch_bounds__(128) k_drift(sfx_dmesh m, double dt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= m.n_cells) return;
    const int n = m.n_cells;
#pragma unroll
    for(int l = 0; l < D; ++l)
        m.newpos[(size_t)l * n + i] = m.pos[(size_t)l * n + i] + dt * m.vgen[(size_t)l * n + i];
}

/* ---------------------------- local time steps ----------------------------
 * TimeLine::calculate_timestep (src/TimeLine.cpp:233-317, the gas particles
 * of a run without gravity or a global step) for the cells whose step ends
 * at t_next: h = VorCell::get_h (src/VorCell.cpp:948-956), the CFL step
 * h / (|v - v_gen| + c) with the generator velocity set at the start of the
 * step, S = cfl x that; the step is max_step when max_step is shorter than
 * S, otherwise the largest power-of-two fraction of the timeline not longer
 * than S, halved until the timeline's end is a whole number of steps from
 * the cell's end (synchronisation), then clamped to [min_step, max_step].
 * The cell's next step is [end, end + step).  A zero step (the reference's
 * "Timestep 0!" exit) is SFX_ERR_TIMESTEP. */
template <int D>
__global__ void __launch_bounds__(128) k_timestep_bins(sfx_dmesh m, double gamma, double cfl,
                                                       unsigned long long max_step,
                                                       unsigned long long min_step,
                                                       unsigned long long* smin) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= m.n_cells) return;
    const uint64_t end = m.tend[i];
    if(end != m.t_next) return;
    const int n = m.n_cells;
    const double V = m.vol[i];
    const double h = D == 3 ? sfx_cbrt(V * 3. / 4. / kPi) : sqrt(V / kPi);
    const double rho = m.W[i], p = m.W[(size_t)(D + 1) * n + i];
    double v[D];
#pragma unroll
    for(int l = 0; l < D; ++l)
        v[l] = m.W[(size_t)(1 + l) * n + i] - (m.vgen ? m.vgen[(size_t)l * n + i] : 0.);
    double v2 = v[0] * v[0] + v[1] * v[1];
    if(D == 3) v2 = v2 + v[2] * v[2];
    const double vi = sqrt(v2);
    const double ci = rho != 0. ? sqrt(gamma * p / rho) : 0.;
    const double S = cfl * (h / (vi + ci));
    const uint64_t Smax = max_step;
    uint64_t S2;
    if(sfx_realtime_interval(m.t_total, Smax) < S) {
        S2 = Smax;
    } else {
        S2 = SFX_TIMELINE_TICKS;
        while(S2 && sfx_realtime_interval(m.t_total, S2) > S) S2 >>= 1;
        if(!S2) {
            report_cell(m.err, i, SFX_ERR_TIMESTEP);
            return;
        }
        while((SFX_TIMELINE_TICKS - end) % S2) S2 >>= 1;
        S2 = S2 > min_step ? S2 : min_step;
        S2 = S2 < Smax ? S2 : Smax;
    }
    m.tstart[i] = end;
    m.tend[i] = end + S2;
    atomicMin(smin, (unsigned long long)S2);
}

}  // namespace

int sfx_fp64_timestep_bins(const sfx_dmesh* m, double gamma, double cfl, uint64_t max_step,
                           uint64_t min_step, unsigned long long* d_smin, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    const int gc = (m->n_cells + 127) / 128;
    if(m->dim == 3)
        k_timestep_bins<3><<<gc, 128, 0, s>>>(*m, gamma, cfl, max_step, min_step, d_smin);
    else
        k_timestep_bins<2><<<gc, 128, 0, s>>>(*m, gamma, cfl, max_step, min_step, d_smin);
    sfx_count_launches(1);
    return cudaGetLastError() == cudaSuccess ? SFX_OK : SFX_ERR_CUDA;
}

int sfx_fp64_move_velocities(const sfx_dmesh* m, double gamma, double dt, int periodic,
                             int faces, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    const int gc = (m->n_cells + 127) / 128, gf = faces ? (m->n_faces + 127) / 128 : 0;
    if(m->dim == 3) {
        k_gen_velocity<3><<<gc, 128, 0, s>>>(*m, gamma, dt, periodic);
        if(gf) k_face_velocity<3><<<gf, 128, 0, s>>>(*m);
    } else {
        k_gen_velocity<2><<<gc, 128, 0, s>>>(*m, gamma, dt, periodic);
        if(gf) k_face_velocity<2><<<gf, 128, 0, s>>>(*m);
    }
    sfx_count_launches(gf ? 2 : 1);
    return cudaGetLastError() == cudaSuccess ? SFX_OK : SFX_ERR_CUDA;
}

int sfx_fp64_drift(const sfx_dmesh* m, double dt, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    const int gc = (m->n_cells + 127) / 128;
    if(m->dim == 3)
        k_drift<3><<<gc, 128, 0, s>>>(*m, dt);
    else
        k_drift<2><<<gc, 128, 0, s>>>(*m, dt);
    sfx_count_launches(1);
    return cudaGetLastError() == cudaSuccess ? SFX_OK : SFX_ERR_CUDA;
}

void sfx_solver_params_init(sfx_solver_params* p, int kind, double g, double tol,
                            double cutoff) {
    p->kind = kind;
    p->gamma = g;
    p->tol = tol;
    p->cutoff = cutoff;
    /* ExactRiemannSolver.cpp:48-64 */
    p->gp1d2g = 0.5 * (g + 1.) / g;
    p->gm1d2g = 0.5 * (g - 1.) / g;
    p->gm1dgp1 = (g - 1.) / (g + 1.);
    p->tdgp1 = 2. / (g + 1.);
    p->tdgm1 = 2. / (g - 1.);
    p->gm1d2 = 0.5 * (g - 1.);
    p->tgdgm1 = 2. * g / (g - 1.);
    p->ginv = 1. / g;
}

/* threads for `cells` cells of the kernels with one lane per cell and variable */
static int cell_lane_blocks(int dim, int cells, int block) {
    const int per_warp = dim == 3 ? Rec<3>::cells : Rec<2>::cells;
    return grid_for((cells + per_warp - 1) / per_warp * 32ll, block);
}

int sfx_fp64_record_bytes(int dim, int what) {
    const int v3[5] = {Rec<3>::ws, Rec<3>::grec, Rec<3>::dq, Rec<3>::ggeo, Rec<3>::fgeo};
    const int v2[5] = {Rec<2>::ws, Rec<2>::grec, Rec<2>::dq, Rec<2>::ggeo, Rec<2>::fgeo};
    return (int)sizeof(double) * (dim == 3 ? v3 : v2)[what];
}

int64_t sfx_fp64_list_room(int64_t n_faces) {
    return n_faces > kListFrom ? n_faces : 0;
}

int sfx_from_rows(const double* rows, int64_t n, int w, double* out, void* stream) {
    if(n == 0) return SFX_OK;
    k_from_rows<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(rows, n, w, out);
    sfx_count_launches(1);
    return cuda_status(cudaGetLastError());
}

int sfx_to_rows(const double* in, int64_t n, int w, double* rows, void* stream) {
    if(n == 0) return SFX_OK;
    k_to_rows<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(in, n, w, rows);
    sfx_count_launches(1);
    return cuda_status(cudaGetLastError());
}

int sfx_strided_rows(double* a, int64_t rs, int64_t cs, int64_t count, int w, double* rows, int in,
                     void* stream) {
    if(count == 0) return SFX_OK;
    const int G = grid_for(count * w, 256);
    if(in)
        k_strided_rows<true><<<G, 256, 0, (cudaStream_t)stream>>>(a, rs, cs, count, w, rows);
    else
        k_strided_rows<false><<<G, 256, 0, (cudaStream_t)stream>>>(a, rs, cs, count, w, rows);
    sfx_count_launches(1);
    return cuda_status(cudaGetLastError());
}

int sfx_fp64_csr_neighbours(const sfx_dmesh* m, void* stream) {
    if(m->nnz == 0) return SFX_OK;
    k_csr_neighbours<<<grid_for(m->nnz, 256), 256, 0, (cudaStream_t)stream>>>(*m);
    sfx_count_launches(1);
    return cuda_status(cudaGetLastError());
}

int sfx_fp64_face_records(const sfx_dmesh* m, void* stream) {
    if(m->n_faces == 0) return SFX_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if(m->dim == 3)
        k_face_records<3><<<grid_for(m->n_faces, 128), 128, 0, s>>>(*m);
    else
        k_face_records<2><<<grid_for(m->n_faces, 128), 128, 0, s>>>(*m);
    sfx_count_launches(1);
    return cuda_status(cudaGetLastError());
}

int sfx_fp64_load_rows(const sfx_dmesh* m, const double* W, const double* Q, void* stream) {
    if(m->n_cells == 0) return SFX_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if(m->dim == 3)
        k_load_rows<3><<<grid_for(m->n_cells, 128), 128, 0, s>>>(*m, W, Q);
    else
        k_load_rows<2><<<grid_for(m->n_cells, 128), 128, 0, s>>>(*m, W, Q);
    sfx_count_launches(1);
    return cuda_status(cudaGetLastError());
}

/* k_grad_cells needs the records and face positions that are the cells' (see
 * there); other meshes take k_gradients, caller-owned arrays and meshes whose
 * records did not fit its field-major form */
template <int D>
static void launch_gradients(const sfx_dmesh* m, double gamma, int nc, cudaStream_t s) {
    const int B = 128;
    if(m->ws && m->gshare)
        k_grad_cells<D><<<cell_lane_blocks(D, nc, kGradBlock), kGradBlock, 0,
                          s>>>(*m, gamma);
    else if(m->ws)
        k_gradients<D, true><<<grid_for(nc, B), B, 0, s>>>(*m, gamma);
    else
        k_gradients<D, false><<<grid_for(nc, B), B, 0, s>>>(*m, gamma);
}

int sfx_fp64_gradients(const sfx_dmesh* m, const sfx_solver_params* sp, void* stream) {
    const int nc = sfx_grad_cells(*m);
    if(nc == 0) {
        /* no gradient launch to empty the face list (a part without cells) */
        if(!m->listed_n) return SFX_OK;
        return cuda_status(
                cudaMemsetAsync(m->listed_n, 0, sizeof(int32_t), (cudaStream_t)stream));
    }
    if(m->dim == 3)
        launch_gradients<3>(m, sp->gamma, nc, (cudaStream_t)stream);
    else
        launch_gradients<2>(m, sp->gamma, nc, (cudaStream_t)stream);
    sfx_count_launches(1);
    return cuda_status(cudaGetLastError());
}

template <int D, int MODE>
static int launch_faces(const sfx_dmesh* m, const sfx_solver_params* sp, double dt,
                        int write_branch, int nf, cudaStream_t s) {
    const int B = 128, G = grid_for(nf, B);
    if(sp->kind != SFX_SOLVER_EXACT) {
        k_faces<D, SFX_SOLVER_HLLC, MODE><<<G, B, 0, s>>>(*m, *sp, dt, write_branch);
        return 1;
    }
    if constexpr(MODE == kFaceArrays) {
        k_faces<D, SFX_SOLVER_EXACT, MODE><<<G, B, 0, s>>>(*m, *sp, dt, write_branch);
        return 1;
    } else {
        const int list = nf > kListFrom;
        k_faces_exact<D, MODE><<<grid_for(nf, kExactBlock), kExactBlock, 0, s>>>(
                *m, *sp, dt, write_branch, list);
        if(!list) return 1;
        k_faces_listed<D, MODE>
                <<<kListedBlocks, kListedBlock, 0, s>>>(*m, *sp, dt, write_branch);
        return 2;
    }
}

template <int D>
static int launch_faces(const sfx_dmesh* m, const sfx_solver_params* sp, double dt,
                        int write_branch, int nf, cudaStream_t s) {
    if(!m->ws) return launch_faces<D, kFaceArrays>(m, sp, dt, write_branch, nf, s);
    if(m->vel || m->local) return launch_faces<D, kFaceMoving>(m, sp, dt, write_branch, nf, s);
    return launch_faces<D, kFaceRecords>(m, sp, dt, write_branch, nf, s);
}

int sfx_fp64_faces(const sfx_dmesh* m, const sfx_solver_params* sp, double dt,
                   int write_branch, void* stream) {
    const int nf = sfx_flux_faces(*m);
    if(nf == 0) return SFX_OK;
    cudaStream_t s = (cudaStream_t)stream;
    sfx_count_launches(m->dim == 3 ? launch_faces<3>(m, sp, dt, write_branch, nf, s)
                                   : launch_faces<2>(m, sp, dt, write_branch, nf, s));
    return cuda_status(cudaGetLastError());
}

int sfx_fp64_apply(const sfx_dmesh* m, const sfx_solver_params* sp, void* stream) {
    const int nc = sfx_update_cells(*m);
    if(nc == 0) return SFX_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const int B = kApplyBlock, G = grid_for(nc, B);
    if(m->dim == 3 && m->ws)
        k_apply<3, true><<<G, B, 0, s>>>(*m, sp->gamma);
    else if(m->dim == 3)
        k_apply<3, false><<<G, B, 0, s>>>(*m, sp->gamma);
    else if(m->ws)
        k_apply<2, true><<<G, B, 0, s>>>(*m, sp->gamma);
    else
        k_apply<2, false><<<G, B, 0, s>>>(*m, sp->gamma);
    sfx_count_launches(1);
    return cuda_status(cudaGetLastError());
}

int sfx_fp64_init_Q(const sfx_dmesh* m, const sfx_solver_params* sp, const double* rows,
                    void* stream) {
    if(m->n_cells == 0) return SFX_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const int B = 128;
    if(m->dim == 3)
        k_init_Q<3><<<grid_for(m->n_cells, B), B, 0, s>>>(*m, sp->gamma, sp->kind, rows);
    else
        k_init_Q<2><<<grid_for(m->n_cells, B), B, 0, s>>>(*m, sp->gamma, sp->kind, rows);
    sfx_count_launches(1);
    return cuda_status(cudaGetLastError());
}

int sfx_fp64_totals(const sfx_dmesh* m, double* host_out, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    const dim3 grid(kTotBlocks, m->S);
    k_totals_partial<<<grid, kTotThreads, 0, s>>>(m->Q, m->n_cells, sfx_update_cells(*m),
                                                  m->totals_scratch);
    k_totals_final<<<m->S, 256, 0, s>>>(m->totals_scratch, m->S, m->err);
    sfx_count_launches(2);
    cudaError_t e = cudaMemcpyAsync(host_out, m->totals_scratch + (size_t)m->S * kTotBlocks,
                                    sizeof(double) * (m->S + 2), cudaMemcpyDeviceToHost, s);
    if(e != cudaSuccess) return SFX_ERR_CUDA;
    return cuda_status(cudaStreamSynchronize(s));
}

int sfx_fp64_riemann(int dim, const sfx_solver_params* sp, int n, const double* dWL,
                     const double* dWR, const double* dn, int reflective, double* dhalf,
                     double* dflux, int32_t* dcode, void* stream) {
    if(n == 0) return SFX_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const int B = 128, G = grid_for(n, B);
    if(dim == 3) {
        if(sp->kind == SFX_SOLVER_EXACT)
            k_riemann<3, SFX_SOLVER_EXACT><<<G, B, 0, s>>>(*sp, n, dWL, dWR, dn, reflective,
                                                          dhalf, dflux, dcode);
        else
            k_riemann<3, SFX_SOLVER_HLLC><<<G, B, 0, s>>>(*sp, n, dWL, dWR, dn, reflective,
                                                         dhalf, dflux, dcode);
    } else {
        if(sp->kind == SFX_SOLVER_EXACT)
            k_riemann<2, SFX_SOLVER_EXACT><<<G, B, 0, s>>>(*sp, n, dWL, dWR, dn, reflective,
                                                          dhalf, dflux, dcode);
        else
            k_riemann<2, SFX_SOLVER_HLLC><<<G, B, 0, s>>>(*sp, n, dWL, dWR, dn, reflective,
                                                         dhalf, dflux, dcode);
    }
    sfx_count_launches(1);
    return cuda_status(cudaGetLastError());
}

int sfx_fp64_pack_cells(const sfx_dmesh* m, const int32_t* idx, int count, double* out,
                        void* stream) {
    if(count <= 0) return SFX_OK;
    const long long t = (long long)count * (m->S + 1);
    k_pack_cells<<<grid_for(t, 256), 256, 0, (cudaStream_t)stream>>>(*m, idx, count, out);
    sfx_count_launches(1);
    return cuda_status(cudaGetLastError());
}

int sfx_fp64_unpack_cells(const sfx_dmesh* m, const int32_t* idx, int count, const double* in,
                          void* stream) {
    if(count <= 0) return SFX_OK;
    const long long t = (long long)count * (m->S + 1);
    k_unpack_cells<<<grid_for(t, 256), 256, 0, (cudaStream_t)stream>>>(*m, idx, count, in);
    sfx_count_launches(1);
    return cuda_status(cudaGetLastError());
}
