// cg_stokes_kernels.cuh — device code of the VE Stokes PT kernels shared by the per-kernel
// entry points (cg_stokes.cu) and the defect-correction solver (cg_stokes_dc.cu).
#pragma once

#include <cmath>

#include "cg_common.cuh"

namespace cgk {


template <class T>
struct SV {  // device views of the Stokes field set
    DF<T> V[3], rV[3], P, divV, tau[6], tau_old[6], eta, ieta, rho[3], Tt, To, qT[3];
    // continuity forcing of the defect-correction solve: the pressure update and the divV
    // output use (divV + fP); the deviatoric strain rate uses divV alone
    DF<T> fP;
    int has_rV, has_divV, has_eta, has_ieta, has_rho[3], has_fP;
    // 1/eta at a cell: the precomputed field when given, else an IEEE division (same bits)
    __device__ __forceinline__ T inv_eta(int i, int j, int k) const {
        return has_ieta ? ieta(i, j, k) : T(1) / eta(i, j, k);
    }
};

template <class T>
struct SP {  // scalars in the field precision
    T eta, eta_ve, G, dt, dtau_Pr, dtau_r, nu_dtau, lam;
    T inv_Gdt, third;
    T idx[3];
};

// Body force per velocity component as a device FunctionField, and the grid's coordinates. A
// separate kernel argument of the two kernels that evaluate it (the velocity update and the
// FP64 defect): the march kernels keep the small SP as their scalar argument.
template <class T>
struct BodyFn {
    FnDev<T> fn[3];
    T org[3], dx[3];
};

// Body-force function of velocity component `comp` at its point (i, j, k): Vertex along comp,
// Center along the other dimensions.
template <class T>
__device__ __forceinline__ T body_fn(const BodyFn<T>& s, int comp, int nd, int i, int j, int k) {
    const int I[3] = {i, j, k};
    T x[3] = {T(0), T(0), T(0)};
    for (int e = 0; e < nd; ++e) x[e] = grid_coord(s.org[e], s.dx[e], I[e], e == comp);
    return fn_eval(s.fn[comp], nd, x);
}

template <class T>
SV<T> views(const cg_stokes_fields* f, int nd) {
    SV<T> v;
    std::memset(&v, 0, sizeof(v));
    const int nt = nd == 2 ? 3 : 6;
    for (int d = 0; d < nd; ++d) {
        v.V[d] = cg_view<T>(f->V[d]);
        if (cg_present(f->r_V[d])) v.rV[d] = cg_view<T>(f->r_V[d]);
        if (cg_present(f->rho_g[d])) {
            v.rho[d] = cg_view<T>(f->rho_g[d]);
            v.has_rho[d] = 1;
        }
        if (cg_present(f->qT[d])) v.qT[d] = cg_view<T>(f->qT[d]);
    }
    v.has_rV = cg_present(f->r_V[0]);
    for (int c = 0; c < nt; ++c) {
        v.tau[c] = cg_view<T>(f->tau[c]);
        if (cg_present(f->tau_old[c])) v.tau_old[c] = cg_view<T>(f->tau_old[c]);
    }
    v.P = cg_view<T>(f->P);
    if (cg_present(f->divV)) {
        v.divV = cg_view<T>(f->divV);
        v.has_divV = 1;
    }
    if (cg_present(f->eta)) {
        v.eta = cg_view<T>(f->eta);
        v.has_eta = 1;
    }
    if (cg_present(f->inv_eta)) {
        v.ieta = cg_view<T>(f->inv_eta);
        v.has_ieta = 1;
        v.has_eta = 1;
    }
    if (cg_present(f->T)) v.Tt = cg_view<T>(f->T);
    if (cg_present(f->T_old)) v.To = cg_view<T>(f->T_old);
    return v;
}

template <class T>
SP<T> scalars(const cg_grid* g, const cg_stokes_params* p) {
    SP<T> s;
    s.eta = (T)p->eta;
    s.eta_ve = (T)p->eta_ve;
    s.G = (T)p->G;
    s.dt = (T)p->dt;
    s.dtau_Pr = (T)p->dtau_Pr;
    s.dtau_r = (T)p->dtau_r;
    s.nu_dtau = (T)p->nu_dtau;
    s.lam = (T)p->lambda_rhoCp;
    s.inv_Gdt = T(1) / (s.G * s.dt);
    s.third = T(1) / T(3);
    for (int d = 0; d < 3; ++d) s.idx[d] = (T)g->inv_spacing[d];
    return s;
}

template <class T>
BodyFn<T> body_fns(const cg_grid* g, const cg_stokes_params* p) {
    BodyFn<T> b;
    for (int d = 0; d < 3; ++d) {
        b.org[d] = (T)g->origin[d];
        b.dx[d] = (T)g->spacing[d];
        b.fn[d].kind = p->rho_g_fn[d].kind;
        for (int q = 0; q < 8; ++q) b.fn[d].p[q] = (T)p->rho_g_fn[d].p[q];
    }
    return b;
}

// The divisors of the scalar-viscosity form.
template <class T>
struct ScalarDiv {
    ConstDiv<T> Gdt, eta, eve, three;
};
template <class T>
inline ScalarDiv<T> scalar_divs(const SP<T>& s) {
    return {const_div<T>(s.G * s.dt), const_div<T>(s.eta), const_div<T>(s.eta_ve), const_div<T>(T(3))};
}

template <class T>
__device__ __forceinline__ T eta_ve_of(T eta, T G, T dt) {
    return T(1.0) / (T(1.0) / eta + T(1.0) / (G * dt));
}

// 2D/3D launch: x, y threads over [0, n+1]; z over blockIdx.z.
template <int ND>
inline dim3 range_grid(const cg_grid* g, dim3 block) {
    return point_grid<ND>(g->n, block);
}

// 1/eta on the (a, b) shear edge of point I: the Linear rule over the 4 cells around it, dim a
// innermost (interpolation.jl:217-221), i.e. the harmonic average of eta.
template <class T>
__device__ __forceinline__ T shear_inv_eta(const SV<T>& v, int i, int j, int k, int a, int b) {
    const int ai = a == 0, aj = a == 1, ak = a == 2;
    const int bi = b == 0, bj = b == 1, bk = b == 2;
    const T e00 = v.inv_eta(i - ai - bi, j - aj - bj, k - ak - bk);
    const T e10 = v.inv_eta(i - bi, j - bj, k - bk);
    const T e01 = v.inv_eta(i - ai, j - aj, k - ak);
    const T e11 = v.inv_eta(i, j, k);
    const T lo = fma(T(0.5), e10 - e00, e00);
    const T hi = fma(T(0.5), e11 - e01, e01);
    return fma(T(0.5), hi - lo, lo);
}

// Operand readers of the stress and velocity kernels. NoMask reads a value; FieldMaskW is
// Chmy's FieldMask (src/GridOperators/field_mask.jl:1-117) seen by the masked operators
// (src/GridOperators/masked_operators.jl:11-39): every operand of a derivative is multiplied by
// the mask at its own location and index. `loc` is the operand's location bits (bit d set for
// Vertex along d), the index into the mask's weight fields. With unit weights both readers give
// the same bits (x * 1 == x, also under contraction into a fused multiply-add).
template <class T>
struct NoMask {
    __device__ __forceinline__ T operator()(int, const DF<T>& f, int i, int j, int k) const { return f(i, j, k); }
};
template <class T>
struct FieldMaskW {
    DF<T> w[8];
    __device__ __forceinline__ T operator()(int loc, const DF<T>& f, int i, int j, int k) const {
        return f(i, j, k) * w[loc](i, j, k);
    }
};

// update_stress! at one point. Tensor order 2D (xx, yy, xy), 3D (xx, yy, zz, xy, xz, yz).
// M reads the operands of the strain-rate derivatives (NoMask, or FieldMaskW for the masked
// operators ∂(V.d, ω, g, I) and divg(V, ω, g, I)); V.d sits at location bits 1 << d.
template <class T, int ND, bool WRITE_RES, class M>
__device__ __forceinline__ void stress_point(const SV<T>& v, const SP<T>& s, const ScalarDiv<T>& sd, int i, int j, int k, const M& m) {
    const DF<T>& Vx = v.V[0];
    const DF<T>& Vy = v.V[1];
    // ∂x(V.x) at Center: V.x is Vertex in x -> V.x[i+1] - V.x[i]
    const T exx = (m(1, Vx, i + 1, j, k) - m(1, Vx, i, j, k)) * s.idx[0];
    const T eyy = (m(2, Vy, i, j + 1, k) - m(2, Vy, i, j, k)) * s.idx[1];
    T dv = exx + eyy;
    T ezz = T(0);
    if (ND > 2) {
        const DF<T>& Vz = v.V[2];
        ezz = (m(4, Vz, i, j, k + 1) - m(4, Vz, i, j, k)) * s.idx[2];
        dv = dv + ezz;
    }
    const T dvP = v.has_fP ? dv + v.fP(i, j, k) : dv;
    if (WRITE_RES && v.has_divV) v.divV(i, j, k) = dvP;
    T ieta_c = T(0), eve_c = s.eta_ve;
    if (v.has_eta) {
        ieta_c = v.inv_eta(i, j, k);
        eve_c = T(1) / (ieta_c + s.inv_Gdt);
    }
    v.P(i, j, k) = v.P(i, j, k) - dvP * eve_c * s.dtau_Pr;
    auto diag = [&](int c, T edd) {
        const T t = v.tau[c](i, j, k), to = v.tau_old[c](i, j, k);
        T r;
        if (v.has_eta)
            r = -(t - to) * s.inv_Gdt - t * ieta_c + T(2.0) * (edd - dv * s.third);
        else  // examples/stokes_2d_inc_ve_T.jl:28-29, literally
            r = divide(-(t - to), sd.Gdt) - divide(t, sd.eta) + T(2.0) * (edd - divide(dv, sd.three));
        v.tau[c](i, j, k) = t + r * eve_c * s.dtau_r;
    };
    // shear component on the (a, b) edge: 1/eta interpolated with the Linear rule over the 4
    // cells around it, dim a innermost (interpolation.jl:217-221) = harmonic mean of eta
    auto shear = [&](int c, T eod, int a, int b) {
        const T t = v.tau[c](i, j, k), to = v.tau_old[c](i, j, k);
        if (v.has_eta) {
            const T iev = shear_inv_eta(v, i, j, k, a, b);
            const T eve = T(1) / (iev + s.inv_Gdt);
            const T r = -(t - to) * s.inv_Gdt - t * iev + T(2.0) * eod;
            v.tau[c](i, j, k) = t + r * eve * s.dtau_r;
        } else {  // examples/stokes_2d_inc_ve_T.jl:30
            const T r = divide(-(t - to), sd.Gdt) - divide(t, sd.eta) + T(2.0) * eod;
            v.tau[c](i, j, k) = t + r * s.eta_ve * s.dtau_r;
        }
    };
    // ∂y(V.x) at the xy vertex: V.x is Center in y -> V.x[j] - V.x[j-1]
    const T exy = T(0.5) * ((m(1, Vx, i, j, k) - m(1, Vx, i, j - 1, k)) * s.idx[1] +
                            (m(2, Vy, i, j, k) - m(2, Vy, i - 1, j, k)) * s.idx[0]);
    if (ND == 2) {
        diag(0, exx);
        diag(1, eyy);
        shear(2, exy, 0, 1);
    } else {
        const DF<T>& Vz = v.V[2];
        const T exz = T(0.5) * ((m(1, Vx, i, j, k) - m(1, Vx, i, j, k - 1)) * s.idx[2] +
                                (m(4, Vz, i, j, k) - m(4, Vz, i - 1, j, k)) * s.idx[0]);
        const T eyz = T(0.5) * ((m(2, Vy, i, j, k) - m(2, Vy, i, j, k - 1)) * s.idx[2] +
                                (m(4, Vz, i, j, k) - m(4, Vz, i, j - 1, k)) * s.idx[1]);
        diag(0, exx);
        diag(1, eyy);
        diag(2, ezz);
        shear(3, exy, 0, 1);
        shear(4, exz, 0, 2);
        shear(5, eyz, 1, 2);
    }
}

template <class T, int ND, bool WRITE_RES, class M, bool FLAT>
__global__ void stress_kernel(const SV<T> v, const SP<T> s, const ScalarDiv<T> sd, int e0, int e1, const M m) {
    cg_dep_wait();
    cg_dep_release();
    int i, j, k;
    if (!launch_point<ND, FLAT>(e0, e1, i, j, k)) return;
    stress_point<T, ND, WRITE_RES>(v, s, sd, i, j, k, m);
}

// update_velocity! at one point. M reads the operands of the pressure and stress derivatives
// (P and τ_dd at location bits 0, τ_xy 3, τ_xz 5, τ_yz 6).
template <class T, int ND, bool WRITE_RES, class M, bool FLAT>
__global__ void velocity_kernel(const SV<T> v, const SP<T> s, const ScalarDiv<T> sd, const BodyFn<T> bf, int e0, int e1, const M m) {
    cg_dep_wait();
    cg_dep_release();
    int i, j, k;
    if (!launch_point<ND, FLAT>(e0, e1, i, j, k)) return;
    const DF<T>& P = v.P;
    // tensor components: 2D xx=0 yy=1 xy=2; 3D xx=0 yy=1 zz=2 xy=3 xz=4 yz=5
    const int XY = ND == 2 ? 2 : 3;
    const DF<T>& txx = v.tau[0];
    const DF<T>& tyy = v.tau[1];
    const DF<T>& txy = v.tau[XY];
    // P, τ_dd are Center: at a face along d, left = I - e_d, right = I.
    // τ_xy is Vertex in x and y: ∂y(τxy) at a V.x face (Vertex x, Center y) -> τxy[j+1] - τxy[j].
    const int LXY = 3, LXZ = 5, LYZ = 6;  // location bits of the shear components
    T rx = -((m(0, P, i, j, k) - m(0, P, i - 1, j, k)) * s.idx[0]) + (m(0, txx, i, j, k) - m(0, txx, i - 1, j, k)) * s.idx[0];
    rx = rx + (m(LXY, txy, i, j + 1, k) - m(LXY, txy, i, j, k)) * s.idx[1];
    T ry = -((m(0, P, i, j, k) - m(0, P, i, j - 1, k)) * s.idx[1]) + (m(0, tyy, i, j, k) - m(0, tyy, i, j - 1, k)) * s.idx[1];
    ry = ry + (m(LXY, txy, i + 1, j, k) - m(LXY, txy, i, j, k)) * s.idx[0];
    T rz = T(0);
    if (ND > 2) {
        const DF<T>& tzz = v.tau[2];
        const DF<T>& txz = v.tau[4];
        const DF<T>& tyz = v.tau[5];
        rx = rx + (m(LXZ, txz, i, j, k + 1) - m(LXZ, txz, i, j, k)) * s.idx[2];
        ry = ry + (m(LYZ, tyz, i, j, k + 1) - m(LYZ, tyz, i, j, k)) * s.idx[2];
        rz = -((m(0, P, i, j, k) - m(0, P, i, j, k - 1)) * s.idx[2]) + (m(0, tzz, i, j, k) - m(0, tzz, i, j, k - 1)) * s.idx[2];
        rz = rz + (m(LXZ, txz, i + 1, j, k) - m(LXZ, txz, i, j, k)) * s.idx[0];
        rz = rz + (m(LYZ, tyz, i, j + 1, k) - m(LYZ, tyz, i, j, k)) * s.idx[1];
    }
    if (v.has_rho[0]) rx = rx - v.rho[0](i, j, k);
    else if (bf.fn[0].kind) rx = rx - body_fn(bf, 0, ND, i, j, k);
    if (v.has_rho[1]) ry = ry - v.rho[1](i, j, k);
    else if (bf.fn[1].kind) ry = ry - body_fn(bf, 1, ND, i, j, k);
    if (ND > 2 && v.has_rho[2]) rz = rz - v.rho[2](i, j, k);
    else if (ND > 2 && bf.fn[2].kind) rz = rz - body_fn(bf, 2, ND, i, j, k);
    if (WRITE_RES && v.has_rV) {
        v.rV[0](i, j, k) = rx;
        v.rV[1](i, j, k) = ry;
        if (ND > 2) v.rV[2](i, j, k) = rz;
    }
    if (v.has_eta) {
        // nu_dtau / max(eta_ve) of the two cells beside the face, without a division
        const T c = v.inv_eta(i, j, k);
        v.V[0](i, j, k) = v.V[0](i, j, k) + rx * (s.nu_dtau * (fmin(v.inv_eta(i - 1, j, k), c) + s.inv_Gdt));
        v.V[1](i, j, k) = v.V[1](i, j, k) + ry * (s.nu_dtau * (fmin(v.inv_eta(i, j - 1, k), c) + s.inv_Gdt));
        if (ND > 2)
            v.V[2](i, j, k) = v.V[2](i, j, k) + rz * (s.nu_dtau * (fmin(v.inv_eta(i, j, k - 1), c) + s.inv_Gdt));
    } else {  // examples/stokes_2d_inc_ve_T.jl:41-42
        v.V[0](i, j, k) = v.V[0](i, j, k) + divide(rx * s.nu_dtau, sd.eve);
        v.V[1](i, j, k) = v.V[1](i, j, k) + divide(ry * s.nu_dtau, sd.eve);
        if (ND > 2) v.V[2](i, j, k) = v.V[2](i, j, k) + divide(rz * s.nu_dtau, sd.eve);
    }
}

// ---- the two kernels of a loop of FP64 PT iterations with variable viscosity ------------------
//
// A loop calls update_stress! and update_velocity! many times with the same viscosity, G, dt and
// PT parameters. FP64 arithmetic bounds both kernels on GB300 (two FP64 instructions per clock and
// SM; stress_kernel kept that pipe 84 % busy at 0.41 of the HBM time), so the loop's kernels issue
// as few of them as the update allows:
// - what depends on the viscosity alone is computed once per loop (coef_kernel), the 1/eta
//   interpolation and the reciprocals among it: eta_ve dtau_Pr and eta_ve dtau_r at cells, the
//   interpolated 1/eta and its eta_ve dtau_r at every shear component, and nu_dtau / eta_ve at the
//   faces;
// - strain rates are kept doubled (2 idx is exact), which removes the products by 2 and 1/2;
// - the stress residual keeps its form (t_old - t)/(G dt) - t/eta + 2 e, evaluated with fused
//   multiply-adds, and tau += r (eta_ve dtau_r) is one more: the iteration's fixed point is where
//   the residual itself vanishes, exactly as in stress_kernel.
// Per 2D cell that leaves 24 + 14 FP64 instructions of 58 + 20 (3D: 48 + 27 of 122 + 36).
// Measured against a loop of stress_kernel and velocity_kernel: 2D 511^2 stress 29.3 -> 15.2 us,
// velocity 13.3 -> 10.8 us; 3D 95 x 80 x 112 stress 244 -> 84 us, velocity 90 -> 53 us.
// With one scalar viscosity the loop keeps stress_kernel and velocity_kernel, whose divisions by
// scalars are ConstDiv: coupled to the thermal step, whose fixed-point iteration can amplify a last
// bit of V from one iteration to the next, the loop has to leave the same bits as the kernels apart.
template <class T>
struct PtCoef {
    DF<T> ieta, cP, cT, ievE[3], cE[3], step[3];
    T g;  // 1 / (G dt)
    T third, idx[3], idx2[3];
};

// The viscosity terms over [0, n+1]^N. cP carries a factor 1/2 for the doubled divergence.
template <class T, int ND, bool FLAT>
__global__ void coef_kernel(const SV<T> v, const SP<T> s, const PtCoef<T> c, int e0, int e1) {
    int i, j, k;
    if (!launch_point<ND, FLAT>(e0, e1, i, j, k)) return;
    const T ie = v.inv_eta(i, j, k);
    const T eve = T(1) / (ie + s.inv_Gdt);
    c.cP(i, j, k) = T(0.5) * (eve * s.dtau_Pr);
    c.cT(i, j, k) = eve * s.dtau_r;
    const int pairs[3][2] = {{0, 1}, {0, 2}, {1, 2}};
    for (int e = 0; e < (ND == 2 ? 1 : 3); ++e) {
        const T iev = shear_inv_eta(v, i, j, k, pairs[e][0], pairs[e][1]);
        c.ievE[e](i, j, k) = iev;
        c.cE[e](i, j, k) = T(1) / (iev + s.inv_Gdt) * s.dtau_r;
    }
    for (int d = 0; d < ND; ++d)
        c.step[d](i, j, k) = s.nu_dtau * (fmin(v.inv_eta(i - (d == 0), j - (d == 1), k - (d == 2)), ie) + s.inv_Gdt);
}

// update_stress! of a PT loop at one point.
template <class T, int ND, bool WRITE_RES, class M>
__device__ __forceinline__ void stress_loop_point(const SV<T>& v, const PtCoef<T>& c, int i, int j, int k, const M& m) {
    const DF<T>& Vx = v.V[0];
    const DF<T>& Vy = v.V[1];
    const DF<T>& Vz = v.V[2];
    const T vx = m(1, Vx, i, j, k), vy = m(2, Vy, i, j, k), vz = ND > 2 ? m(4, Vz, i, j, k) : T(0);
    // doubled strain rates and divergence
    const T exx = (m(1, Vx, i + 1, j, k) - vx) * c.idx2[0];
    const T eyy = (m(2, Vy, i, j + 1, k) - vy) * c.idx2[1];
    T dv = exx + eyy, ezz = T(0);
    if (ND > 2) {
        ezz = (m(4, Vz, i, j, k + 1) - vz) * c.idx2[2];
        dv = dv + ezz;
    }
    if (WRITE_RES && v.has_divV) v.divV(i, j, k) = T(0.5) * dv;
    v.P(i, j, k) = fma(-dv, c.cP(i, j, k), v.P(i, j, k));
    auto update = [&](int q, T e2, T ie, T ct) {  // e2 = 2 e
        const T t = v.tau[q](i, j, k), to = v.tau_old[q](i, j, k);
        const T r = fma(to - t, c.g, fma(-t, ie, e2));
        v.tau[q](i, j, k) = fma(r, ct, t);
    };
    const T ie = c.ieta(i, j, k), ct = c.cT(i, j, k);
    update(0, fma(-dv, c.third, exx), ie, ct);
    update(1, fma(-dv, c.third, eyy), ie, ct);
    if (ND > 2) update(2, fma(-dv, c.third, ezz), ie, ct);
    auto shear = [&](int q, int e, T e2) { update(q, e2, c.ievE[e](i, j, k), c.cE[e](i, j, k)); };
    shear(ND == 2 ? 2 : 3, 0, fma(vx - m(1, Vx, i, j - 1, k), c.idx[1], (vy - m(2, Vy, i - 1, j, k)) * c.idx[0]));
    if (ND > 2) {
        shear(4, 1, fma(vx - m(1, Vx, i, j, k - 1), c.idx[2], (vz - m(4, Vz, i - 1, j, k)) * c.idx[0]));
        shear(5, 2, fma(vy - m(2, Vy, i, j, k - 1), c.idx[2], (vz - m(4, Vz, i, j - 1, k)) * c.idx[1]));
    }
}

template <class T, int ND, bool WRITE_RES, class M, bool FLAT>
__global__ void stress_loop_kernel(const SV<T> v, const PtCoef<T> c, int e0, int e1, const M m) {
    cg_dep_wait();
    cg_dep_release();
    int i, j, k;
    if (!launch_point<ND, FLAT>(e0, e1, i, j, k)) return;
    stress_loop_point<T, ND, WRITE_RES>(v, c, i, j, k, m);
}

// update_velocity! of a PT loop at one point. The differences of tau_dd and of P are formed
// separately (each is small against its operands) and share one product by idx.
template <class T, int ND, bool WRITE_RES, class M, bool FLAT>
__global__ void velocity_loop_kernel(const SV<T> v, const PtCoef<T> c, const BodyFn<T> bf, int e0, int e1, const M m) {
    cg_dep_wait();
    cg_dep_release();
    int i, j, k;
    if (!launch_point<ND, FLAT>(e0, e1, i, j, k)) return;
    constexpr int XY = ND == 2 ? 2 : 3, XZ = 4, YZ = 5;
    const int LXY = 3, LXZ = 5, LYZ = 6;  // location bits of the shear components
    const T p = m(0, v.P, i, j, k);
    auto normal = [&](int d) {  // d(tau_dd) - d(P) along d
        const int l = i - (d == 0), r = j - (d == 1), q = k - (d == 2);
        return ((m(0, v.tau[d], i, j, k) - m(0, v.tau[d], l, r, q)) - (p - m(0, v.P, l, r, q))) * c.idx[d];
    };
    auto finish = [&](int d, T r) {
        if (v.has_rho[d]) r = r - v.rho[d](i, j, k);
        else if (bf.fn[d].kind) r = r - body_fn(bf, d, ND, i, j, k);
        if (WRITE_RES && v.has_rV) v.rV[d](i, j, k) = r;
        v.V[d](i, j, k) = fma(r, c.step[d](i, j, k), v.V[d](i, j, k));
    };
    const T xy = m(LXY, v.tau[XY], i, j, k);
    T rx = fma(m(LXY, v.tau[XY], i, j + 1, k) - xy, c.idx[1], normal(0));
    T ry = fma(m(LXY, v.tau[XY], i + 1, j, k) - xy, c.idx[0], normal(1));
    if (ND > 2) {
        const T xz = m(LXZ, v.tau[XZ], i, j, k), yz = m(LYZ, v.tau[YZ], i, j, k);
        rx = fma(m(LXZ, v.tau[XZ], i, j, k + 1) - xz, c.idx[2], rx);
        ry = fma(m(LYZ, v.tau[YZ], i, j, k + 1) - yz, c.idx[2], ry);
        T rz = fma(m(LXZ, v.tau[XZ], i + 1, j, k) - xz, c.idx[0], normal(2));
        rz = fma(m(LYZ, v.tau[YZ], i, j + 1, k) - yz, c.idx[1], rz);
        finish(2, rz);
    }
    finish(0, rx);
    finish(1, ry);
}

template <class T, int ND>
__global__ void update_old_kernel(const SV<T> v, int has_T, int e0, int e1) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = ND > 2 ? blockIdx.z : 0;
    if (i > e0 || j > e1) return;
    if (has_T) v.To(i, j, k) = v.Tt(i, j, k);
#pragma unroll
    for (int c = 0; c < (ND == 2 ? 3 : 6); ++c) v.tau_old[c](i, j, k) = v.tau[c](i, j, k);
}

template <class T, int ND>
__global__ void thermal_flux_kernel(const SV<T> v, const SP<T> s, int e0, int e1) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = ND > 2 ? blockIdx.z : 0;
    if (i > e0 || j > e1) return;
    const DF<T>& Tt = v.Tt;
    const T c = Tt(i, j, k);
    const T mlam = -s.lam;
    {
        const T l = Tt(i - 1, j, k), vv = v.V[0](i, j, k);
        v.qT[0](i, j, k) = mlam * ((c - l) * s.idx[0]) + fmax(vv, T(0.0)) * l + fmin(vv, T(0.0)) * c;
    }
    {
        const T l = Tt(i, j - 1, k), vv = v.V[1](i, j, k);
        v.qT[1](i, j, k) = mlam * ((c - l) * s.idx[1]) + fmax(vv, T(0.0)) * l + fmin(vv, T(0.0)) * c;
    }
    if (ND > 2) {
        const T l = Tt(i, j, k - 1), vv = v.V[2](i, j, k);
        v.qT[2](i, j, k) = mlam * ((c - l) * s.idx[2]) + fmax(vv, T(0.0)) * l + fmin(vv, T(0.0)) * c;
    }
}

template <class T, int ND>
__global__ void thermal_kernel(const SV<T> v, const SP<T> s, int e0, int e1) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = ND > 2 ? blockIdx.z : 0;
    if (i > e0 || j > e1) return;
    T dv = (v.qT[0](i + 1, j, k) - v.qT[0](i, j, k)) * s.idx[0];
    dv = dv + (v.qT[1](i, j + 1, k) - v.qT[1](i, j, k)) * s.idx[1];
    if (ND > 2) dv = dv + (v.qT[2](i, j, k + 1) - v.qT[2](i, j, k)) * s.idx[2];
    v.Tt(i, j, k) = v.To(i, j, k) - s.dt * dv;
}

// ---- fused thermal step: update_thermal_flux! + update_thermal! ------------------------------
//
// T_out = T_old - dt * divg(qT) with qT_d = -lambda * d_d(T) + max(V_d, 0) * T_left +
// min(V_d, 0) * T_right (examples/stokes_2d_inc_ve_T.jl:35-50, 3D :59-77) computed on the fly
// at the two faces of each cell, over Chmy's launch range. A face flux at index n+2 lies beyond
// the flux kernel's launch range, so in the two-kernel form it reads the untouched allocation:
// zero here. Every operation is rounded once in the oracle's order (max/min as std::max/min).
//
// FP64 arithmetic bounds it: 7 instructions per face and 7 per cell. Blocks own 31 columns and each
// x face is computed once (lane 31 only supplies lane 30's), y faces pass through shared memory, and
// the signs of V are read from its bits: about 22 FP64 instructions per 2D cell for 43.
// Measured at 254^2: 7.7 -> 4.8 us per launch.
__device__ __forceinline__ bool is_neg(double v) {  // v < 0
    const unsigned long long b = bits_of(v);
    return b > 0x8000000000000000ull && b <= 0xFFF0000000000000ull;
}
__device__ __forceinline__ bool is_pos(double v) { return bits_of(v) - 1ull < 0x7FF0000000000000ull; }  // v > 0
__device__ __forceinline__ bool is_neg(float v) { return v < 0.f; }
__device__ __forceinline__ bool is_pos(float v) { return 0.f < v; }

template <class T>
__device__ __forceinline__ T heat_flux(T mlam, T tl, T tr, T v, T idx) {
    const T vp = is_neg(v) ? T(0) : v;  // std::max(v, 0)
    const T vm = is_pos(v) ? T(0) : v;  // std::min(v, 0)
    return radd(radd(rmul(mlam, rmul(rsub(tr, tl), idx)), rmul(vp, tl)), rmul(vm, tr));
}

template <class T>
struct ThermalStep {
    DF<T> Tin, Told, Tout, V[3];
    T mlam, dt, idx[3];
};

constexpr int kThermalCols = 31;

// Tile (bx, by) of plane k, by a block of 32 x ROWS.
template <class T, int ND, int ROWS>
__device__ __forceinline__ void thermal_tile(const ThermalStep<T>& a, int bx, int by, int k, int e0, int e1, int e2) {
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ T qy[ROWS + 1][32];
    const int lane = threadIdx.x, row = threadIdx.y;
    const int i = bx * kThermalCols + lane, j = by * ROWS + row;
    const bool in = i <= e0 && j <= e1;
    T c = T(0), qx0 = T(0), qy0 = T(0);
    if (in) {
        c = a.Tin(i, j, k);
        qx0 = heat_flux(a.mlam, a.Tin(i - 1, j, k), c, a.V[0](i, j, k), a.idx[0]);
        qy0 = heat_flux(a.mlam, a.Tin(i, j - 1, k), c, a.V[1](i, j, k), a.idx[1]);
    }
    qy[row][lane] = qy0;
    if (row == ROWS - 1) qy[ROWS][lane] = in && j + 1 <= e1 ? heat_flux(a.mlam, c, a.Tin(i, j + 1, k), a.V[1](i, j + 1, k), a.idx[1]) : T(0);
    const T qx1 = __shfl_down_sync(FULL, qx0, 1);  // 0 beyond the launch range
    __syncthreads();
    if (!in || lane == kThermalCols) return;
    T dq = rmul(rsub(qx1, qx0), a.idx[0]);
    dq = radd(dq, rmul(rsub(qy[row + 1][lane], qy0), a.idx[1]));
    if (ND > 2) {
        const T qz0 = heat_flux(a.mlam, a.Tin(i, j, k - 1), c, a.V[2](i, j, k), a.idx[2]);
        const T qz1 = k + 1 <= e2 ? heat_flux(a.mlam, c, a.Tin(i, j, k + 1), a.V[2](i, j, k + 1), a.idx[2]) : T(0);
        dq = radd(dq, rmul(rsub(qz1, qz0), a.idx[2]));
    }
    a.Tout(i, j, k) = rsub(a.Told(i, j, k), rmul(a.dt, dq));
}

template <class T, int ND>
__global__ void __launch_bounds__(256) thermal_step_kernel(const ThermalStep<T> a, int e0, int e1, int e2) {
    cg_dep_wait();
    cg_dep_release();
    thermal_tile<T, ND, 8>(a, blockIdx.x, blockIdx.y, ND > 2 ? blockIdx.z : 0, e0, e1, e2);
}

// The thermal step of one PT iteration and update_stress! of the next in one 2D launch: both read V as
// bc!(V) left it and neither reads what the other writes. The first ns blocks take the
// stress (points in order, as launch_point), the others (tx across) the thermal tiles. LOOP: the stress from a loop's coefficients.
//
// A thermal iteration on a small grid is a chain of launches, each with its own latency and with SMs idle
// in its last wave. With this launch, and bc!(T) beside the next bc!(V), a chain of five becomes one of
// three. Blocks of 4 rows: the FP64 work is per SM, and at 254^2 blocks of 8 rows put 4 on some SMs
// where 3.7 is the mean. Measured per iteration, apart -> paired (FP64 scalar viscosity): 62 x 80 16.2
// -> 10.3 us, 254^2 25.0 -> 21.2 (8 rows 23; 2 rows 20.4, but FP32 511^2 12.3 -> 15.5), 700 x 610 96.4
// -> 91.9; FP32 254^2 11.9 -> 8.3.
constexpr int kPairRows = 4;

template <class T, bool LOOP, bool WRITE_RES>
__global__ void __launch_bounds__(32 * kPairRows)
    stress_thermal_kernel(const SV<T> v, const SP<T> s, const ScalarDiv<T> sd, const PtCoef<T> c, const ThermalStep<T> a, int e0,
                          int e1, int ns, int tx) {
    cg_dep_wait();
    cg_dep_release();
    const int b = blockIdx.x;
    if (b >= ns) {
        thermal_tile<T, 2, kPairRows>(a, (b - ns) % tx, (b - ns) / tx, 0, e0, e1, 0);
        return;
    }
    const unsigned q = (unsigned)b * (32 * kPairRows) + threadIdx.y * 32 + threadIdx.x, w = (unsigned)e0 + 1u;
    const int j = (int)(q / w), i = (int)(q - (unsigned)j * w);
    if (j > e1) return;
    if constexpr (LOOP) stress_loop_point<T, 2, WRITE_RES>(v, c, i, j, 0, NoMask<T>{});
    else stress_point<T, 2, WRITE_RES>(v, s, sd, i, j, 0, NoMask<T>{});
}

// ---- bc!(V) folded into the velocity reads of the marching kernels -------------------------
//
// A PT iteration ends with bc!(V) (examples/stokes_2d_inc_ve_T.jl:81-89): its boundary planes
// are functions of the interior the iteration just wrote. The marching kernel can instead read
// the unpatched velocity of the previous iteration and apply the same rules to each value it
// uses, which leaves one boundary-condition launch at the end of a run of iterations instead
// of one per iteration. The rules are those of cg_bc_apply for Dirichlet and Neumann kinds
// (Chmy's FirstOrderBC): per velocity component a, dimension d and side s, the planes g (an
// index along d) become a constant (Dirichlet on a Vertex dimension), 2 v - F[src]
// (Dirichlet on a Center dimension) or F[src] -/+ h v (Neumann), applied over the tangential
// range 0..n+2, dimension y (then z in 3D) before x, side 0 before side 1, with the same
// fused multiply-adds, so the folded value equals the patched one bit for bit. Periodic
// kinds are not folded. A value the later phase reads (a corner) is the earlier phase's
// result, exactly as in the chain the boundary-condition kernel walks.
enum { FOLD_NONE = 0, FOLD_CONST = 1, FOLD_DIRC = 2, FOLD_NEU = 3 };

template <class T>
struct VFold {
    int on;
    signed char rule[3][3][2];  // [component][dimension][side]
    int g[3][3][2], src[3][3][2];
    T val[3][3][2];             // Dirichlet value; Neumann: -v on side 0, +v on side 1
    T h[3];
    int lim[3];                 // tangential range 0..n+2 of each dimension
};

template <class T>
__device__ __forceinline__ T fold_rule(int r, T base, T v, T h) {
    return r == FOLD_DIRC ? rfma(T(2), rsub(v, base), base) : rfma(h, v, base);
}

// The rules of cg_bc_apply for velocity component a (Vertex along a, Center along the others)
// of a grid with n[d] cells. Returns false when a kind cannot be folded (periodic).
template <class T>
inline bool make_vfold(const cg_grid* g, const cg_bc* bc_V, VFold<T>* out) {
    std::memset(out, 0, sizeof(*out));
    if (!bc_V) return false;
    const int nd = g->ndim;
    for (int d = 0; d < nd; ++d) {
        out->h[d] = (T)g->spacing[d];
        out->lim[d] = g->n[d] + 2;
    }
    for (int a = 0; a < nd; ++a)
        for (int d = 0; d < nd; ++d) {
            const bool vtx = d == a;
            const int ext = vtx ? g->n[d] + 1 : g->n[d];
            for (int s = 0; s < 2; ++s) {
                if (bc_V[a].values[d][s]) return false;  // per-point values: not folded
                const T v = (T)bc_V[a].value[d][s];
                signed char& r = out->rule[a][d][s];
                switch (bc_V[a].kind[d][s]) {
                    case CG_BC_NONE: r = FOLD_NONE; break;
                    case CG_BC_DIRICHLET:
                        if (vtx) {
                            r = FOLD_CONST;
                            out->g[a][d][s] = s ? ext : 1;
                        } else {
                            r = FOLD_DIRC;
                            out->g[a][d][s] = s ? ext + 1 : 0;
                            out->src[a][d][s] = s ? ext : 1;
                        }
                        out->val[a][d][s] = v;
                        break;
                    case CG_BC_NEUMANN:
                        r = FOLD_NEU;
                        out->g[a][d][s] = s ? ext + 1 : 0;
                        out->src[a][d][s] = s ? ext : 1;
                        out->val[a][d][s] = s ? v : -v;
                        break;
                    default: return false;
                }
            }
        }
    out->on = 1;
    return true;
}

// ---- fused 2D PT iteration (variable viscosity): update_stress! + update_velocity! -----------
//
// One launch per PT iteration, reading the `in` buffers and writing the `out` buffers
// (ping-pong). Points outside Chmy's launch range [0, n+1] keep their old values, exactly as in
// the two-kernel form.
template <class T>
struct Fused2D {
    DF<T> Vx_in, Vy_in, Vx_out, Vy_out;
    DF<T> txx_in, tyy_in, txy_in, txx_out, tyy_out, txy_out, P_in, P_out;
    DF<T> txx_o, tyy_o, txy_o, ieta, fP, rhox, rhoy, divV, rVx, rVy;
    int has_fP, has_rho;
    VFold<T> bc;  // bc.on: the V_in values are read through bc!(V)
};

// ---- warp-marching fused 2D PT iteration --------------------------------------------------
//
// update_stress! followed by update_velocity! in one launch, without shared memory. It writes
// the new P, tau_xx, tau_yy, tau_xy and V on [0, n+1]^2 (and divV, r_V when asked); points
// outside that range keep the values the out buffers hold. A warp owns 30
// launch columns i = c0 .. c0+29 and a segment of rows js .. je. Lane l holds column
// c0 - 1 + l, so lanes 0 and 31 are one-column halos. Each lane reads every input of its
// column once per row; x-neighbours come from shuffles. The warp then marches up the rows,
// keeping in registers the previous row's velocity, 1/eta and the new P, tau_yy and tau_xy.
// Iteration j computes the new cell row j and vertex row j+1, then the velocity of row j.
// The segment's prologue computes cell row js-1 and vertex row js.
//
// Shuffle validity: a cell at lane l needs Vx of lane l+1, so lane 31's cell is invalid; a
// vertex at lane l needs Vy and 1/eta of lane l-1, so lane 0's vertex is invalid. The owned
// lanes 1..30 read cells of lanes l-1, l and vertices of lanes l, l+1, all valid.
// Ix is the element-offset type: int where every offset fits in 32 bits, else long.
// LAY says how the arrays' strides are related. kLayOwn: each array has its own; kLayOne: all
// share one (the defect-correction pool); kLayLoc: arrays at one location share theirs, which is
// Chmy's dense layout and every layout that pads fields of one location alike. In 2D the location
// class is 0 for Center along x (P, tau_dd, 1/eta, V.y) and 1 for Vertex along x (V.x, tau_xy). A
// lane keeps one offset per class; with own strides each access takes its own multiplication and
// the kernel 114 registers, 4 blocks per SM instead of 8. Measured at 2047 x 1535 FP32 in
// the dense layout: 51.0 us per iteration with own strides, 39.9 us with class strides.
constexpr int kLayOwn = 0, kLayOne = 1, kLayLoc = 2;
struct MStr2 {
    long s1[2];
};
template <class T, class Ix, int LAY>
struct MAt {  // column i of a lane
    int i;
    Ix s1[2];
    __device__ __forceinline__ MAt(int i_, const MStr2& m) : i(i_), s1{(Ix)m.s1[0], (Ix)m.s1[LAY == kLayLoc ? 1 : 0]} {}
    // c: the array's location class
    __device__ __forceinline__ Ix off(int c, const DF<T>& f, int j) const {
        return (Ix)i + (Ix)j * (LAY == kLayOwn ? (Ix)f.s1 : s1[LAY == kLayLoc ? c : 0]);
    }
    // ld: an array that the launch before writes (V, P, tau); ldc: one that no launch of the chain
    // writes. A dependent launch is resident while the one before it still writes, and a
    // non-coherent load is only defined where the data does not change during the kernel.
    __device__ __forceinline__ T ld(int c, const DF<T>& f, int j, bool ok) const { return ok ? f.p[off(c, f, j)] : T(0); }
    __device__ __forceinline__ T ldc(int c, const DF<T>& f, int j, bool ok) const {
        return ok ? __ldg(f.p + off(c, f, j)) : T(0);
    }
    __device__ __forceinline__ void st(int c, const DF<T>& f, int j, T v) const { f.p[off(c, f, j)] = v; }
};

// Inputs of one marching step at column i: row j+1 of the vertex-row inputs, row j of the
// cell-row inputs.
template <class T>
struct MarchRow {
    T Vx, Vy, ie, txy, txyo;                   // row j+1
    T P, txx, tyy, txo, tyo, fp, rhox, rhoy;  // row j
};

template <class T, class Ix, int LAY>
__device__ __forceinline__ MarchRow<T> march_load(const Fused2D<T>& f, const MAt<T, Ix, LAY>& at, int j, int e1,
                                                  bool inV, bool inC) {
    MarchRow<T> r;
    const int jn = j + 1;
    const bool vn = inV && jn <= e1 + 1;
    r.Vx = at.ld(1, f.Vx_in, jn, vn);
    r.Vy = at.ld(0, f.Vy_in, jn, vn);
    r.ie = at.ldc(0, f.ieta, jn, vn);
    r.txy = at.ld(1, f.txy_in, jn, vn);
    r.txyo = at.ldc(1, f.txy_o, jn, inC && jn <= e1);
    const bool c = inC && j <= e1;
    r.P = at.ld(0, f.P_in, j, c);
    r.txx = at.ld(0, f.txx_in, j, c);
    r.tyy = at.ld(0, f.tyy_in, j, c);
    r.txo = at.ldc(0, f.txx_o, j, c);
    r.tyo = at.ldc(0, f.tyy_o, j, c);
    r.fp = f.has_fP ? at.ldc(0, f.fP, j, c) : T(0);
    r.rhox = f.has_rho ? at.ldc(1, f.rhox, j, c) : T(0);
    r.rhoy = f.has_rho ? at.ldc(0, f.rhoy, j, c) : T(0);
    return r;
}

// Velocity component a at column i, row j of a marching warp, read through bc!(V), in two
// steps. fold_y (rows; the caller tests that row j can hold a y-plane, uniformly in the warp):
// v is the stored value, vprev the folded value of row j-1 and vnext the stored value of row
// j+1. A y-plane's source row is always the adjacent one (row 0 from row 1, row n+1 from n,
// row n+2 from n+1; rows 1 and n+1 of a Vertex dimension are constants) and never a y-plane
// itself. The previous row's folded value equals its stored one except in an x-plane column,
// where fold_x overrides the y result anyway.
template <class T>
__device__ __forceinline__ T fold_y(const VFold<T>& b, int a, int i, int j, T v, T vprev, T vnext) {
    if (i >= 0 && i <= b.lim[0]) {
        const int r0 = b.rule[a][1][0], r1 = b.rule[a][1][1];
        if (r0 != FOLD_NONE && j == b.g[a][1][0])
            v = r0 == FOLD_CONST ? b.val[a][1][0] : fold_rule(r0, vnext, b.val[a][1][0], b.h[1]);
        if (r1 != FOLD_NONE && j == b.g[a][1][1])
            v = r1 == FOLD_CONST ? b.val[a][1][1] : fold_rule(r1, vprev, b.val[a][1][1], b.h[1]);
    }
    return v;
}

// fold_x (columns; called by the whole warp when its strip holds an x-plane, for a row in the
// tangential range 0..n+2): an x-plane takes its neighbour lane's y-folded value. Lanes 0 and
// 31 are halos: a left plane (column 0 or 1) sits at lane >= 1 with its source one lane up, a
// right plane (column n+1 or n+2) at lane >= 1 of any strip that owns a column, its source one
// lane down.
template <class T>
__device__ __forceinline__ T fold_x(const VFold<T>& b, int a, int i, T v) {
    constexpr unsigned FULL = 0xffffffffu;
    const int r0 = b.rule[a][0][0], r1 = b.rule[a][0][1];
    T vr = v, vl = v;
    if (r0 > FOLD_CONST || r1 > FOLD_CONST) {  // a rule with a source: the neighbours' values
        vr = __shfl_down_sync(FULL, v, 1);
        vl = __shfl_up_sync(FULL, v, 1);
    }
    if (r0 != FOLD_NONE && i == b.g[a][0][0])
        v = r0 == FOLD_CONST ? b.val[a][0][0] : fold_rule(r0, vr, b.val[a][0][0], b.h[0]);
    if (r1 != FOLD_NONE && i == b.g[a][0][1])
        v = r1 == FOLD_CONST ? b.val[a][0][1] : fold_rule(r1, vl, b.val[a][0][1], b.h[0]);
    return v;
}

// -(t - t_old) * inv_Gdt - t * ieta + 2 * e: the VE stress residual, left to right.
template <class T>
__device__ __forceinline__ T stress_res(const SP<T>& s, T t, T to, T ie, T e) {
    return radd(rsub(rmul(-rsub(t, to), s.inv_Gdt), rmul(t, ie)), rmul(T(2.0), e));
}

template <class T>
struct CellNew {
    T P, txx, tyy, dvP;
};

// New P, tau_xx, tau_yy at cell (i, j) from Vx(i, j), Vx(i+1, j), Vy(i, j), Vy(i, j+1) and the
// cell's inputs (update_stress!, variable-viscosity form).
template <class T>
__device__ __forceinline__ CellNew<T> march_cell(const SP<T>& s, bool has_fP, T vx, T vxR, T vy, T vyU, T ie, T P,
                                                 T txx, T txo, T tyy, T tyo, T fp) {
    const T exx = rmul(rsub(vxR, vx), s.idx[0]);
    const T eyy = rmul(rsub(vyU, vy), s.idx[1]);
    const T dv = radd(exx, eyy);
    const T dvt = rmul(dv, s.third);
    const T eve = rrcp(radd(ie, s.inv_Gdt));
    CellNew<T> c;
    c.dvP = has_fP ? radd(dv, fp) : dv;
    c.P = rsub(P, rmul(rmul(c.dvP, eve), s.dtau_Pr));
    c.txx = radd(txx, rmul(rmul(stress_res(s, txx, txo, ie, rsub(exx, dvt)), eve), s.dtau_r));
    c.tyy = radd(tyy, rmul(rmul(stress_res(s, tyy, tyo, ie, rsub(eyy, dvt)), eve), s.dtau_r));
    return c;
}

// New tau_xy at vertex (i, jv) from Vx(i, jv-1), Vx(i, jv), Vy(i-1, jv), Vy(i, jv) and the four
// cells' 1/eta around it (e00 = (i-1, jv-1), e10 = (i, jv-1), e01 = (i-1, jv), e11 = (i, jv)),
// interpolated with the Linear rule, x innermost.
template <class T>
__device__ __forceinline__ T march_vertex(const SP<T>& s, T vx0, T vx1, T vyl, T vy, T e00, T e10, T e01, T e11,
                                          T t2, T o2) {
    const T half = T(0.5);
    const T exy = rmul(half, radd(rmul(rsub(vx1, vx0), s.idx[1]), rmul(rsub(vy, vyl), s.idx[0])));
    const T lo = rfma(half, rsub(e10, e00), e00);
    const T hi = rfma(half, rsub(e11, e01), e01);
    const T iev = rfma(half, rsub(hi, lo), lo);
    const T eve = rrcp(radd(iev, s.inv_Gdt));
    return radd(t2, rmul(rmul(stress_res(s, t2, o2, iev, exy), eve), s.dtau_r));
}

template <class T, class Ix, int LAY, bool WRITE_RES, int MINB = 1>
__global__ void __launch_bounds__(128, MINB) march2d_kernel(const Fused2D<T> f, const SP<T> s, int e0, int e1,
                                                            int nstrip, int nwarps, int seg_rows, const MStr2 str) {
    constexpr unsigned FULL = 0xffffffffu;
    cg_dep_wait();
    cg_dep_release();
    const int lane = threadIdx.x & 31;
    const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (gw >= nwarps) return;  // whole warp
    const int strip = gw % nstrip;
    const int js = (gw / nstrip) * seg_rows;
    if (js > e1) return;  // whole warp
    const int je = min(js + seg_rows - 1, e1);
    const int i = strip * 30 - 1 + lane;
    const MAt<T, Ix, LAY> at(i, str);
    const bool own = lane >= 1 && lane <= 30 && i <= e0;
    const bool inV = i <= e0 + 1;  // V, 1/eta, tau_xy readable
    const bool inC = i <= e0;      // cell inputs, tau_xy_old readable
    const bool oldcell = i < 0;    // column -1 keeps its old cell values
    // bc!(V) folded into the reads: the strip holds an x-plane (columns 0, 1, n+1, n+2) / the
    // rows js-1 .. je+1 hold a y-plane (rows 0, 1, n+1, n+2)
    const bool xb = f.bc.on && (strip == 0 || strip * 30 + 30 >= e0);
    const bool ylow = js <= 2, yhigh = je + 2 >= e1;
    const bool yb = f.bc.on && (ylow || yhigh);
    // rows ylo..yhi of the marching steps can hold a y-plane (0..1, n+1..n+2, or all)
    const int ylo = ylow ? 0 : e1, yhi = yhigh ? e1 + 1 : 1;

    // ---- prologue: new cell row js-1 (P and tau_yy only) and new vertex row js ----
    T Vx_c, Vy_c, ie_c, ieL_c, ie_p, Pn_p, Tyyn_p, txy_c;
    MarchRow<T> cur;
    {
        const int jp = js - 1;  // >= -1
        T vxp = at.ld(1, f.Vx_in, jp, inV);
        T vyp = at.ld(0, f.Vy_in, jp, inV);
        const T iep = at.ldc(0, f.ieta, jp, inV);
        const T pp = at.ld(0, f.P_in, jp, inC);
        const T typ = at.ld(0, f.tyy_in, jp, inC);
        const T tyop = at.ldc(0, f.tyy_o, jp, inC);
        const T fpp = f.has_fP ? at.ldc(0, f.fP, jp, inC) : T(0);
        Vx_c = at.ld(1, f.Vx_in, js, inV);
        Vy_c = at.ld(0, f.Vy_in, js, inV);
        ie_c = at.ldc(0, f.ieta, js, inV);
        const T t2 = at.ld(1, f.txy_in, js, inV);
        const T o2 = at.ldc(1, f.txy_o, js, inC);
        // the first marching step's loads (row js+1) are issued before the prologue computes
        cur = march_load(f, at, js, e1, inV, inC);
        if (yb) {
            // row js+1 is the source of a plane at row js = 0; row js-1 can be no side-1 plane
            vxp = fold_y(f.bc, 0, i, jp, vxp, T(0), Vx_c);
            vyp = fold_y(f.bc, 1, i, jp, vyp, T(0), Vy_c);
        }
        if (xb && jp >= 0) {
            vxp = fold_x(f.bc, 0, i, vxp);
            vyp = fold_x(f.bc, 1, i, vyp);
        }
        if (yb) {
            Vx_c = fold_y(f.bc, 0, i, js, Vx_c, vxp, cur.Vx);
            Vy_c = fold_y(f.bc, 1, i, js, Vy_c, vyp, cur.Vy);
        }
        if (xb) {
            Vx_c = fold_x(f.bc, 0, i, Vx_c);
            Vy_c = fold_x(f.bc, 1, i, Vy_c);
        }
        // cell (i, js-1); row -1 and column -1 keep their old values
        const T vxpR = __shfl_down_sync(FULL, vxp, 1);
        const CellNew<T> cp = march_cell(s, f.has_fP != 0, vxp, vxpR, vyp, Vy_c, iep, pp, T(0), T(0), typ, tyop, fpp);
        const bool keep = jp < 0 || oldcell;
        Pn_p = keep ? pp : cp.P;
        Tyyn_p = keep ? typ : cp.tyy;
        // vertex (i, js)
        const T vyL = __shfl_up_sync(FULL, Vy_c, 1);
        const T iepL = __shfl_up_sync(FULL, iep, 1);
        ieL_c = __shfl_up_sync(FULL, ie_c, 1);
        txy_c = (i > e0) ? t2 : march_vertex(s, vxp, Vx_c, vyL, Vy_c, iepL, iep, ieL_c, ie_c, t2, o2);
        if (own) at.st(1, f.txy_out, js, txy_c);
        ie_p = iep;
    }

    // the next row's loads are issued before the current row is computed
    for (int j = js; j <= je; ++j) {
        MarchRow<T> nxt;
        if (j < je) nxt = march_load(f, at, j + 1, e1, inV, inC);
        // row j+1 in 1..n+2: a side-0 y-plane there is a constant (row 1 of a Vertex dimension)
        if (yb && j + 1 >= ylo && j + 1 <= yhi) {
            cur.Vx = fold_y(f.bc, 0, i, j + 1, cur.Vx, Vx_c, T(0));
            cur.Vy = fold_y(f.bc, 1, i, j + 1, cur.Vy, Vy_c, T(0));
        }
        if (xb) {
            cur.Vx = fold_x(f.bc, 0, i, cur.Vx);
            cur.Vy = fold_x(f.bc, 1, i, cur.Vy);
        }
        // new cell (i, j)
        const T vxR = __shfl_down_sync(FULL, Vx_c, 1);
        CellNew<T> c = march_cell(s, f.has_fP != 0, Vx_c, vxR, Vy_c, cur.Vy, ie_c, cur.P, cur.txx, cur.txo, cur.tyy,
                                  cur.tyo, cur.fp);
        if (oldcell) {
            c.P = cur.P;
            c.txx = cur.txx;
            c.tyy = cur.tyy;
        }
        // new vertex (i, j+1)
        const T vyL = __shfl_up_sync(FULL, cur.Vy, 1);
        const T ieL_n = __shfl_up_sync(FULL, cur.ie, 1);
        const T tn = (i > e0 || j + 1 > e1)
                         ? cur.txy
                         : march_vertex(s, Vx_c, cur.Vx, vyL, cur.Vy, ieL_c, ie_c, ieL_n, cur.ie, cur.txy, cur.txyo);
        // velocity (i, j): r_V = -d(P) + d(tau_dd) + d(tau_xy) - rho g, left to right
        const T PL = __shfl_up_sync(FULL, c.P, 1);
        const T TxxL = __shfl_up_sync(FULL, c.txx, 1);
        const T txyR = __shfl_down_sync(FULL, txy_c, 1);
        if (own) {
            T rx = radd(-rmul(rsub(c.P, PL), s.idx[0]), rmul(rsub(c.txx, TxxL), s.idx[0]));
            rx = radd(rx, rmul(rsub(tn, txy_c), s.idx[1]));
            T ry = radd(-rmul(rsub(c.P, Pn_p), s.idx[1]), rmul(rsub(c.tyy, Tyyn_p), s.idx[1]));
            ry = radd(ry, rmul(rsub(txyR, txy_c), s.idx[0]));
            if (f.has_rho) {
                rx = rsub(rx, cur.rhox);
                ry = rsub(ry, cur.rhoy);
            }
            at.st(0, f.P_out, j, c.P);
            at.st(0, f.txx_out, j, c.txx);
            at.st(0, f.tyy_out, j, c.tyy);
            if (j + 1 <= je) at.st(1, f.txy_out, j + 1, tn);
            if (WRITE_RES) {
                at.st(0, f.divV, j, c.dvP);
                at.st(1, f.rVx, j, rx);
                at.st(0, f.rVy, j, ry);
            }
            at.st(1, f.Vx_out, j, radd(Vx_c, rmul(rx, rmul(s.nu_dtau, radd(fmin(ieL_c, ie_c), s.inv_Gdt)))));
            at.st(0, f.Vy_out, j, radd(Vy_c, rmul(ry, rmul(s.nu_dtau, radd(fmin(ie_p, ie_c), s.inv_Gdt)))));
        }
        // advance one row
        Vx_c = cur.Vx;
        Vy_c = cur.Vy;
        ie_p = ie_c;
        ie_c = cur.ie;
        ieL_c = ieL_n;
        Pn_p = c.P;
        Tyyn_p = c.tyy;
        txy_c = tn;
        cur = nxt;
    }
}

// The arrays of a fused view, for host-side checks.
template <class T>
inline void fused_arrays(const Fused2D<T>& f, const DF<T>* out[22]) {
    const DF<T>* all[22] = {&f.Vx_in, &f.Vy_in, &f.Vx_out, &f.Vy_out, &f.txx_in, &f.tyy_in, &f.txy_in, &f.txx_out,
                            &f.tyy_out, &f.txy_out, &f.P_in, &f.P_out, &f.txx_o, &f.tyy_o, &f.txy_o, &f.ieta,
                            &f.fP, &f.rhox, &f.rhoy, &f.divV, &f.rVx, &f.rVy};
    for (int k = 0; k < 22; ++k) out[k] = all[k];
}

// True when every element offset i + j*s1 the marching kernel forms (i, j in [-1, e+1]) fits
// in a 32-bit int for all of f's arrays.
template <class T>
inline bool march_fits_int(const Fused2D<T>& f, int e0, int e1) {
    const DF<T>* all[22];
    fused_arrays(f, all);
    const long lim = 2147483647L;
    for (const DF<T>* d : all) {
        const long s1 = d->s1 < 0 ? -d->s1 : d->s1;
        if ((long)e0 + 1 + ((long)e1 + 1) * s1 > lim) return false;
    }
    return true;
}

// The layout of a view's present arrays and their row strides by location class.
template <class T>
inline int march_layout(const Fused2D<T>& f, MStr2* str) {
    const DF<T>* const c0[15] = {&f.P_in, &f.P_out, &f.txx_in, &f.txx_out, &f.tyy_in, &f.tyy_out, &f.txx_o, &f.tyy_o,
                                 &f.ieta, &f.fP, &f.Vy_in, &f.Vy_out, &f.rhoy, &f.divV, &f.rVy};
    const DF<T>* const c1[7] = {&f.Vx_in, &f.Vx_out, &f.txy_in, &f.txy_out, &f.txy_o, &f.rhox, &f.rVx};
    *str = MStr2{{f.P_in.s1, f.Vx_in.s1}};
    for (const DF<T>* d : c0)
        if (d->p && d->s1 != str->s1[0]) return kLayOwn;
    for (const DF<T>* d : c1)
        if (d->p && d->s1 != str->s1[1]) return kLayOwn;
    return str->s1[0] == str->s1[1] ? kLayOne : kLayLoc;
}

// Rows per warp of the marching kernel: the length at which the strips x segments warps fill
// every SM once at the kernel's occupancy (one wave), kept within [8, 32] rows. Shorter
// segments re-read more boundary rows; longer ones leave the memory system fewer warps'
// worth of loads in flight (measured on 1024^2 to 4096^2 grids).
template <class T, class Ix, int LAY, bool WRITE_RES, int MINB = 1>
inline int march_seg_rows(int num_sms, int nstrip, int rows) {
    static const int blocks_per_sm = [] {
        int nb = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, march2d_kernel<T, Ix, LAY, WRITE_RES, MINB>, 128,
                                                          0) != cudaSuccess)
            nb = 0;
        return nb > 0 ? nb : 4;
    }();
    const long capacity = (long)num_sms * blocks_per_sm * 4;
    const long nseg = capacity / nstrip > 1 ? capacity / nstrip : 1;
    const int seg = (int)((rows + nseg - 1) / nseg);
    return seg < 8 ? 8 : (seg > 32 ? 32 : seg);
}

template <class T, class Ix, int LAY, bool WRITE_RES, int MINB = 1>
inline cudaError_t launch_march2d_ix(const Fused2D<T>& f, const SP<T>& s, int n0, int n1, int num_sms, int seg_rows,
                                     const MStr2& str, cudaStream_t st, bool dep = false) {
    const int e0 = n0 + 1, e1 = n1 + 1;
    const int nstrip = cg_div_up(e0 + 1, 30);
    if (seg_rows <= 0) seg_rows = march_seg_rows<T, Ix, LAY, WRITE_RES, MINB>(num_sms, nstrip, e1 + 1);
    const int nseg = cg_div_up(e1 + 1, seg_rows);
    const int nwarps = nstrip * nseg;
    return cg_launch(march2d_kernel<T, Ix, LAY, WRITE_RES, MINB>, dim3(cg_div_up(nwarps, 4)), dim3(128), 0, st, dep, f,
                     s, e0, e1, nstrip, nwarps, seg_rows, str);
}

// Launch of the warp-marching kernel over [0, n0+1] x [0, n1+1]; seg_rows <= 0 picks the
// segment length from the occupancy; dep = true makes it a dependent launch (cg_launch).
template <class T, bool WRITE_RES>
inline cudaError_t launch_march2d(const Fused2D<T>& f, const SP<T>& s, int n0, int n1, int num_sms, int seg_rows,
                                  cudaStream_t st, bool dep = false) {
    MStr2 str;
    const int lay = march_layout(f, &str);
    // FP32 with shared or class strides fits in 64 registers without spills: 8 blocks (32 warps) per SM
    constexpr int minb = sizeof(T) == 4 ? 8 : 1;
    // 64-bit offsets: 1000 x 2100 FP32 in rows of 4 MB 35 us per iteration with one stride, 36 with class strides and
    // 40 with own strides
    if (!march_fits_int(f, n0 + 1, n1 + 1)) {
        if (lay == kLayOwn) return launch_march2d_ix<T, long, kLayOwn, WRITE_RES>(f, s, n0, n1, num_sms, seg_rows, str, st, dep);
        if (lay == kLayOne) return launch_march2d_ix<T, long, kLayOne, WRITE_RES>(f, s, n0, n1, num_sms, seg_rows, str, st, dep);
        return launch_march2d_ix<T, long, kLayLoc, WRITE_RES>(f, s, n0, n1, num_sms, seg_rows, str, st, dep);
    }
    if (lay == kLayOne) return launch_march2d_ix<T, int, kLayOne, WRITE_RES, minb>(f, s, n0, n1, num_sms, seg_rows, str, st, dep);
    if (lay == kLayLoc) return launch_march2d_ix<T, int, kLayLoc, WRITE_RES, minb>(f, s, n0, n1, num_sms, seg_rows, str, st, dep);
    return launch_march2d_ix<T, int, kLayOwn, WRITE_RES>(f, s, n0, n1, num_sms, seg_rows, str, st, dep);
}

}  // namespace cgk
