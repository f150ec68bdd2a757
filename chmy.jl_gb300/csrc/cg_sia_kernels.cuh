// cg_sia_kernels.cuh — device arithmetic shared by the single-member and ensemble shallow-ice
// solvers (Chmy.jl examples/sia.jl:30-54).
//
// The SIA step runs in FP64, and on GB300 it is bound by the FP64 pipe, not by HBM: a cell
// needs tens of FP64 instructions for 24 bytes of traffic. The arithmetic is therefore
// arranged to issue as few FP64 instructions as possible.
// - Integer powers use repeated squaring, written out for Glen's exponent 3.
// - For odd n, vmag(∇S)^(n-1) is an integer power of |∇S|^2, with no square root.
// - D = h^n (Gamma h^2 + As) |∇S|^(n-1) shares the h^n factor of the reference's
//   Gamma h^(n+2) + As h^n.
// - The mean of a cell's two face gradients is (S_i+1 - S_i-1) (idx/2): two instructions for six.
// - A face's flux -(D_l + D_r) ((S_r - S_l) idx/2) takes four for the five of the mean and the
//   gradient, and each face is computed once (x by lane shuffle, y through shared memory).
// A plain step takes about 31 FP64 instructions per cell, 57 before (-lerp, gradients per face twice).
// These forms differ from the reference's evaluation order only in rounding, a few ulp, and every
// operation is rounded by itself or by an explicit fma, so that kernels that recompute a quantity
// (the reverse step's masks) get its bits.
// The maximum of D over a member, which sets the adaptive Δt, is reduced within a block first
// (warp shuffles, then shared memory). One atomic per block then updates the member's slot,
// where an atomic per cell would serialise on a single address.
#pragma once

#include "cg_common.cuh"

namespace cgsia {

// x^m for m >= 0 by repeated squaring (x^1 is x itself, with no multiplication)
template <class T>
__device__ __forceinline__ T pow_int(T x, int m) {
    T r = (m & 1) ? x : T(1);
    m >>= 1;
    while (m) {
        x = x * x;
        if (m & 1) r = r * x;
        m >>= 1;
    }
    return r;
}

// ∇S at a cell along one dimension from the cells beside it; hid = idx/2 (examples/sia.jl:43-45).
template <class T>
__device__ __forceinline__ T slope(T sl, T sr, T hid) {
    return cgk::rmul(cgk::rsub(sr, sl), hid);
}

// q = -lerp(D) ∂S at the face between cells l and r (examples/sia.jl:50-53).
template <class T>
__device__ __forceinline__ T face_flux(T dl, T dr, T sl, T sr, T hid) {
    return cgk::rmul(cgk::radd(dl, dr), cgk::rmul(cgk::rsub(sl, sr), hid));
}

// W = -divg(q) + M at a cell from its four faces and its mass balance.
template <class T>
__device__ __forceinline__ T rate(T qxl, T qxr, T qyl, T qyr, T idx, T idy, T M) {
    return cgk::rsub(M, cgk::rfma(cgk::rsub(qyr, qyl), idy, cgk::rmul(cgk::rsub(qxr, qxl), idx)));
}

// D = (Gamma h^(n+2) + As h^n) vmag^(n-1) at a cell, where vmag^2 = ax^2 + ay^2 and ax, ay are
// the components of ∇S interpolated to the cell (examples/sia.jl:46-49).
template <class T>
__device__ __forceinline__ T D_cell(T h, T ax, T ay, T Gamma, T As, int n) {
    using cgk::rmul;
    const T vm2 = cgk::rfma(ax, ax, rmul(ay, ay)), h2 = rmul(h, h);
    if (n == 3) return rmul(rmul(rmul(h, h2), cgk::rfma(Gamma, h2, As)), vm2);
    const int e = n - 1;
    T vp = pow_int(vm2, e >> 1);
    if (e & 1) vp = rmul(vp, sqrt(vm2));
    return rmul(rmul(pow_int(h, n), cgk::rfma(Gamma, h2, As)), vp);
}

// D at a cell (bit for bit the value of D_cell) and the derivatives a taped forward step
// records, from the same subexpressions: dD/dh, c ax and c ay with c = 2 dD/dV (V = ax^2 + ay^2;
// these are dD/dax and dD/day), and dD/dGamma = h^(n+2) V^((n-1)/2). Gn2 = Gamma (n+2) and
// Asn = As n are the caller's constants.
template <class T>
__device__ __forceinline__ T D_and_factors(T h, T ax, T ay, T Gamma, T As, T Gn2, T Asn, int n, T* dh, T* ex, T* ey,
                                           T* gf) {
    using cgk::rmul;
    const T V = cgk::rfma(ax, ax, rmul(ay, ay)), h2 = rmul(h, h);
    if (n == 3) {
        const T h3 = rmul(h, h2), A = rmul(h3, cgk::rfma(Gamma, h2, As)), c = A + A;
        *dh = fma(Gn2, h2, Asn) * h2 * V;
        *ex = c * ax;
        *ey = c * ay;
        *gf = h3 * h2 * V;
        return rmul(A, V);
    }
    const int e = n - 1;
    T vp = pow_int(V, e >> 1);
    if (e & 1) vp = rmul(vp, sqrt(V));
    const T hn = pow_int(h, n);
    const T A = rmul(hn, cgk::rfma(Gamma, h2, As));
    const T D = rmul(A, vp);
    T c = T(0);
    if (n >= 3) {
        T vq = pow_int(V, (n - 3) >> 1);
        if ((n - 3) & 1) vq = vq * sqrt(V);
        c = A * T(n - 1) * vq;
    } else if (n == 2 && V > T(0)) {
        c = A / sqrt(V);
    }
    *dh = fma(Gn2, h2, Asn) * pow_int(h, n - 1) * vp;
    *ex = c * ax;
    *ey = c * ay;
    *gf = hn * h2 * vp;
    return D;
}

using cgk::bits_of;

using cgk::block_max_bits;

// fmax(u, 0), a NaN's included, from the bits: no FP64 comparison.
__device__ __forceinline__ double pos_part(double u) { return bits_of(u) <= 0x7FF0000000000000ull ? u : 0.0; }
__device__ __forceinline__ float pos_part(float u) { return fmaxf(u, 0.f); }

// Sum over the block (valid in thread 0). Every thread calls it; it may be called more than
// once per kernel (the leading barrier keeps a call's writes after the previous call's reads).
__device__ __forceinline__ double block_sum(double x) {
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ double part[32];
    __syncthreads();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(FULL, x, o);
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    const int lane = tid & 31, warp = tid >> 5, nw = (blockDim.x * blockDim.y + 31) >> 5;
    if (lane == 0) part[warp] = x;
    __syncthreads();
    x = 0.0;
    if (warp == 0) {
        x = lane < nw ? part[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(FULL, x, o);
    }
    return x;  // valid in thread 0
}

// ---- tape of a forward run, read by the reverse sweep ---------------------------------------
//
// A taped forward step records what the reverse step would otherwise recompute in FP64. This
// trades HBM traffic, which the SIA kernels barely use, for FP64 instructions, which bound them.
// Layout: a 256-byte header, then per step a 256-byte word block and kArrays arrays of `cnt`
// elements in H's padded layout (each rounded up to 256 bytes).
enum TapeArray {
    kD = 0,   // D over the interior cells [1, n]^2
    kGX = 1,  // dS/dx at the cell's lower x face ((S_i - S_i-1)/dx)
    kGY = 2,  // dS/dy at the lower y face
    kDH = 3,  // dD/dh
    kEX = 4,  // dD/dax = 2 dD/dV ax  (V = ax^2 + ay^2)
    kEY = 5,  // dD/day = 2 dD/dV ay
    kGF = 6,  // dD/dGamma = h^(n+2) V^((n-1)/2)
    kW = 7,   // W = -divg(q) + M
    kFL = 8,  // one byte per cell: 1 if H + dt W > 0, plus 2 if the mass balance is not capped
    kArrays = 9
};

struct TapeHeader {
    unsigned long long magic;
    int dtype, nx, ny, nsteps;
    long long stride0, stride1, halo0, halo1, n0, n1, cnt, step_bytes;
    double Gamma, As, beta, ela, m_max, cfl, dt_max;
    int n, pad;
};
constexpr unsigned long long kTapeMagic = 0x3145504154414953ull;  // "SIATAPE1"

// per step: the forward's Dmax bits, the first interior argmax (j (nx+2) + i), dt and whether
// dt was capped at dt_max
struct TapeWords {
    unsigned long long dmax;
    unsigned long long arg;
    double dt;
    double capped;
};

struct TapeGeom {
    size_t cnt, abytes, step_bytes;
};

// elements per array: H's allocation (row stride x padded rows)
inline TapeGeom tape_geom(const cg_field& H, size_t elem) {
    TapeGeom g;
    g.cnt = (size_t)H.stride[1] * (size_t)(H.n[1] + 4 * H.halo[1]);
    g.abytes = (g.cnt * elem + 255) & ~(size_t)255;
    g.step_bytes = 256 + (size_t)kArrays * g.abytes;
    return g;
}

// ---- the two kernels of a time step ----------------------------------------------------------
//
// A step is two launches over 32 x rows tiles of the interior cells: D and its maximum
// (D_tile), then Δt, the fluxes, the thickness and its boundary copies together (H_tile). The
// fluxes stay in registers and shared memory; only the last step of a run stores them (nothing
// else reads q). H_tile reads its neighbours' S = B + H while other tiles update theirs, so S has
// two buffers that alternate by step, and the maximum of D two slots. Of D only the interior cells
// are read: the faces on the boundary carry no flux. Measured against six launches per step (D, q,
// bc!(q), Δt, H, bc!(H)) and four for an ensemble (D, q, Δt, H): 383 x 255 22.7 -> 14.6 us per step, 64
// members of 128^2 to 1024^2 (26.3 M cells, 1.3 ms at the FP64 pipe's rate) 2.42 -> 1.71 ms, 64 members
// of 32^2 to 128^2 62 -> 42 us. Boundary conditions are those of bc!: q.x =>
// (x = Dirichlet()) is 0 on the faces 1 and n+1 (q.y likewise), and H => Neumann() copies the first
// interior value into the ghost layer, a corner the diagonal interior cell's.
template <class T>
struct Member {
    DF<T> H, B, qx, qy, D, S[2];
    T Gamma, As, beta, ela, m_max, idx, idy, hidx, hidy;
    T Gn2, Asn;  // Gamma (n+2) and As n, for the taped derivatives of D
    double dx2, dt_max;
    cgk::ConstDiv<T> cfl;
    int n, nx, ny;
    // taped runs: the member's tape block within a step's block (256 bytes of words, then kArrays
    // arrays of `tab` bytes in H's layout, H's origin at element `orig`)
    long long toff, tab, orig;
};

struct Words {
    unsigned long long dmax[3];  // the step's maximum of D, by step parity (one launch per step: modulo 3)
    double t;
};

// The member's tape array k (TapeArray) of the step whose block starts at `sb`.
template <class T>
__device__ __forceinline__ DF<T> tape_arr(const Member<T>& v, char* sb, int k) {
    DF<T> a = v.H;
    a.p = reinterpret_cast<T*>(sb + v.toff + 256 + (long long)k * v.tab) + v.orig;
    return a;
}
template <class T>
__device__ __forceinline__ DF<unsigned char> tape_flags(const Member<T>& v, char* sb) {
    DF<unsigned char> a;
    a.p = reinterpret_cast<unsigned char*>(sb + v.toff + 256 + (long long)kFL * v.tab) + v.orig;
    a.s1 = v.H.s1;
    a.s2 = v.H.s2;
    return a;
}
template <class T>
__device__ __forceinline__ TapeWords* tape_words(const Member<T>& v, char* sb) {
    return reinterpret_cast<TapeWords*>(sb + v.toff);
}

// S = B + H of the run's start over [0, n+1]^2 (tile t of 32 x blockDim.y points).
template <class T>
__device__ __forceinline__ void S_tile(const Member<T>& v, int t) {
    const int tx = (v.nx + 2 + 31) / 32;
    const int i = (t % tx) * 32 + threadIdx.x, j = (t / tx) * (int)blockDim.y + threadIdx.y;
    if (i > v.nx + 1 || j > v.ny + 1) return;
    v.S[0](i, j, 0) = v.B(i, j, 0) + v.H(i, j, 0);
}

// H of the run's start over its interior cells into `dst` (the same tiles).
template <class T>
__device__ __forceinline__ void H_copy_tile(const Member<T>& v, const DF<T>& dst, int t) {
    const int tx = (v.nx + 2 + 31) / 32;
    const int i = (t % tx) * 32 + threadIdx.x, j = (t / tx) * (int)blockDim.y + threadIdx.y;
    if (i >= 1 && i <= v.nx && j >= 1 && j <= v.ny) dst(i, j, 0) = v.H(i, j, 0);
}

// D at the interior cells of tile t and its maximum. TAPE: D goes to the step's tape block, with
// the lower faces' gradients and D's derivatives.
template <class T, bool TAPE>
__device__ __forceinline__ void D_tile(const Member<T>& v, Words* w, int t, int par, char* sb) {
    const int tx = (v.nx + 31) / 32;
    const int i = (t % tx) * 32 + threadIdx.x + 1, j = (t / tx) * (int)blockDim.y + threadIdx.y + 1;
    const bool in = i <= v.nx && j <= v.ny;
    const DF<T>& S = v.S[par];
    T d = T(0);
    if (in) {
        const T sl = S(i - 1, j, 0), sb0 = S(i, j - 1, 0);
        const T ax = slope(sl, S(i + 1, j, 0), v.hidx), ay = slope(sb0, S(i, j + 1, 0), v.hidy);
        const T h = v.H(i, j, 0);
        if (TAPE) {
            const T s = S(i, j, 0);
            T dh, ex, ey, gf;
            d = D_and_factors(h, ax, ay, v.Gamma, v.As, v.Gn2, v.Asn, v.n, &dh, &ex, &ey, &gf);
            tape_arr(v, sb, kD)(i, j, 0) = d;
            tape_arr(v, sb, kGX)(i, j, 0) = (s - sl) * v.idx;
            tape_arr(v, sb, kGY)(i, j, 0) = (s - sb0) * v.idy;
            tape_arr(v, sb, kDH)(i, j, 0) = dh;
            tape_arr(v, sb, kEX)(i, j, 0) = ex;
            tape_arr(v, sb, kEY)(i, j, 0) = ey;
            tape_arr(v, sb, kGF)(i, j, 0) = gf;
            if (t == 0 && threadIdx.x == 0 && threadIdx.y == 0) tape_words(v, sb)->arg = ~0ull;
        } else {
            d = D_cell(h, ax, ay, v.Gamma, v.As, v.n);
            v.D(i, j, 0) = d;
        }
    }
    block_max_bits(in ? bits_of(d) : 0ull, &w->dmax[par]);
}

// Δt = min(min(Δ)^2 / max(D) / cfl, dt_max) (examples/sia.jl:73-75, in the grid type).
template <class T>
__device__ __forceinline__ double step_dt(const Member<T>& v, unsigned long long b, bool* capped) {
    const double dmax = sizeof(T) == 8 ? __longlong_as_double((long long)b) : (double)__int_as_float((int)(unsigned)b);
    const T q = cgk::divide((T)v.dx2 / (T)dmax, v.cfl);
    double d = fmin((double)q, v.dt_max);
    *capped = !((double)q < v.dt_max);
    if (!(dmax > 0.0)) {
        d = v.dt_max;
        *capped = true;
    }
    return d;
}

constexpr int kMaxRows = 16;  // tile rows
constexpr int kHCols = 31;    // columns a tile of H_tile owns

// The rest of the step on tile t of 31 x rows cells. Every face is computed once: lane l takes the
// left face of its cell and lane l-1 gets it as its right face (lane 31 only supplies lane 30's; a
// 32nd column would cost the warp a second face's four instructions); the rows pass the y faces
// through shared memory. LAST: the fluxes are stored (with their boundary values). DRY: nothing is
// stored (the autotuner's launches). NANMAX: std::min/std::max semantics, in which a NaN propagates;
// else fmin/fmax.
template <class T, bool TAPE, bool NANMAX>
__device__ __forceinline__ void H_tile(const Member<T>& v, Words* w, int t, int par, bool last, bool dry, char* sb) {
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ T qy[kMaxRows + 1][32];
    __shared__ T s_dt;
    const int lane = threadIdx.x, row = threadIdx.y, rows = blockDim.y;
    const int tx = (v.nx + kHCols - 1) / kHCols;
    const int i = (t % tx) * kHCols + lane + 1, j = (t / tx) * rows + row + 1;
    const bool in = i <= v.nx && j <= v.ny;
    const unsigned long long bits = w->dmax[par];
    const DF<T>& S = v.S[par];
    const DF<T> D = TAPE ? tape_arr(v, sb, kD) : v.D;
    T dc = T(0), s = T(0), h = T(0), b = T(0), dl = T(0), sl = T(0), dd = T(0), sd = T(0);
    if (in) {
        dc = D(i, j, 0);
        s = S(i, j, 0);
        if (i > 1) {
            dl = D(i - 1, j, 0);
            sl = S(i - 1, j, 0);
        }
        if (j > 1) {
            dd = D(i, j - 1, 0);
            sd = S(i, j - 1, 0);
        }
        h = v.H(i, j, 0);
        b = v.B(i, j, 0);
    }
    if (lane == 0 && row == 0) {  // two divisions, while the loads arrive
        bool capped;
        const double d = step_dt(v, bits, &capped);
        s_dt = (T)d;
        if (t == 0 && !dry) {
            w->t += d;
            w->dmax[par ^ 1] = 0ull;
            if (TAPE) {
                TapeWords* tw = tape_words(v, sb);
                tw->dmax = bits;
                tw->dt = d;
                tw->capped = capped ? 1.0 : 0.0;
            }
        }
    }
    const T qxl = in && i > 1 ? face_flux(dl, dc, sl, s, v.hidx) : T(0);
    const T qyl = in && j > 1 ? face_flux(dd, dc, sd, s, v.hidy) : T(0);
    qy[row][lane] = qyl;
    if (row == rows - 1) qy[rows][lane] = in && j < v.ny ? face_flux(dc, D(i, j + 1, 0), s, S(i, j + 1, 0), v.hidy) : T(0);
    const T qxr = __shfl_down_sync(FULL, qxl, 1);  // 0 beyond the last column
    __syncthreads();
    if (!in || lane == kHCols) return;
    const T qyr = qy[row + 1][lane];
    // M = min(beta (S - ela), m_max) and H = max(H + dt (-divg q + M), 0)
    const T x = cgk::rmul(v.beta, cgk::rsub(s, v.ela));
    const T mb = NANMAX ? (v.m_max < x ? v.m_max : x) : fmin(x, v.m_max);
    const T W = rate(qxl, qxr, qyl, qyr, v.idx, v.idy, mb);
    const T u = cgk::rfma(s_dt, W, h);
    const T hn = NANMAX ? (u < T(0) ? T(0) : u) : pos_part(u);
    if (dry && hn != T(-1)) return;  // hn is never -1: the work is done, nothing is stored
    if (TAPE) {
        tape_arr(v, sb, kW)(i, j, 0) = W;
        tape_flags(v, sb)(i, j, 0) = (unsigned char)((u > T(0) ? 1 : 0) + ((NANMAX ? !(v.m_max < x) : x < v.m_max) ? 2 : 0));
        if (bits_of(dc) == bits) atomicMin(&tape_words(v, sb)->arg, (unsigned long long)((long)j * (v.nx + 2) + i));
    }
    const DF<T>& Sn = v.S[par ^ 1];
    v.H(i, j, 0) = hn;
    Sn(i, j, 0) = b + hn;
    const bool l = i == 1, r = i == v.nx, lo = j == 1, hi = j == v.ny;
    if (last) {
        v.qx(i, j, 0) = qxl;
        v.qy(i, j, 0) = qyl;
        if (r) v.qx(i + 1, j, 0) = T(0);
        if (hi) v.qy(i, j + 1, 0) = T(0);
    }
    if (!(l || r || lo || hi)) return;
    auto ghost = [&](int gi, int gj) {
        v.H(gi, gj, 0) = hn;
        Sn(gi, gj, 0) = v.B(gi, gj, 0) + hn;
    };
    if (l) ghost(0, j);
    if (r) ghost(v.nx + 1, j);
    if (lo) ghost(i, 0);
    if (hi) ghost(i, v.ny + 1);
    if (l && lo) ghost(0, 0);
    if (r && lo) ghost(v.nx + 1, 0);
    if (l && hi) ghost(0, v.ny + 1);
    if (r && hi) ghost(v.nx + 1, v.ny + 1);
}

// The descriptor of one member on the host (scratch: D and the two S buffers, in H's layout).
template <class T>
inline Member<T> make_member(const cg_grid& g, const cg_field& H, const cg_field& B, const cg_field* q, const cg_sia_params& p,
                             char* D, char* S0, char* S1) {
    Member<T> v;
    std::memset(&v, 0, sizeof(v));
    v.H = cg_view<T>(H);
    v.B = cg_view<T>(B);
    v.qx = cg_view<T>(q[0]);
    v.qy = cg_view<T>(q[1]);
    v.D = v.S[0] = v.S[1] = v.H;
    v.D.p = reinterpret_cast<T*>(D) + cg_origin_offset(H);
    v.S[0].p = reinterpret_cast<T*>(S0) + cg_origin_offset(H);
    v.S[1].p = reinterpret_cast<T*>(S1) + cg_origin_offset(H);
    v.Gamma = (T)p.Gamma;
    v.As = (T)p.As;
    v.beta = (T)p.beta;
    v.ela = (T)p.ela;
    v.m_max = (T)p.m_max;
    v.Gn2 = v.Gamma * T(p.n + 2);
    v.Asn = v.As * T(p.n);
    v.idx = (T)g.inv_spacing[0];
    v.idy = (T)g.inv_spacing[1];
    v.hidx = T(0.5) * v.idx;
    v.hidy = T(0.5) * v.idy;
    const double dx = std::min(g.spacing[0], g.spacing[1]);
    v.dx2 = (double)((T)dx * (T)dx);
    v.cfl = cgk::const_div<T>((T)p.cfl);
    v.dt_max = p.dt_max;
    v.n = p.n;
    v.nx = g.n[0];
    v.ny = g.n[1];
    return v;
}

// Bytes of one scratch array in H's layout.
inline size_t layout_bytes(const cg_field& H, size_t elem) {
    return ((size_t)H.stride[1] * (size_t)(H.n[1] + 4 * H.halo[1]) * elem + 255) & ~(size_t)255;
}

}  // namespace cgsia
