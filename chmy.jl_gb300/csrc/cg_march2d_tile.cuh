// cg_march2d_tile.cuh — several 2D PT iterations per launch on tiles kept in registers
// (update_stress! + update_velocity! + bc!(V), examples/stokes_2d_inc_ve_T.jl:20-43,144-146,
// variable-viscosity form).
#pragma once

#include "cg_stokes_kernels.cuh"

namespace cgk {

// A block of W warps holds a tile of 32 columns x W*R rows: lane l holds column i0 + l, warp w the
// rows j0 + w*R .. j0 + w*R + R - 1, one point per lane and row with its whole state in registers.
// It reads the tile once, takes up to K iterations on it and writes the points it owns. Every
// iteration reads one ring of neighbours (a new velocity depends on the old state of the points
// around it), so the values of the outermost ring turn stale with each one: a tile owns what lies
// K rings inside its edges, except on a side where it reaches the end of the grid. x-neighbours come
// from shuffles, y-neighbours from registers or, at the edge of a warp's rows, from shared memory
// (two barriers per iteration). What an iteration uses of the viscosity alone is computed once per
// launch. Points outside the launch range [0, n+1] keep their values; bc!(V) is applied to the
// registers with cg_bc_apply's rules between iterations (VFold), as the marching kernel applies it
// to its reads. Every operation is march2d_kernel's, in its order, so a launch leaves the bits of as
// many launches of that kernel.
//
// What it buys: one launch of march2d_kernel reads and writes every array once per iteration, and on
// a small grid a PT iteration cannot be shorter than one kernel's latency chain (about 10 us at
// 191^2, where the data would take 0.5 us). K iterations per launch divide both.
//
// Static points (outside the launch range, read by their neighbours): a sequence of single
// iterations reads them from the buffer whose turn it is. The two buffers of a ping-pong pair
// normally agree there, and then the registers are right for every iteration; `differ` (device
// memory, kDifferBlocks flags, may be null) says that they do not, and the tile re-reads them before each iteration.
template <class T>
struct TileStatic {
    const int* differ;
    int odd;  // 1: the launch's first iteration takes its turn from the out buffer
};

// Tiles along one dimension of `e` + 1 points (0..e; columns -1 and e+1 are static), `t` points per
// tile, `h` rings of halo.
__host__ __device__ inline int tile_count(int e, int t, int h) {
    if (t - 2 >= e + 1) return 1;  // tile 0 holds -1 .. t-2
    const int rest = e + 1 - (2 * t - 2 - 2 * h);  // beyond tile 1's last point
    return 2 + (rest > 0 ? (rest + t - 2 * h - 1) / (t - 2 * h) : 0);
}
// First owned point of tile q >= 1; its first point lies h before, tile 0's is -1.
__host__ __device__ inline int tile_own(int q, int t, int h) { return q == 0 ? 0 : t - 1 - h + (q - 1) * (t - 2 * h); }

// The x-plane of bc!(V) that lane `lane` (column i) holds for velocity component a: the rule, its
// side and the lane of its source column, packed; 0 where it holds none. A tile is a chain of
// dependent steps, so the rule is one shuffle and selects instead of fold_x's tests on every row:
// with those, and fold_y's, an edge tile took twice an interior one's time (15.2 against 7.0 us for 4
// iterations at 97^2).
template <class T>
__device__ __forceinline__ int tile_xcode(const VFold<T>& b, int a, int i, int lane) {
    const int r0 = b.rule[a][0][0], r1 = b.rule[a][0][1];
    int code = lane << 3;
    if (r0 != FOLD_NONE && i == b.g[a][0][0]) code = r0 | ((r0 == FOLD_CONST ? lane : lane + 1) & 31) << 3;
    if (r1 != FOLD_NONE && i == b.g[a][0][1]) code = r1 | 4 | ((r1 == FOLD_CONST ? lane : lane - 1) & 31) << 3;
    return code;
}

// The value v of component a in a row (on: one of the tangential rows 0..n+2) through its x-plane.
template <class T>
__device__ __forceinline__ T tile_fold_x(const VFold<T>& b, int a, int code, bool on, T v) {
    const T base = __shfl_sync(0xffffffffu, v, code >> 3);
    const T val = (code & 4) ? b.val[a][0][1] : b.val[a][0][0];
    const int t = on ? code & 3 : 0;
    const T dir = rfma(T(2), rsub(val, base), base), neu = rfma(b.h[0], val, base);
    return t == FOLD_NONE ? v : t == FOLD_CONST ? val : t == FOLD_DIRC ? dir : neu;
}

// The value v of component a at row j (column i, between rows of values vprev and vnext) through its
// y-plane: fold_y by selects.
template <class T>
__device__ __forceinline__ T tile_fold_y(const VFold<T>& b, int a, int i, int j, T v, T vprev, T vnext) {
    const int t0 = j == b.g[a][1][0] ? b.rule[a][1][0] : FOLD_NONE, t1 = j == b.g[a][1][1] ? b.rule[a][1][1] : FOLD_NONE;
    const int t = i >= 0 && i <= b.lim[0] ? t0 | t1 : FOLD_NONE;  // a row is one side's plane at most
    const T base = t1 ? vprev : vnext, val = t1 ? b.val[a][1][1] : b.val[a][1][0];
    const T dir = rfma(T(2), rsub(val, base), base), neu = rfma(b.h[1], val, base);
    return t == FOLD_NONE ? v : t == FOLD_CONST ? val : t == FOLD_DIRC ? dir : neu;
}

// Whether row j can be a y-plane of bc!(V): rows 0, 1, n+1 and n+2.
__device__ __forceinline__ bool tile_yrow(int j, int e1) { return j == 0 || j == 1 || j == e1 || j == e1 + 1; }

template <class T, int LAY, bool WRITE_RES, int W, int R, int K, int MINB>
__global__ void __launch_bounds__(32 * W, MINB)
    march2d_tile_kernel(const Fused2D<T> f, const SP<T> s, int e0, int e1, int ntx, int nty, int kit, const MStr2 str,
                        int fold_first, const TileStatic<T> stat) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int TY = W * R;
    // rows at the edges of each warp's rows: velocities (first and last row), then the new P and
    // tau_yy of the last row and the new tau_xy of the first
    __shared__ T sv[4][W][32];
    __shared__ T sn[3][W][32];
    cg_dep_wait();
    cg_dep_release();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int tx = blockIdx.x % ntx, ty = blockIdx.x / ntx;
    const int own_x = tile_own(tx, 32, K), own_y = tile_own(ty, TY, K);
    const int i0 = tx == 0 ? -1 : own_x - K, j0 = ty == 0 ? -1 : own_y - K;
    const int end_x = tx == ntx - 1 ? e0 : tile_own(tx + 1, 32, K) - 1;
    const int end_y = ty == nty - 1 ? e1 : tile_own(ty + 1, TY, K) - 1;
    const int i = i0 + lane, jw = j0 + w * R;
    // Loads have no guards: columns and rows beyond the stored range read its last ones (index n + 2), whose
    // values no owned point depends on, and 1/eta, which the barrier below waits for, comes first. Guarded, in
    // the order of the other arrays, these plain loads took 35.2 us per iteration at 2047 x 1535, this way
    // 29.3 (the same loads by __ldg, which the state does not allow: 33.3).
    const MAt<T, int, LAY> at(i, str), al(min(i, e0 + 1), str);
    const bool inV = i <= e0 + 1, inC = i <= e0;
    const int wd = w > 0 ? w - 1 : 0, wu = w + 1 < W ? w + 1 : W - 1;

    T Vx[R], Vy[R], P[R], txx[R], tyy[R], txy[R];
    T ie[R], eve[R], iev[R], evv[R], sx[R], sy[R], txo[R], tyo[R], txyo[R], fp[R], rhox[R], rhoy[R];
    bool act[R];  // inside the launch range
#pragma unroll
    for (int r = 0; r < R; ++r) ie[r] = al.ldc(0, f.ieta, min(jw + r, e1 + 1), true);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int j = jw + r, jc = min(j, e1 + 1);
        act[r] = i >= 0 && j >= 0 && inC && j <= e1;
        Vx[r] = al.ld(1, f.Vx_in, jc, true);
        Vy[r] = al.ld(0, f.Vy_in, jc, true);
        txy[r] = al.ld(1, f.txy_in, jc, true);
        txyo[r] = al.ldc(1, f.txy_o, jc, true);
        P[r] = al.ld(0, f.P_in, jc, true);
        txx[r] = al.ld(0, f.txx_in, jc, true);
        tyy[r] = al.ld(0, f.tyy_in, jc, true);
        txo[r] = al.ldc(0, f.txx_o, jc, true);
        tyo[r] = al.ldc(0, f.tyy_o, jc, true);
        fp[r] = f.has_fP ? al.ldc(0, f.fP, jc, true) : T(0);
        rhox[r] = f.has_rho ? al.ldc(1, f.rhox, jc, true) : T(0);
        rhoy[r] = f.has_rho ? al.ldc(0, f.rhoy, jc, true) : T(0);
    }
    // the viscosity terms of the tile
    sn[0][w][lane] = ie[R - 1];
    __syncthreads();
    {
        T ieD = sn[0][wd][lane];  // 1/eta of row j-1 (garbage on the tile's first row: halo)
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const T ieL = __shfl_up_sync(FULL, ie[r], 1), ieDL = __shfl_up_sync(FULL, ieD, 1);
            const T half = T(0.5);
            const T lo = rfma(half, rsub(ieD, ieDL), ieDL);
            const T hi = rfma(half, rsub(ie[r], ieL), ieL);
            iev[r] = rfma(half, rsub(hi, lo), lo);
            evv[r] = rrcp(radd(iev[r], s.inv_Gdt));
            eve[r] = rrcp(radd(ie[r], s.inv_Gdt));
            sx[r] = rmul(s.nu_dtau, radd(fmin(ieL, ie[r]), s.inv_Gdt));
            sy[r] = rmul(s.nu_dtau, radd(fmin(ieD, ie[r]), s.inv_Gdt));
            ieD = ie[r];
        }
    }
    const bool differ = stat.differ && __any_sync(FULL, stat.differ[lane] != 0);
    // the tile holds an x-plane / a y-plane of bc!(V) that a row or column of it uses
    const bool xb = f.bc.on && (tx == 0 || i0 + 31 >= e0);
    const bool yb = f.bc.on && (ty == 0 || j0 + TY - 1 >= e1);
    const int xcode = xb ? tile_xcode(f.bc, 0, i, lane) | tile_xcode(f.bc, 1, i, lane) << 8 : 0;
    // rows jw-1 .. jw+R that can be a y-plane
    int yrows = 0;
#pragma unroll
    for (int r = -1; r <= R; ++r) yrows |= (yb && tile_yrow(jw + r, e1)) << (r + 1);

    for (int q = 0; q < kit; ++q) {
        if (differ) {
            const bool out = ((q ^ stat.odd) & 1) != 0;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int j = jw + r;
                if (act[r]) continue;
                const bool v = inV && j <= e1 + 1, c = inC && j <= e1;
                Vx[r] = at.ld(1, out ? f.Vx_out : f.Vx_in, j, v);
                Vy[r] = at.ld(0, out ? f.Vy_out : f.Vy_in, j, v);
                txy[r] = at.ld(1, out ? f.txy_out : f.txy_in, j, v);
                P[r] = at.ld(0, out ? f.P_out : f.P_in, j, c);
                txx[r] = at.ld(0, out ? f.txx_out : f.txx_in, j, c);
                tyy[r] = at.ld(0, out ? f.tyy_out : f.tyy_in, j, c);
            }
        }
        sv[0][w][lane] = Vx[0];
        sv[1][w][lane] = Vy[0];
        sv[2][w][lane] = Vx[R - 1];
        sv[3][w][lane] = Vy[R - 1];
        __syncthreads();
        T vxD = sv[2][wd][lane], vyU = sv[1][wu][lane];  // Vx of row jw-1, Vy of row jw+R
        if (f.bc.on && (q > 0 || fold_first)) {
            if (yrows) {
                const T vyD = sv[3][wd][lane], vxU = sv[0][wu][lane];
                // a plane's source row is the adjacent one and never a y-plane itself
                const T vxD0 = yrows & 1 ? tile_fold_y(f.bc, 0, i, jw - 1, vxD, T(0), Vx[0]) : vxD;
                const T vyU0 = yrows >> (R + 1) ? tile_fold_y(f.bc, 1, i, jw + R, vyU, Vy[R - 1], T(0)) : vyU;
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (yrows >> (r + 1) & 1) {
                        Vx[r] = tile_fold_y(f.bc, 0, i, jw + r, Vx[r], r ? Vx[r ? r - 1 : 0] : vxD, r + 1 < R ? Vx[r + 1 < R ? r + 1 : r] : vxU);
                        Vy[r] = tile_fold_y(f.bc, 1, i, jw + r, Vy[r], r ? Vy[r ? r - 1 : 0] : vyD, r + 1 < R ? Vy[r + 1 < R ? r + 1 : r] : vyU);
                    }
                vxD = vxD0;
                vyU = vyU0;
            }
            if (xb) {  // x-planes over the tangential rows 0..n+2
                const int cx = xcode & 255, cy = xcode >> 8;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const bool on = jw + r >= 0 && jw + r <= e1 + 1;
                    Vx[r] = tile_fold_x(f.bc, 0, cx, on, Vx[r]);
                    Vy[r] = tile_fold_x(f.bc, 1, cy, on, Vy[r]);
                }
                vxD = tile_fold_x(f.bc, 0, cx, jw - 1 >= 0 && jw - 1 <= e1 + 1, vxD);
                vyU = tile_fold_x(f.bc, 1, cy, jw + R >= 0 && jw + R <= e1 + 1, vyU);
            }
        }
        const bool last = WRITE_RES && q == kit - 1;
        // update_stress!
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const T exx = rmul(rsub(__shfl_down_sync(FULL, Vx[r], 1), Vx[r]), s.idx[0]);
            const T eyy = rmul(rsub(r + 1 < R ? Vy[r + 1 < R ? r + 1 : r] : vyU, Vy[r]), s.idx[1]);
            const T vyL = __shfl_up_sync(FULL, Vy[r], 1);
            const T dv = radd(exx, eyy);
            const T dvt = rmul(dv, s.third);
            const T dvP = f.has_fP ? radd(dv, fp[r]) : dv;
            const T exy = rmul(T(0.5), radd(rmul(rsub(Vx[r], r ? Vx[r ? r - 1 : 0] : vxD), s.idx[1]), rmul(rsub(Vy[r], vyL), s.idx[0])));
            const T Pn = rsub(P[r], rmul(rmul(dvP, eve[r]), s.dtau_Pr));
            const T xx = radd(txx[r], rmul(rmul(stress_res(s, txx[r], txo[r], ie[r], rsub(exx, dvt)), eve[r]), s.dtau_r));
            const T yy = radd(tyy[r], rmul(rmul(stress_res(s, tyy[r], tyo[r], ie[r], rsub(eyy, dvt)), eve[r]), s.dtau_r));
            const T xy = radd(txy[r], rmul(rmul(stress_res(s, txy[r], txyo[r], iev[r], exy), evv[r]), s.dtau_r));
            if (act[r]) {
                P[r] = Pn;
                txx[r] = xx;
                tyy[r] = yy;
                txy[r] = xy;
            }
            if (last && act[r] && i >= own_x && i <= end_x && jw + r >= own_y && jw + r <= end_y) at.st(0, f.divV, jw + r, dvP);
        }
        sn[0][w][lane] = P[R - 1];
        sn[1][w][lane] = tyy[R - 1];
        sn[2][w][lane] = txy[0];
        __syncthreads();
        T PD = sn[0][wd][lane], yyD = sn[1][wd][lane];
        const T xyU = sn[2][wu][lane];
        // update_velocity!: r_V = -d(P) + d(tau_dd) + d(tau_xy) - rho g, left to right
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const T PL = __shfl_up_sync(FULL, P[r], 1), xxL = __shfl_up_sync(FULL, txx[r], 1);
            const T xyR = __shfl_down_sync(FULL, txy[r], 1);
            T rx = radd(-rmul(rsub(P[r], PL), s.idx[0]), rmul(rsub(txx[r], xxL), s.idx[0]));
            rx = radd(rx, rmul(rsub(r + 1 < R ? txy[r + 1 < R ? r + 1 : r] : xyU, txy[r]), s.idx[1]));
            T ry = radd(-rmul(rsub(P[r], PD), s.idx[1]), rmul(rsub(tyy[r], yyD), s.idx[1]));
            ry = radd(ry, rmul(rsub(xyR, txy[r]), s.idx[0]));
            if (f.has_rho) {
                rx = rsub(rx, rhox[r]);
                ry = rsub(ry, rhoy[r]);
            }
            PD = P[r];
            yyD = tyy[r];
            if (act[r]) {
                Vx[r] = radd(Vx[r], rmul(rx, sx[r]));
                Vy[r] = radd(Vy[r], rmul(ry, sy[r]));
            }
            if (last && act[r] && i >= own_x && i <= end_x && jw + r >= own_y && jw + r <= end_y) {
                at.st(1, f.rVx, jw + r, rx);
                at.st(0, f.rVy, jw + r, ry);
            }
        }
    }
    if (i < own_x || i > end_x) return;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int j = jw + r;
        if (j < own_y || j > end_y) continue;
        at.st(1, f.Vx_out, j, Vx[r]);
        at.st(0, f.Vy_out, j, Vy[r]);
        at.st(0, f.P_out, j, P[r]);
        at.st(0, f.txx_out, j, txx[r]);
        at.st(0, f.tyy_out, j, tyy[r]);
        at.st(1, f.txy_out, j, txy[r]);
    }
}

// Whether the pair's buffers differ in a static point: the ring -1, e+1 around the launch range. Each
// of the kDifferBlocks blocks writes its part's answer to differ[block].
constexpr int kDifferBlocks = 32;
template <class T>
__global__ void __launch_bounds__(256) static_differ_kernel(const Fused2D<T> f, int e0, int e1, int* differ) {
    const int nx = e0 + 3, ny = e1 + 3;
    int bad = 0;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < 2 * (nx + ny); q += gridDim.x * blockDim.x) {
        int i, j;
        if (q < 2 * nx) {
            i = (q < nx ? q : q - nx) - 1;
            j = q < nx ? -1 : e1 + 1;
        } else {
            const int p = q - 2 * nx;
            i = p < ny ? -1 : e0 + 1;
            j = (p < ny ? p : p - ny) - 1;
        }
        const DF<T>* const a[6] = {&f.Vx_in, &f.Vy_in, &f.P_in, &f.txx_in, &f.tyy_in, &f.txy_in};
        const DF<T>* const b[6] = {&f.Vx_out, &f.Vy_out, &f.P_out, &f.txx_out, &f.tyy_out, &f.txy_out};
#pragma unroll
        for (int c = 0; c < 6; ++c) bad |= bits_of((*a[c])(i, j, 0)) != bits_of((*b[c])(i, j, 0));
    }
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) differ[blockIdx.x] = bad;
}

// The tile shapes (the 2D layouts' variants 1 and up), W x R and K. Measured per iteration against
// the one-iteration kernel's best segment length, in runs of 50 iterations:
//   97^2      1.7 us (variant 2), 8.3 us      1023^2        10.8 us (variant 1), 17.3 us
//   192^2     1.9 us (variant 2), 8.4 us      2047 x 1535   29.0 us (variant 1), 41.1 us
//   384^2     3.0 us (variant 3), 8.9 us      4000^2         137 us (variant 1), 190 us
//   768 x 700 6.5 us (variant 3), 11.0 us
// 32 x 32 tiles of 8 warps with 4 iterations (56 % of the points owned, two blocks per SM) are bound
// by instruction issue from 1023^2 on; up to about 256^2 the grid does not fill the SMs, and 16 warps
// of 2 rows with 8 iterations shorten the chain; 64-row tiles own 66 % but leave one block per SM.
// 3 and 6 iterations per launch, 16-row tiles and 8 warps of 4 rows with 8 iterations lost at every size.
constexpr int kTileVariants = 3;
constexpr int kTileIters[kTileVariants] = {4, 8, 4};

template <class T, bool WRITE_RES, int W, int R, int K, int MINB>
inline cudaError_t launch_tile_shape(const Fused2D<T>& f, const SP<T>& s, int n0, int n1, int kit, bool fold_first,
                                     const TileStatic<T>& stat, cudaStream_t st, bool dep) {
    MStr2 str;
    const int lay = march_layout(f, &str);
    const int e0 = n0 + 1, e1 = n1 + 1;
    const int ntx = tile_count(e0, 32, K), nty = tile_count(e1, W * R, K);
    if (lay == kLayOne)
        return cg_launch(march2d_tile_kernel<T, kLayOne, WRITE_RES, W, R, K, MINB>, dim3(ntx * nty), dim3(32 * W), 0, st, dep, f, s,
                         e0, e1, ntx, nty, kit, str, (int)fold_first, stat);
    return cg_launch(march2d_tile_kernel<T, kLayLoc, WRITE_RES, W, R, K, MINB>, dim3(ntx * nty), dim3(32 * W), 0, st, dep, f, s, e0,
                     e1, ntx, nty, kit, str, (int)fold_first, stat);
}

// `kit` iterations (at most kTileIters[variant - 1]) `in` -> `out` in one launch; fold_first: the
// first one reads its velocities through bc!(V). Only for views that march_tile_ok admits.
template <class T, bool WRITE_RES>
inline cudaError_t launch_march2d_tile(const Fused2D<T>& f, const SP<T>& s, int n0, int n1, int variant, int kit, bool fold_first,
                                       const TileStatic<T>& stat, cudaStream_t st, bool dep = false) {
    switch (variant) {
        case 1: return launch_tile_shape<T, WRITE_RES, 8, 4, 4, 2>(f, s, n0, n1, kit, fold_first, stat, st, dep);
        case 2: return launch_tile_shape<T, WRITE_RES, 16, 2, 8, 1>(f, s, n0, n1, kit, fold_first, stat, st, dep);
        default: return launch_tile_shape<T, WRITE_RES, 16, 4, 4, 1>(f, s, n0, n1, kit, fold_first, stat, st, dep);
    }
}

// Whether the tile kernel can take a view: FP32 (in FP64 the halo's recomputation costs more of the
// FP64 pipe than it saves), strides by location, 32-bit offsets, CG_MARCH_X2 not set to 0.
template <class T>
inline bool march_tile_ok(const Fused2D<T>& f, int n0, int n1) {
    static const bool on = [] {
        const char* e = std::getenv("CG_MARCH_X2");
        return !(e && e[0] == '0');
    }();
    MStr2 str;
    return sizeof(T) == 4 && on && march_layout(f, &str) != kLayOwn && march_fits_int(f, n0 + 1, n1 + 1);
}

}  // namespace cgk
