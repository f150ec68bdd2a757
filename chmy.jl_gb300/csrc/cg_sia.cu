// cg_sia.cu — shallow-ice flow (Chmy.jl examples/sia.jl:7-16,30-54,71-81).
#include "cg_common.cuh"
#include "cg_sia_kernels.cuh"

int cg_maxabs_collect(cg_ctx* ctx, int nfields, const cg_field* fields, double* out, int32_t* nonfinite);
void* cg_scratch(cg_ctx* ctx, int slot, size_t bytes, int* rc);

namespace {

template <class T>
struct SiaV {
    DF<T> H, B, qx, qy;
    T Gamma, As, beta, ela, m_max;
    T idx, idy;
    int n;
};

template <class T>
__device__ __forceinline__ T S_at(const SiaV<T>& v, int i, int j) {
    return v.B(i, j, 0) + v.H(i, j, 0);
}

// D = (Gamma H^(n+2) + As H^n) vmag(∇S)^(n-1) at cell (i, j) (sia.jl:43-49)
template <class T>
__device__ __forceinline__ T D_at(const SiaV<T>& v, int i, int j) {
    const T ax = cgsia::slope(S_at(v, i - 1, j), S_at(v, i + 1, j), T(0.5) * v.idx);
    const T ay = cgsia::slope(S_at(v, i, j - 1), S_at(v, i, j + 1), T(0.5) * v.idy);
    return cgsia::D_cell(v.H(i, j, 0), ax, ay, v.Gamma, v.As, v.n);
}

using cgsia::bits_of;

// update_q! over [1, n]^2 with D evaluated on the fly (the reference's FunctionField);
// optional max(interior D) into *dmax_bits (D >= 0, so the bit patterns order like values).
template <class T>
__global__ void sia_q_kernel(const SiaV<T> v, int nx, int ny, unsigned long long* dmax_bits) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const bool in = i <= nx && j <= ny;
    T dc = T(0);
    if (in) {
        dc = D_at(v, i, j);
        const T dl = D_at(v, i - 1, j), dd = D_at(v, i, j - 1);
        const T Dx = fma(T(0.5), dc - dl, dl);
        const T Dy = fma(T(0.5), dc - dd, dd);
        const T sc = S_at(v, i, j);
        v.qx(i, j, 0) = -Dx * ((sc - S_at(v, i - 1, j)) * v.idx);
        v.qy(i, j, 0) = -Dy * ((sc - S_at(v, i, j - 1)) * v.idy);
    }
    if (dmax_bits) cgsia::block_max_bits(in ? bits_of(dc) : 0ull, dmax_bits);
}

// The kernels of a time step (cgsia::D_tile, cgsia::H_tile) on one member.
template <class T>
__global__ void sia_S_kernel(const cgsia::Member<T> v, const DF<T> Hcopy, int copy) {
    cgsia::S_tile(v, blockIdx.x);
    if (copy) cgsia::H_copy_tile(v, Hcopy, blockIdx.x);
}
template <class T, bool TAPE>
__global__ void __launch_bounds__(256) sia_D_kernel(const cgsia::Member<T> v, cgsia::Words* w, int par, char* sb) {
    cg_dep_wait();
    cg_dep_release();
    cgsia::D_tile<T, TAPE>(v, w, blockIdx.x, par, sb);
}
template <class T, bool TAPE>
__global__ void __launch_bounds__(256) sia_step_kernel(const cgsia::Member<T> v, cgsia::Words* w, int par, int last, int dry, char* sb) {
    cg_dep_wait();
    cg_dep_release();
    cgsia::H_tile<T, TAPE, false>(v, w, blockIdx.x, par, last != 0, dry != 0, sb);
}

// ---- a whole time step in one launch ----------------------------------------------------------
//
// Small grids are bound by the step's two launches, each a chain of dependent launch, loads, a few
// FP64 operations and stores, not by their arithmetic. One launch does Δt, the fluxes, the thickness
// and then the next step's D, whose maximum the next launch reads. A tile owns 29 x R cells and works
// on one more cell each way: it computes the thickness of the ring around its cells too, for the
// slopes of the new S (in shared memory; beside the boundary from H's Neumann copy), so nothing
// waits on another tile. H, D and S alternate between two buffers, the maximum between three words
// (read, raised, cleared). A warp of its own computes Δt's divisions while the others load. Every
// operation is that of D_tile and H_tile, so the bits are those of the two launches.
// The repeated work (1.38 times the thickness of R = 8) bounds larger grids. Measured per step, two
// launches -> one: FP64 64 x 90 6.4 -> 4.4 us, 200^2 8.9 -> 7.3, 383 x 255 14.3 -> 11.8; FP32 64 x 90
// 4.2 -> 2.5, 383 x 255 4.8 -> 3.4, 511^2 7.1 -> 5.6.
constexpr int kOwn = 29;  // columns a tile owns

template <class T>
struct StepBufs {
    DF<T> H, D, S;     // the step's thickness, D and S
    DF<T> Hn, Dn, Sn;  // the next step's
};

template <class T, int R>
__global__ void __launch_bounds__(32 * (R + 3))
    sia_whole_step_kernel(const cgsia::Member<T> v, const StepBufs<T> f, cgsia::Words* w, int slot, int last) {
    using namespace cgsia;
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ T qy[R + 3][32];  // lower-face flux of row r; [R + 2]: the last row's upper face
    __shared__ T Sh[R + 2][32];  // the next step's S
    __shared__ T s_dt;
    const int lane = threadIdx.x, row = threadIdx.y;
    const int tx = (v.nx + kOwn - 1) / kOwn;
    const int i = ((int)blockIdx.x % tx) * kOwn + lane, j = ((int)blockIdx.x / tx) * R + row;
    const bool in = row < R + 2 && i >= 1 && i <= v.nx && j >= 1 && j <= v.ny;
    const bool own = in && lane >= 1 && lane <= kOwn && row >= 1 && row <= R;
    const bool l = i == 1, r = i == v.nx, lo = j == 1, hi = j == v.ny;
    // no kernel of a run writes B: it is read before the wait
    T b = T(0), bl = T(0), br = T(0), bd = T(0), bu = T(0);
    if (in) {
        b = v.B(i, j, 0);
        if (l) bl = v.B(i - 1, j, 0);
        if (r) br = v.B(i + 1, j, 0);
        if (lo) bd = v.B(i, j - 1, 0);
        if (hi) bu = v.B(i, j + 1, 0);
    }
    cg_dep_wait();
    cg_dep_release();
    T dc = T(0), s = T(0), h = T(0), dl = T(0), sl = T(0), dd = T(0), sd = T(0), du = T(0), su = T(0);
    if (in) {
        dc = f.D(i, j, 0);
        s = f.S(i, j, 0);
        if (!l) {
            dl = f.D(i - 1, j, 0);
            sl = f.S(i - 1, j, 0);
        }
        if (!lo) {
            dd = f.D(i, j - 1, 0);
            sd = f.S(i, j - 1, 0);
        }
        if (row == R + 1 && !hi) {
            du = f.D(i, j + 1, 0);
            su = f.S(i, j + 1, 0);
        }
        h = f.H(i, j, 0);
    }
    if (row == R + 2 && lane == 0) {
        bool capped;
        const double d = step_dt(v, w->dmax[slot], &capped);
        s_dt = (T)d;
        if (blockIdx.x == 0) {
            w->t += d;
            w->dmax[slot == 0 ? 2 : slot - 1] = 0ull;  // the previous step's: the one after the next uses it
        }
    }
    const T qxl = in && !l ? face_flux(dl, dc, sl, s, v.hidx) : T(0);
    const T qyl = in && !lo ? face_flux(dd, dc, sd, s, v.hidy) : T(0);
    if (row < R + 2) qy[row][lane] = qyl;
    if (row == R + 1) qy[R + 2][lane] = in && !hi ? face_flux(dc, du, s, su, v.hidy) : T(0);
    const T qxr = __shfl_down_sync(FULL, qxl, 1);  // 0 beyond the last column
    __syncthreads();
    T hn = T(0);
    if (in && lane < 31) {
        const T W = rate(qxl, qxr, qyl, qy[row + 1][lane], v.idx, v.idy, fmin(cgk::rmul(v.beta, cgk::rsub(s, v.ela)), v.m_max));
        hn = pos_part(cgk::rfma(s_dt, W, h));
        Sh[row][lane] = b + hn;
        // S beside the boundary: H's Neumann copy
        if (l) Sh[row][lane - 1] = bl + hn;
        if (r) Sh[row][lane + 1] = br + hn;
        if (lo) Sh[row - 1][lane] = bd + hn;
        if (hi && row <= R) Sh[row + 1][lane] = bu + hn;
    }
    if (own) {
        f.Hn(i, j, 0) = hn;
        if (!last) {
            f.Sn(i, j, 0) = b + hn;
        } else {
            v.qx(i, j, 0) = qxl;
            v.qy(i, j, 0) = qyl;
            if (r) v.qx(i + 1, j, 0) = T(0);
            if (hi) v.qy(i, j + 1, 0) = T(0);
            if (l) f.Hn(0, j, 0) = hn;
            if (r) f.Hn(v.nx + 1, j, 0) = hn;
            if (lo) f.Hn(i, 0, 0) = hn;
            if (hi) f.Hn(i, v.ny + 1, 0) = hn;
            if (l && lo) f.Hn(0, 0, 0) = hn;
            if (r && lo) f.Hn(v.nx + 1, 0, 0) = hn;
            if (l && hi) f.Hn(0, v.ny + 1, 0) = hn;
            if (r && hi) f.Hn(v.nx + 1, v.ny + 1, 0) = hn;
        }
    }
    if (last) return;
    __syncthreads();
    T d = T(0);
    if (own) {
        const T ax = slope(Sh[row][lane - 1], Sh[row][lane + 1], v.hidx);
        const T ay = slope(Sh[row - 1][lane], Sh[row + 1][lane], v.hidy);
        d = D_cell(hn, ax, ay, v.Gamma, v.As, v.n);
        f.Dn(i, j, 0) = d;
    }
    block_max_bits(own ? bits_of(d) : 0ull, &w->dmax[slot == 2 ? 0 : slot + 1]);
}

// update_H! over [1, n]^2.
template <class T>
__global__ void sia_H_kernel(const SiaV<T> v, int nx, int ny, T dt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    if (i > nx || j > ny) return;
    const T m = fmin(v.beta * (S_at(v, i, j) - v.ela), v.m_max);
    T dv = (v.qx(i + 1, j, 0) - v.qx(i, j, 0)) * v.idx;
    dv = dv + (v.qy(i, j + 1, 0) - v.qy(i, j, 0)) * v.idy;
    v.H(i, j, 0) = fmax(v.H(i, j, 0) + dt * (-dv + m), T(0.0));
}

template <class T>
SiaV<T> make_view(const cg_grid* g, const cg_field* H, const cg_field* B, const cg_field* q, const cg_sia_params* p) {
    SiaV<T> v;
    std::memset(&v, 0, sizeof(v));
    v.H = cg_view<T>(*H);
    v.B = cg_view<T>(*B);
    if (q) {
        v.qx = cg_view<T>(q[0]);
        v.qy = cg_view<T>(q[1]);
    }
    v.Gamma = (T)p->Gamma;
    v.As = (T)p->As;
    v.beta = (T)p->beta;
    v.ela = (T)p->ela;
    v.m_max = (T)p->m_max;
    v.idx = (T)g->inv_spacing[0];
    v.idy = (T)g->inv_spacing[1];
    v.n = p->n;
    return v;
}

int check_sia(cg_ctx* ctx, const cg_grid* g, const cg_field* H, const cg_field* B, const cg_field* q,
              const cg_sia_params* p) {
    int rc = cg_check_grid(ctx, g);
    if (rc) return rc;
    if (g->ndim != 2) return cg_fail(ctx, CG_ERR_UNSUPPORTED, "sia: 2D grids only");
    if (!H || !B || !p) return cg_fail(ctx, CG_ERR_ARG, "sia: NULL argument");
    if ((rc = cg_check_field(ctx, g, *H, H->dtype, 0, "H"))) return rc;
    if ((rc = cg_check_field(ctx, g, *B, H->dtype, 0, "B"))) return rc;
    if (q) {
        if ((rc = cg_check_field(ctx, g, q[0], H->dtype, 1, "q.x"))) return rc;
        if ((rc = cg_check_field(ctx, g, q[1], H->dtype, 2, "q.y"))) return rc;
    }
    if (p->n < 1 || p->n > 16) return cg_fail(ctx, CG_ERR_ARG, "sia: Glen exponent %d not in 1..16", p->n);
    return CG_OK;
}

void sia_bcs(cg_bc* qb, cg_bc* hb) {
    std::memset(qb, 0, 2 * sizeof(cg_bc));
    qb[0].kind[0][0] = qb[0].kind[0][1] = CG_BC_DIRICHLET;
    qb[1].kind[1][0] = qb[1].kind[1][1] = CG_BC_DIRICHLET;
    std::memset(hb, 0, sizeof(cg_bc));
    hb->kind[0][0] = hb->kind[0][1] = hb->kind[1][0] = hb->kind[1][1] = CG_BC_NEUMANN;
}

template <class T>
int update_q_t(cg_ctx* ctx, const cg_grid* g, const cg_field* q, const cg_field* H, const cg_field* B,
               const cg_sia_params* p, double* dmax) {
    const SiaV<T> v = make_view<T>(g, H, B, q, p);
    const dim3 block(32, 8), grid(cg_div_up(g->n[0], 32), cg_div_up(g->n[1], 8));
    if (dmax) CG_CUDA(ctx, cudaMemsetAsync(ctx->d_red, 0, sizeof(unsigned long long), ctx->stream));
    sia_q_kernel<T><<<grid, block, 0, ctx->stream>>>(v, g->n[0], g->n[1], dmax ? ctx->d_red : nullptr);
    CG_CHECK_LAUNCH(ctx);
    cg_bc qb[2], hb;
    sia_bcs(qb, &hb);
    int rc = cg_bc_apply_impl(ctx, g, 2, q, qb);
    if (rc) return rc;
    if (dmax) {
        cg_field probe = *H;  // dtype of the reduction slot
        double m;
        return cg_maxabs_collect(ctx, 1, &probe, &m, nullptr) ? CG_ERR_CUDA : ((*dmax = m), CG_OK);
    }
    return CG_OK;
}

template <class T>
int update_H_t(cg_ctx* ctx, const cg_grid* g, const cg_field* H, const cg_field* q, const cg_field* B, double dt,
               const cg_sia_params* p) {
    const SiaV<T> v = make_view<T>(g, H, B, q, p);
    const dim3 block(32, 8), grid(cg_div_up(g->n[0], 32), cg_div_up(g->n[1], 8));
    sia_H_kernel<T><<<grid, block, 0, ctx->stream>>>(v, g->n[0], g->n[1], (T)dt);
    CG_CHECK_LAUNCH(ctx);
    cg_bc qb[2], hb;
    sia_bcs(qb, &hb);
    return cg_bc_apply_impl(ctx, g, 1, H, &hb);
}

constexpr int kStepRows[3] = {4, 8, 13};  // tile heights of sia_whole_step_kernel

template <class T>
cudaError_t launch_whole_step(int rows, const cgsia::Member<T>& v, const StepBufs<T>& f, cgsia::Words* w, int slot, int last,
                              cudaStream_t st) {
    const dim3 grid(cg_div_up(v.nx, kOwn) * cg_div_up(v.ny, rows)), block(32, rows + 3);
    if (rows == 4) return cg_launch(sia_whole_step_kernel<T, 4>, grid, block, 0, st, true, v, f, w, slot, last);
    if (rows == 8) return cg_launch(sia_whole_step_kernel<T, 8>, grid, block, 0, st, true, v, f, w, slot, last);
    return cg_launch(sia_whole_step_kernel<T, 13>, grid, block, 0, st, true, v, f, w, slot, last);
}

// One launch per step is a candidate up to this many cells: beyond 1200 (FP64) or 4000 (FP32) per SM
// the work that its tiles repeat costs more than the second launch (511^2 FP64 27.0 against 23.2 us per
// step, 1023^2 FP32 17.8 against 16.0).
template <class T>
bool whole_step_fits(const cg_ctx* ctx, const cg_grid* g) {
    return (long)g->n[0] * g->n[1] <= (sizeof(T) == 8 ? 1200l : 4000l) * ctx->num_sms;
}

// The tile height of the one-launch step, or 0 for two launches: CG_SIA_STEP_ROWS when set, else the
// fastest (the time goes in steps of a tile row per SM, so the best height changes from size to size:
// FP64 160^2 to 400 x 300 prefer 4, 13, two launches, 13, 8). Without the autotuner: 8 rows up to 2/3
// of whole_step_fits' range. The candidates write only scratch and the words, which the run clears.
template <class T>
int step_rows(cg_ctx* ctx, const cg_grid* g, const cg_field* H, const cgsia::Member<T>& v, const DF<T>* Hb, const DF<T>* Db,
              cgsia::Words* words) {
    int rows = cg_sia_step_rows_forced();
    if (rows >= 0) return rows;
    if (!cg_autotune_enabled())
        return (long)g->n[0] * g->n[1] * 3 <= (sizeof(T) == 8 ? 2400l : 8000l) * ctx->num_sms ? 8 : 0;
    std::string key = "sia_step";
    cg_key_add(key, g->n);
    cg_key_add(key, (int)sizeof(T));
    cg_key_add(key, H->stride);
    cg_key_add(key, v.n);
    cg_key_add(key, ctx->num_sms);
    cg_tune_cfg c{0, 0};
    if (cg_tune_lookup(key, &c)) return c.seg;
    cudaStream_t st = ctx->stream;
    const dim3 block(32, 8);
    const int nI = cg_div_up(v.nx, 32) * cg_div_up(v.ny, 8), nH = cg_div_up(v.nx, cgsia::kHCols) * cg_div_up(v.ny, 8);
    cudaMemsetAsync(words, 0, sizeof(cgsia::Words), st);
    sia_S_kernel<T><<<cg_div_up(v.nx + 2, 32) * cg_div_up(v.ny + 2, 8), block, 0, st>>>(v, Hb[1], 0);
    auto two = [&] {
        cudaError_t e = cg_launch(sia_D_kernel<T, false>, dim3(nI), block, 0, st, true, v, words, 0, (char*)nullptr);
        return e == cudaSuccess
                   ? cg_launch(sia_step_kernel<T, false>, dim3(nH), block, 0, st, true, v, words, 0, 0, 1, (char*)nullptr)
                   : e;
    };
    const StepBufs<T> f{Hb[0], Db[0], v.S[0], Hb[1], Db[1], v.S[1]};
    const std::vector<float> us = cgk::time_candidates(
        4, [&](int c) { return c == 0 ? two() : launch_whole_step(kStepRows[c - 1], v, f, words, 0, 0, st); }, st);
    for (int c = 0; cg_tune_verbose() && c < 4; ++c)
        std::fprintf(stderr, "sia step tune: %s, %d rows: %.1f us\n", c ? "one launch" : "two launches", c ? kStepRows[c - 1] : 8, us[c]);
    if (cgk::fastest(us) > 0) rows = kStepRows[cgk::fastest(us) - 1];
    cudaGetLastError();
    rows = std::max(rows, 0);
    cg_tune_store(key, cg_tune_cfg{rows, 0});
    return rows;
}

template <class T>
int run_t(cg_ctx* ctx, const cg_grid* g, const cg_field* H, const cg_field* B, const cg_field* q,
          const cg_sia_params* p, int nsteps, double* t_host, char* tape = nullptr) {
    // scratch: D and the two S buffers (H's padded layout), a second D and H where a step may be one
    // launch, and the words
    const size_t ab = cgsia::layout_bytes(*H, sizeof(T));
    int rc = CG_OK;
    bool whole = !tape && (cg_sia_step_rows_forced() > 0 || whole_step_fits<T>(ctx, g));
    char* base = whole ? static_cast<char*>(cg_scratch_optional(ctx, 1, 5 * ab + 256, "sia second buffers")) : nullptr;
    whole = base != nullptr;
    if (!whole) base = static_cast<char*>(cg_scratch(ctx, 1, 3 * ab + 256, &rc));
    if (rc) return rc;
    cgsia::Words* words = reinterpret_cast<cgsia::Words*>(base + (whole ? 5 : 3) * ab);
    cgsia::Member<T> v = cgsia::make_member<T>(*g, *H, *B, q, *p, base, base + ab, base + 2 * ab);
    const cgsia::TapeGeom tg = cgsia::tape_geom(*H, sizeof(T));
    v.tab = (long long)tg.abytes;
    v.orig = (long long)cg_origin_offset(*H);
    DF<T> Hb[2] = {v.H, v.H}, Db[2] = {v.D, v.D};
    if (whole) {
        Db[1].p = reinterpret_cast<T*>(base + 3 * ab) + v.orig;
        Hb[1].p = reinterpret_cast<T*>(base + 4 * ab) + v.orig;
    }
    const int rows = whole ? step_rows(ctx, g, H, v, Hb, Db, words) : 0;
    whole = rows > 0;
    const dim3 block(32, 8);
    const int nS = cg_div_up(v.nx + 2, 32) * cg_div_up(v.ny + 2, 8), nI = cg_div_up(v.nx, 32) * cg_div_up(v.ny, 8);
    const int nH = cg_div_up(v.nx, cgsia::kHCols) * cg_div_up(v.ny, 8);
    std::string key = "sia_run";
    cg_key_add(key, *g);
    cg_key_add(key, *H);
    cg_key_add(key, *B);
    cg_key_add(key, q[0]);
    cg_key_add(key, q[1]);
    cg_key_add(key, *p);
    cg_key_add(key, nsteps);
    cg_key_add(key, base);
    cg_key_add(key, tape);
    cg_key_add(key, rows);
    rc = cg_graph_run(ctx, key, [&](cudaStream_t st) {
        CG_CUDA(ctx, cudaMemsetAsync(words, 0, sizeof(cgsia::Words), st));
        // one launch per step: H alternates between the field and the scratch copy and ends in the field
        const int h0 = whole ? nsteps & 1 : 0;
        sia_S_kernel<T><<<nS, block, 0, st>>>(v, Hb[1], h0);
        CG_CHECK_LAUNCH(ctx);
        if (whole) CG_CUDA(ctx, cg_launch(sia_D_kernel<T, false>, dim3(nI), block, 0, st, true, v, words, 0, (char*)nullptr));
        for (int s = 0; s < nsteps; ++s) {
            if (whole) {
                const int a = s & 1, c = a ^ 1;
                const StepBufs<T> f{Hb[a ^ h0], Db[a], v.S[a], Hb[c ^ h0], Db[c], v.S[c]};
                CG_CUDA(ctx, launch_whole_step(rows, v, f, words, s % 3, s == nsteps - 1, st));
                continue;
            }
            char* sb = tape ? tape + 256 + (size_t)s * tg.step_bytes : nullptr;
            const int par = s & 1, last = s == nsteps - 1;
            CG_CUDA(ctx, tape ? cg_launch(sia_D_kernel<T, true>, dim3(nI), block, 0, st, s > 0, v, words, par, sb)
                              : cg_launch(sia_D_kernel<T, false>, dim3(nI), block, 0, st, s > 0, v, words, par, sb));
            CG_CUDA(ctx, tape ? cg_launch(sia_step_kernel<T, true>, dim3(nH), block, 0, st, true, v, words, par, last, 0, sb)
                              : cg_launch(sia_step_kernel<T, false>, dim3(nH), block, 0, st, true, v, words, par, last, 0, sb));
        }
        // the tangential points of bc! beyond the ghost layer (index n+2), which no step reads
        cg_bc bcs[3];
        sia_bcs(bcs, bcs + 2);
        const cg_field fs[3] = {q[0], q[1], *H};
        return cg_bc_apply_impl(ctx, g, 3, fs, bcs);
    });
    if (rc) return rc;
    if (t_host) {
        CG_CUDA(ctx, cudaMemcpyAsync(t_host, &words->t, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        CG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    }
    return CG_OK;
}

}  // namespace

extern "C" int cg_sia_update_q(cg_ctx* ctx, const cg_grid* grid, const cg_field* q, const cg_field* H,
                               const cg_field* B, const cg_sia_params* p, double* dmax_host) {
    int rc = check_sia(ctx, grid, H, B, q, p);
    if (rc) return rc;
    if (!q) return cg_fail(ctx, CG_ERR_ARG, "sia_update_q: q is NULL");
    cudaSetDevice(ctx->device);
    return H->dtype == CG_F64 ? update_q_t<double>(ctx, grid, q, H, B, p, dmax_host)
                              : update_q_t<float>(ctx, grid, q, H, B, p, dmax_host);
}

extern "C" int cg_sia_update_H(cg_ctx* ctx, const cg_grid* grid, const cg_field* H, const cg_field* q,
                               const cg_field* B, double dt, const cg_sia_params* p) {
    int rc = check_sia(ctx, grid, H, B, q, p);
    if (rc) return rc;
    if (!q) return cg_fail(ctx, CG_ERR_ARG, "sia_update_H: q is NULL");
    cudaSetDevice(ctx->device);
    return H->dtype == CG_F64 ? update_H_t<double>(ctx, grid, H, q, B, dt, p)
                              : update_H_t<float>(ctx, grid, H, q, B, dt, p);
}

extern "C" int cg_sia_tape_bytes(const cg_grid* grid, const cg_field* H, int nsteps, size_t* bytes) {
    if (!grid || !H || !bytes || nsteps < 0) return CG_ERR_ARG;
    if (grid->ndim != 2 || (H->dtype != CG_F32 && H->dtype != CG_F64)) return CG_ERR_ARG;
    const cgsia::TapeGeom tg = cgsia::tape_geom(*H, H->dtype == CG_F64 ? 8 : 4);
    *bytes = 256 + (size_t)nsteps * tg.step_bytes;
    return CG_OK;
}

extern "C" int cg_sia_run_taped(cg_ctx* ctx, const cg_grid* grid, const cg_field* H, const cg_field* B,
                                const cg_field* q, const cg_sia_params* p, int nsteps, void* tape, size_t tape_bytes,
                                double* t_host) {
    int rc = check_sia(ctx, grid, H, B, q, p);
    if (rc) return rc;
    if (!q) return cg_fail(ctx, CG_ERR_ARG, "sia_run_taped: q is NULL");
    if (nsteps < 1) return cg_fail(ctx, CG_ERR_ARG, "sia_run_taped: nsteps < 1");
    if (p->cfl <= 0 || p->dt_max <= 0) return cg_fail(ctx, CG_ERR_ARG, "sia_run_taped: cfl and dt_max must be > 0");
    size_t need = 0;
    cg_sia_tape_bytes(grid, H, nsteps, &need);
    if (!tape || tape_bytes < need)
        return cg_fail(ctx, CG_ERR_ARG, "sia_run_taped: the tape holds %zu bytes, %d steps need %zu", tape_bytes, nsteps, need);
    if (reinterpret_cast<uintptr_t>(tape) & 255) return cg_fail(ctx, CG_ERR_ARG, "sia_run_taped: the tape is not 256-byte aligned");
    cudaSetDevice(ctx->device);
    const size_t elem = H->dtype == CG_F64 ? 8 : 4;
    const cgsia::TapeGeom tg = cgsia::tape_geom(*H, elem);
    cgsia::TapeHeader hd;
    std::memset(&hd, 0, sizeof(hd));
    hd.magic = cgsia::kTapeMagic;
    hd.dtype = H->dtype;
    hd.nx = grid->n[0];
    hd.ny = grid->n[1];
    hd.nsteps = nsteps;
    hd.stride0 = H->stride[0];
    hd.stride1 = H->stride[1];
    hd.halo0 = H->halo[0];
    hd.halo1 = H->halo[1];
    hd.n0 = H->n[0];
    hd.n1 = H->n[1];
    hd.cnt = (long long)tg.cnt;
    hd.step_bytes = (long long)tg.step_bytes;
    hd.Gamma = p->Gamma;
    hd.As = p->As;
    hd.beta = p->beta;
    hd.ela = p->ela;
    hd.m_max = p->m_max;
    hd.cfl = p->cfl;
    hd.dt_max = p->dt_max;
    hd.n = p->n;
    CG_CUDA(ctx, cudaMemcpyAsync(tape, &hd, sizeof(hd), cudaMemcpyHostToDevice, ctx->stream));
    char* tp = static_cast<char*>(tape);
    return H->dtype == CG_F64 ? run_t<double>(ctx, grid, H, B, q, p, nsteps, t_host, tp)
                              : run_t<float>(ctx, grid, H, B, q, p, nsteps, t_host, tp);
}

extern "C" int cg_sia_run(cg_ctx* ctx, const cg_grid* grid, const cg_field* H, const cg_field* B, const cg_field* q,
                          const cg_sia_params* p, int nsteps, double* t_host) {
    int rc = check_sia(ctx, grid, H, B, q, p);
    if (rc) return rc;
    if (!q) return cg_fail(ctx, CG_ERR_ARG, "sia_run: q is NULL");
    if (nsteps < 0) return cg_fail(ctx, CG_ERR_ARG, "sia_run: nsteps < 0");
    if (p->cfl <= 0 || p->dt_max <= 0) return cg_fail(ctx, CG_ERR_ARG, "sia_run: cfl and dt_max must be > 0");
    cudaSetDevice(ctx->device);
    if (nsteps == 0) {
        if (t_host) *t_host = 0.0;
        return CG_OK;
    }
    return H->dtype == CG_F64 ? run_t<double>(ctx, grid, H, B, q, p, nsteps, t_host)
                              : run_t<float>(ctx, grid, H, B, q, p, nsteps, t_host);
}
