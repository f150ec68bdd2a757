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
__global__ void sia_S_kernel(const cgsia::Member<T> v) {
    cgsia::S_tile(v, blockIdx.x);
}
template <class T, bool TAPE>
__global__ void __launch_bounds__(256) sia_D_kernel(const cgsia::Member<T> v, cgsia::Words* w, int par, char* sb) {
    cg_dep_wait();
    cg_dep_release();
    cgsia::D_tile<T, TAPE>(v, w, blockIdx.x, par, sb);
}
template <class T, bool TAPE>
__global__ void __launch_bounds__(256) sia_step_kernel(const cgsia::Member<T> v, cgsia::Words* w, int par, int last, char* sb) {
    cg_dep_wait();
    cg_dep_release();
    cgsia::H_tile<T, TAPE, false>(v, w, blockIdx.x, par, last != 0, false, sb);
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

template <class T>
int run_t(cg_ctx* ctx, const cg_grid* g, const cg_field* H, const cg_field* B, const cg_field* q,
          const cg_sia_params* p, int nsteps, double* t_host, char* tape = nullptr) {
    // scratch: D and the two S buffers (H's padded layout) and the words
    const size_t ab = cgsia::layout_bytes(*H, sizeof(T));
    int rc = CG_OK;
    char* base = static_cast<char*>(cg_scratch(ctx, 1, 3 * ab + 256, &rc));
    if (rc) return rc;
    cgsia::Words* words = reinterpret_cast<cgsia::Words*>(base + 3 * ab);
    cgsia::Member<T> v = cgsia::make_member<T>(*g, *H, *B, q, *p, base, base + ab, base + 2 * ab);
    const cgsia::TapeGeom tg = cgsia::tape_geom(*H, sizeof(T));
    v.tab = (long long)tg.abytes;
    v.orig = (long long)cg_origin_offset(*H);
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
    rc = cg_graph_run(ctx, key, [&](cudaStream_t st) {
        CG_CUDA(ctx, cudaMemsetAsync(words, 0, sizeof(cgsia::Words), st));
        sia_S_kernel<T><<<nS, block, 0, st>>>(v);
        CG_CHECK_LAUNCH(ctx);
        for (int s = 0; s < nsteps; ++s) {
            char* sb = tape ? tape + 256 + (size_t)s * tg.step_bytes : nullptr;
            const int par = s & 1, last = s == nsteps - 1;
            CG_CUDA(ctx, tape ? cg_launch(sia_D_kernel<T, true>, dim3(nI), block, 0, st, s > 0, v, words, par, sb)
                              : cg_launch(sia_D_kernel<T, false>, dim3(nI), block, 0, st, s > 0, v, words, par, sb));
            CG_CUDA(ctx, tape ? cg_launch(sia_step_kernel<T, true>, dim3(nH), block, 0, st, true, v, words, par, last, sb)
                              : cg_launch(sia_step_kernel<T, false>, dim3(nH), block, 0, st, true, v, words, par, last, sb));
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
