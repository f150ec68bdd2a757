// cg_sia_ensemble.cu — an ensemble of independent shallow-ice solves of uneven grid sizes
// (examples/sia.jl:7-16,71-81 per member) advanced together. Every phase of a time step covers
// the tiles of all members (a per-member tile prefix table maps tiles to members), and the
// adaptive Δt of every member is computed on the device. The `nsteps` loop is one launch per
// phase, replayed from a CUDA graph. With CG_SIA_PERSISTENT=1 (and cooperative launch support)
// it is instead ONE persistent cooperative launch with grid barriers between the phases. Both
// forms give the same bits. The graph is the default: on GB300 the tiles are bound by the FP64
// pipe, so residency saves nothing, and a grid barrier costs more than a kernel boundary in a
// replayed graph (64 members of 128^2..1024^2: 1.89 vs 1.77 ms per step; of 32^2..128^2:
// 49 vs 43 us).
//
// A step is the two tile functions of cg_sia_kernels.cuh (the single-member run's too), with bc! folded
// into them.
#include <vector>

#include "cg_common.cuh"
#include "cg_sia_kernels.cuh"

void* cg_scratch(cg_ctx* ctx, int slot, size_t bytes, int* rc);

namespace {

using cgsia::Member;
using cgsia::Words;
using cgsia::bits_of;

// The block's member descriptor, copied once into shared memory (every thread of the block
// calls it before reading the member).
// The leading barrier lets a block that loops over tiles (the persistent kernel) call it once
// per tile: the previous tile's reads of the descriptor and of the block-max scratch are done.
template <class T>
__device__ __forceinline__ const Member<T>& member_of(const Member<T>* mem, int m) {
    __shared__ __align__(16) unsigned long long words[(sizeof(Member<T>) + 7) / 8];
    __syncthreads();
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(mem + m);
    for (int k = tid; k < (int)((sizeof(Member<T>) + 7) / 8); k += blockDim.x * blockDim.y) words[k] = src[k];
    __syncthreads();
    return *reinterpret_cast<const Member<T>*>(words);
}

// block -> (member, tile) through the inclusive prefix of per-member tile counts
__device__ __forceinline__ int find_member(const int* prefix, int nm, int blk) {
    int lo = 0, hi = nm - 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (prefix[mid] > blk) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// A tile function on the tile of block `blk`: its member's descriptor in shared memory, and the
// member's words. Neither the descriptors nor the prefix tables change within a run, so a kernel
// launched as a dependent one finds its member (a binary search of dependent loads, 1 to 2 us) while
// the kernel before it drains, and waits for it only then (DEP).
template <class T>
__device__ __forceinline__ void ens_S_tile(const Member<T>* mem, const int* prefix, int nm, int blk) {
    const int m = find_member(prefix, nm, blk);
    cgsia::S_tile(member_of(mem, m), blk - (m ? prefix[m - 1] : 0));
}
template <class T, bool TAPE, bool DEP>
__device__ __forceinline__ void ens_D_tile(const Member<T>* mem, const int* prefix, int nm, Words* w, int blk, int par, char* sb) {
    const int m = find_member(prefix, nm, blk);
    const Member<T>& v = member_of(mem, m);
    const int t = blk - (m ? prefix[m - 1] : 0);
    if (DEP) cg_dep_wait();
    cgsia::D_tile<T, TAPE>(v, w + m, t, par, sb);
}
template <class T, bool TAPE, bool DEP>
__device__ __forceinline__ void ens_H_tile(const Member<T>* mem, const int* prefix, int nm, Words* w, int blk, int par, bool last,
                                           bool dry, char* sb) {
    const int m = find_member(prefix, nm, blk);
    const Member<T>& v = member_of(mem, m);
    const int t = blk - (m ? prefix[m - 1] : 0);
    if (DEP) cg_dep_wait();
    cgsia::H_tile<T, TAPE, true>(v, w + m, t, par, last, dry, sb);
}

template <class T>
__global__ void ens_S_kernel(const Member<T>* mem, const int* prefix, int nm) {
    ens_S_tile(mem, prefix, nm, blockIdx.x);
}
template <class T, bool TAPE>
__global__ void ens_D_kernel(const Member<T>* mem, const int* prefix, int nm, Words* w, int par, char* sb) {
    cg_dep_release();
    ens_D_tile<T, TAPE, true>(mem, prefix, nm, w, blockIdx.x, par, sb);
}
template <class T, bool TAPE>
__global__ void ens_H_kernel(const Member<T>* mem, const int* prefix, int nm, Words* w, int par, int last, int dry, char* sb) {
    cg_dep_release();
    ens_H_tile<T, TAPE, true>(mem, prefix, nm, w, blockIdx.x, par, last != 0, dry != 0, sb);
}

// ---- one persistent launch for the whole run ------------------------------------------------
//
// The same tiles and arithmetic as the per-phase kernels: the resident blocks of a cooperative
// launch loop over each phase's tiles, with a grid barrier between the phases. Per step: D and
// the block maxima; barrier; Δt, the fluxes and the thickness; barrier. The barrier counts arrivals on one monotonic word. Its waits give up
// after a time limit (two seconds of the GPU's global timer unless the host sets another) and
// set a timeout flag: the kernel then returns, and the host reports the error. A cooperative
// launch keeps every block resident, so the waits end.
struct GridBar {
    unsigned long long arrived;  // arrivals since the launch: barrier k completes at (k + 1) x expect
    int timeout;
};

__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Barrier `k` (0, 1, ...) of the launch: one relaxed add per block, then a wait of at most
// `limit_ns` until `expect` blocks (the grid's size) have added. Nothing is reset, so the last
// block to arrive has no extra work.
__device__ __forceinline__ bool grid_barrier(GridBar* b, unsigned expect, unsigned long long limit_ns,
                                             unsigned long long& k) {
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        const unsigned long long target = (++k) * expect;
        __threadfence();
        atomicAdd(&b->arrived, 1ull);
        volatile unsigned long long* va = &b->arrived;
        const unsigned long long t0 = globaltimer_ns();
        while (*va < target) {
            if (globaltimer_ns() - t0 > limit_ns) {
                atomicExch(&b->timeout, 1);
                break;
            }
            __nanosleep(32);
        }
        __threadfence();
    }
    __syncthreads();
    return *(volatile int*)&b->timeout == 0;
}

template <class T>
__global__ void __launch_bounds__(256, 4) ens_persistent_kernel(const Member<T>* mem, const int* pI, const int* pH,
                                                             const int* pS, int nm, int totI, int totH, int totS,
                                                             Words* w, int nsteps, GridBar* bar, unsigned expect,
                                                             unsigned long long limit_ns) {
    const unsigned nb = gridDim.x;
    unsigned long long k = 0;
    for (int b = blockIdx.x; b < totS; b += nb) ens_S_tile(mem, pS, nm, b);
    if (!grid_barrier(bar, expect, limit_ns, k)) return;
    for (int s = 0; s < nsteps; ++s) {
        for (int b = blockIdx.x; b < totI; b += nb) ens_D_tile<T, false, false>(mem, pI, nm, w, b, s & 1, nullptr);
        if (!grid_barrier(bar, expect, limit_ns, k)) return;
        for (int b = blockIdx.x; b < totH; b += nb) ens_H_tile<T, false, false>(mem, pH, nm, w, b, s & 1, s == nsteps - 1, false, nullptr);
        if (!grid_barrier(bar, expect, limit_ns, k)) return;
    }
}

// ---- tape of a taped ensemble run ------------------------------------------------------------
//
// A 256-byte header, then per step one block holding every member's tape in turn, each in the
// single-member layout of cgsia (words, then kArrays arrays in the member's H layout).
struct EnsTape {
    std::vector<long long> toff, tab, orig;
    size_t step_bytes = 0;
};

inline EnsTape ens_tape_layout(int nm, const cg_sia_member* ms, size_t elem) {
    EnsTape e;
    e.toff.resize(nm);
    e.tab.resize(nm);
    e.orig.resize(nm);
    size_t off = 0;
    for (int m = 0; m < nm; ++m) {
        const cgsia::TapeGeom g = cgsia::tape_geom(ms[m].H, elem);
        e.toff[m] = (long long)off;
        e.tab[m] = (long long)g.abytes;
        e.orig[m] = (long long)cg_origin_offset(ms[m].H);
        off += g.step_bytes;
    }
    e.step_bytes = off;
    return e;
}

struct EnsTapeHeader {
    unsigned long long magic;
    int dtype, nm, nsteps, pad;
    unsigned long long step_bytes, hash;
};
constexpr unsigned long long kEnsTapeMagic = 0x31534e4541544953ull;  // "SIATENS1"

// FNV-1a over the members' layouts, grid spacings and parameters: a reverse sweep checks it
// against its own
inline unsigned long long ens_tape_hash(int nm, const cg_sia_member* ms, const cg_sia_params* ps) {
    unsigned long long h = 1469598103934665603ull;
    auto mix = [&](const void* p, size_t n) {
        const unsigned char* c = static_cast<const unsigned char*>(p);
        for (size_t k = 0; k < n; ++k) h = (h ^ c[k]) * 1099511628211ull;
    };
    for (int m = 0; m < nm; ++m) {
        const cg_field& H = ms[m].H;
        const long long lay[8] = {ms[m].grid.n[0], ms[m].grid.n[1], H.n[0], H.n[1], H.halo[0], H.halo[1],
                                  (long long)H.stride[0], (long long)H.stride[1]};
        mix(lay, sizeof(lay));
        const double pr[9] = {ps[m].Gamma,  ps[m].As,     ps[m].beta,
                              ps[m].ela,    ps[m].m_max,  ps[m].cfl,
                              ps[m].dt_max, ms[m].grid.inv_spacing[0], ms[m].grid.inv_spacing[1]};
        mix(pr, sizeof(pr));
        mix(&ps[m].n, sizeof(int));
    }
    return h;
}

template <class T>
int run_t(cg_ctx* ctx, int nm, const cg_sia_member* ms, const cg_sia_params* ps, int nsteps, double* t_host,
          char* tape = nullptr) {
    // scratch slot 3: [members][prefix I][prefix H][prefix S][words][barrier][D, S, S per member]
    size_t off = 0;
    const size_t mem_off = off;
    off += ((size_t)nm * sizeof(Member<T>) + 255) & ~(size_t)255;
    const size_t pI_off = off;
    off += ((size_t)nm * sizeof(int) + 255) & ~(size_t)255;
    const size_t pH_off = off;
    off += ((size_t)nm * sizeof(int) + 255) & ~(size_t)255;
    const size_t pS_off = off;
    off += ((size_t)nm * sizeof(int) + 255) & ~(size_t)255;
    const size_t w_off = off;
    off += ((size_t)nm * sizeof(Words) + 255) & ~(size_t)255;
    const size_t bar_off = off;
    off += 256;
    std::vector<size_t> d_off(nm);
    for (int m = 0; m < nm; ++m) {
        d_off[m] = off;
        off += 3 * cgsia::layout_bytes(ms[m].H, sizeof(T));
    }
    int rc = CG_OK;
    char* base = static_cast<char*>(cg_scratch(ctx, 3, off, &rc));
    if (rc) return rc;
    std::vector<Member<T>> hm(nm);
    std::vector<int> pI(nm), pH(nm), pS(nm);
    const EnsTape et = ens_tape_layout(nm, ms, sizeof(T));
    int totI = 0, totH = 0, totS = 0;
    Member<T>* dmem = reinterpret_cast<Member<T>*>(base + mem_off);
    int* dpI = reinterpret_cast<int*>(base + pI_off);
    int* dpH = reinterpret_cast<int*>(base + pH_off);
    int* dpS = reinterpret_cast<int*>(base + pS_off);
    Words* dw = reinterpret_cast<Words*>(base + w_off);
    // members and tile prefix tables for tiles of 32 x ty points, uploaded to the scratch
    auto layout = [&](int ty) -> int {
        totI = totH = totS = 0;
        for (int m = 0; m < nm; ++m) {
            const cg_sia_member& s = ms[m];
            const size_t ab = cgsia::layout_bytes(s.H, sizeof(T));
            char* sc = base + d_off[m];
            Member<T>& v = hm[m];
            v = cgsia::make_member<T>(s.grid, s.H, s.B, s.q, ps[m], sc, sc + ab, sc + 2 * ab);
            if (tape) {
                v.toff = et.toff[m];
                v.tab = et.tab[m];
                v.orig = et.orig[m];
            }
            totI += cg_div_up(v.nx, 32) * cg_div_up(v.ny, ty);
            totH += cg_div_up(v.nx, cgsia::kHCols) * cg_div_up(v.ny, ty);
            totS += cg_div_up(v.nx + 2, 32) * cg_div_up(v.ny + 2, ty);
            pI[m] = totI;
            pH[m] = totH;
            pS[m] = totS;
        }
        CG_CUDA(ctx, cudaMemcpyAsync(dmem, hm.data(), nm * sizeof(Member<T>), cudaMemcpyHostToDevice, ctx->stream));
        CG_CUDA(ctx, cudaMemcpyAsync(dpI, pI.data(), nm * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
        CG_CUDA(ctx, cudaMemcpyAsync(dpH, pH.data(), nm * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
        CG_CUDA(ctx, cudaMemcpyAsync(dpS, pS.data(), nm * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
        CG_CUDA(ctx, cudaMemsetAsync(dw, 0, nm * sizeof(Words), ctx->stream));
        // the host tables are read by the copies above before the next layout call rewrites them
        CG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        return CG_OK;
    };
    int coop = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device) != cudaSuccess) coop = 0;
    const bool persistent = coop && !tape && cg_sia_persistent_enabled();
    // tile height: 8 rows for the persistent kernel, else the forced or autotuned choice
    int ty = 8;
    if (!persistent) {
        const int forced = cg_sia_tile_rows_forced();
        if (forced) {
            ty = forced;
        } else if (cg_autotune_enabled()) {
            std::string tkey = "sia_ensemble_tiles";
            cg_key_add(tkey, (int)sizeof(T));
            cg_key_add(tkey, ctx->num_sms);
            for (int m = 0; m < nm; ++m) {
                cg_key_add(tkey, ms[m].grid.n[0]);
                cg_key_add(tkey, ms[m].grid.n[1]);
            }
            cg_tune_cfg tc{0, 0};
            if (cg_tune_lookup(tkey, &tc)) {
                ty = tc.variant;
            } else {
                // time one step for each tile height, its second kernel without its stores: the
                // thickness does not change (D and S = B + H are recomputed by the run, and the
                // words are cleared by the next layout call)
                float best = 1e30f;
                for (int cand : {4, 8, 16}) {
                    if ((rc = layout(cand))) return rc;
                    const dim3 bk(32, cand);
                    const float t = cgk::time_launches(
                        [&] {
                            ens_S_kernel<T><<<totS, bk, 0, ctx->stream>>>(dmem, dpS, nm);
                            ens_D_kernel<T, false><<<totI, bk, 0, ctx->stream>>>(dmem, dpI, nm, dw, 0, nullptr);
                            ens_H_kernel<T, false><<<totH, bk, 0, ctx->stream>>>(dmem, dpH, nm, dw, 0, 0, 1, nullptr);
                            return cudaGetLastError();
                        },
                        ctx->stream);
                    if (cg_tune_verbose())
                        std::fprintf(stderr, "sia ensemble tune (%d members): 32x%d tiles: %.1f us\n", nm, cand,
                                     t);
                    if (t >= 0.f && t < best) {
                        best = t;
                        ty = cand;
                    }
                }
                cudaGetLastError();
                cg_tune_store(tkey, cg_tune_cfg{0, ty});
            }
        }
    }
    if ((rc = layout(ty))) return rc;
    const dim3 block(32, ty);
    // cooperative-launch support and residency of the persistent kernel are queried per call on
    // this context's device (a process may hold contexts on different GPU models)
    if (persistent) {
        // the whole run in one cooperative launch of the resident blocks
        int bps = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, ens_persistent_kernel<T>, 256, 0) != cudaSuccess) bps = 0;
        if (bps < 1) return cg_fail(ctx, CG_ERR_CUDA, "sia_ensemble_run: the persistent kernel does not fit on an SM");
        GridBar* bar = reinterpret_cast<GridBar*>(base + bar_off);
        CG_CUDA(ctx, cudaMemsetAsync(bar, 0, sizeof(GridBar), ctx->stream));
        const Member<T>* cmem = dmem;
        const int *cpI = dpI, *cpH = dpH, *cpS = dpS;
        int anm = nm, atI = totI, atH = totH, atS = totS, ans = nsteps;
        const unsigned nblocks = (unsigned)(bps * ctx->num_sms);
        const cg_barrier_cfg bcfg = cg_sia_barrier_cfg();
        unsigned expect = nblocks + (unsigned)bcfg.withheld;
        unsigned long long limit_ns = bcfg.limit_ns;
        void* args[] = {&cmem, &cpI, &cpH, &cpS, &anm, &atI, &atH, &atS, &dw, &ans, &bar, &expect, &limit_ns};
        CG_CUDA(ctx, cudaLaunchCooperativeKernel((const void*)ens_persistent_kernel<T>, dim3(nblocks), block,
                                                 args, 0, ctx->stream));
        int timed_out = 0;
        CG_CUDA(ctx, cudaMemcpyAsync(&timed_out, &bar->timeout, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
        CG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (timed_out) return cg_fail(ctx, CG_ERR_TIMEOUT, "sia_ensemble_run: a grid barrier of the persistent kernel timed out");
    } else {
    std::string key = "sia_ensemble";
    cg_key_add(key, ty);
    cg_key_add(key, nm);
    cg_key_add(key, nsteps);
    cg_key_add(key, base);
    cg_key_add(key, tape);
    key.append(reinterpret_cast<const char*>(hm.data()), nm * sizeof(Member<T>));
    rc = cg_graph_run(ctx, key, [&](cudaStream_t st) {
        ens_S_kernel<T><<<totS, block, 0, st>>>(dmem, dpS, nm);
        for (int s = 0; s < nsteps; ++s) {
            const int par = s & 1, last = s == nsteps - 1;
            char* sb = tape ? tape + 256 + (size_t)s * et.step_bytes : nullptr;
            const Member<T>* cm = dmem;
            const int *ci = dpI, *ch = dpH;
            CG_CUDA(ctx, tape ? cg_launch(ens_D_kernel<T, true>, dim3(totI), block, 0, st, s > 0, cm, ci, nm, dw, par, sb)
                              : cg_launch(ens_D_kernel<T, false>, dim3(totI), block, 0, st, s > 0, cm, ci, nm, dw, par, sb));
            CG_CUDA(ctx, tape ? cg_launch(ens_H_kernel<T, true>, dim3(totH), block, 0, st, true, cm, ch, nm, dw, par, last, 0, sb)
                              : cg_launch(ens_H_kernel<T, false>, dim3(totH), block, 0, st, true, cm, ch, nm, dw, par, last, 0, sb));
            CG_CHECK_LAUNCH(ctx);
        }
        return (int)CG_OK;
    });
    if (rc) return rc;
    }
    if (t_host) {
        std::vector<Words> hw(nm);
        CG_CUDA(ctx, cudaMemcpyAsync(hw.data(), dw, nm * sizeof(Words), cudaMemcpyDeviceToHost, ctx->stream));
        CG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        for (int m = 0; m < nm; ++m) t_host[m] = hw[m].t;
    }
    return CG_OK;
}

// ---- reverse sweep over an ensemble tape ----------------------------------------------------
//
// The reverse step of cg_sia_adjoint_run applied to every member at once: per step, the cell
// kernel over all members' interior tiles and the gather kernel over all tiles, which also adds the
// dt term at each member's argmax cell. (A launch of its own for the sums of dJ/ddt took 5.9 us of a
// step's 45 us at 10 members of 64^2 to 224^2.)
template <class T>
struct AdjMember {
    DF<T> L, Wk, lo, pax, pay;  // lambda and work (in/out by turns), the step's scratch
    DF<double> aG, aE;          // per-cell sums over the sweep's steps of dJ/dGamma and dJ/dela
    T beta, idx, idy;
    int nx, ny;
    long long toff, tab, orig;
};

template <class T>
__device__ __forceinline__ const AdjMember<T>& adj_member_of(const AdjMember<T>* am, int m) {
    __shared__ __align__(16) unsigned long long words[(sizeof(AdjMember<T>) + 7) / 8];
    __syncthreads();
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(am + m);
    for (int k = tid; k < (int)((sizeof(AdjMember<T>) + 7) / 8); k += blockDim.x * blockDim.y) words[k] = src[k];
    __syncthreads();
    return *reinterpret_cast<const AdjMember<T>*>(words);
}

template <class T>
__device__ __forceinline__ DF<T> adj_tape(const AdjMember<T>& v, const char* sb, int k) {
    DF<T> a = v.L;
    a.p = reinterpret_cast<T*>(const_cast<char*>(sb) + v.toff + 256 + (long long)k * v.tab) + v.orig;
    return a;
}

template <class T>
__device__ __forceinline__ DF<unsigned char> adj_flags(const AdjMember<T>& v, const char* sb) {
    DF<unsigned char> a;
    a.p = reinterpret_cast<unsigned char*>(const_cast<char*>(sb) + v.toff + 256 + (long long)cgsia::kFL * v.tab) + v.orig;
    a.s1 = v.L.s1;
    a.s2 = v.L.s2;
    return a;
}

template <class T>
__device__ __forceinline__ T ens_mu(const DF<unsigned char>& fl, const DF<T>& lam, int i, int j) {
    return (fl(i, j, 0) & 1) ? lam(i, j, 0) : T(0);
}

// Cell tiles of the reverse step: 31 owned columns x 8 rows. Every face term is computed once
// and used by both its cells: lane l computes the lower x face of its cell and lane l - 1 takes
// it as its upper face (shuffle); row r computes its lower y face and row r - 1 takes it
// through shared memory (the top row computes the face above it). Lane 31 only supplies the
// face of lane 30. Each cell sums its face terms in the order lower x, upper x, lower y,
// upper y, as a cell that evaluates all four itself does.
constexpr int kCW = 31;

template <class T>
__global__ void __launch_bounds__(256) ens_adj_cell_kernel(const AdjMember<T>* am, const int* prefix, int nm,
                                                           const char* sb, int parity, double* part) {
    using namespace cgsia;
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ T fdy[8][32], fsy[8][32], kc[4];
    __shared__ double sd[8][32];
    cg_dep_release();
    const int blk = blockIdx.x;
    const int m = find_member(prefix, nm, blk);
    const AdjMember<T>& v = adj_member_of(am, m);
    const int t = blk - (m ? prefix[m - 1] : 0);
    const int tx = (v.nx + kCW - 1) / kCW;
    const int lane = threadIdx.x, row = threadIdx.y;
    const int i = (t % tx) * kCW + lane + 1;
    const int j = (t / tx) * 8 + row + 1;
    const bool in = i <= v.nx && j <= v.ny;
    const bool own = in && lane < kCW;
    const DF<T> lam = parity ? v.Wk : v.L;
    const DF<unsigned char> FL = adj_flags(v, sb);
    const DF<T> D = adj_tape(v, sb, kD);
    const TapeWords* w = reinterpret_cast<const TapeWords*>(sb + v.toff);
    // the step's constants, once per block: dt beta, 1 + dt beta, and per dimension -dt idx/2 and idx
    if (lane < 4 && row == 0) {
        const T dt = (T)w->dt, dtb = dt * v.beta;
        kc[lane] = lane == 0 ? dtb : lane == 1 ? T(1) + dtb : -T(0.5) * (dt * (lane == 2 ? v.idx : v.idy));
    }
    // the tape does not change within a sweep: its values load while the kernel before this one
    // drains, and only lambda waits for it
    T dc = T(0), gx = T(0), gy = T(0), dl = T(0), dd = T(0), cdh = T(0), cex = T(0), cey = T(0), cgf = T(0), cw = T(0);
    unsigned char flc = 0, fll = 0, fld = 0;
    if (in) {
        dc = D(i, j, 0);
        flc = FL(i, j, 0);
        if (i >= 2) {
            dl = D(i - 1, j, 0);
            fll = FL(i - 1, j, 0);
            gx = adj_tape(v, sb, kGX)(i, j, 0);
        }
        if (j >= 2) {
            dd = D(i, j - 1, 0);
            fld = FL(i, j - 1, 0);
            gy = adj_tape(v, sb, kGY)(i, j, 0);
        }
        if (own) {
            cdh = adj_tape(v, sb, kDH)(i, j, 0);
            cex = adj_tape(v, sb, kEX)(i, j, 0);
            cey = adj_tape(v, sb, kEY)(i, j, 0);
            cgf = adj_tape(v, sb, kGF)(i, j, 0);
            cw = adj_tape(v, sb, kW)(i, j, 0);
        }
    }
    __syncthreads();
    cg_dep_wait();
    const T muc = flc & 1 ? lam(i, j, 0) : T(0);
    // the lower x face (face i, cells i-1 and i) and the lower y face (face j): with p = -dt idx/2
    // (mu_upper - mu_lower), dJ/dD of both cells gains p g and dJ/dS of them -/+ (D_l + D_u) p idx
    T tDx = T(0), tSx = T(0), tDy = T(0), tSy = T(0);
    if (in && i >= 2) {
        const T px = kc[2] * (muc - (fll & 1 ? lam(i - 1, j, 0) : T(0)));
        tDx = px * gx;
        tSx = (dl + dc) * (px * -v.idx);
    }
    if (in && j >= 2) {
        const T py = kc[3] * (muc - (fld & 1 ? lam(i, j - 1, 0) : T(0)));
        tDy = py * gy;
        tSy = (dd + dc) * (py * -v.idy);
    }
    fdy[row][lane] = tDy;
    fsy[row][lane] = tSy;
    T tDu = T(0), tSu = T(0);
    if (row == 7 && in && j + 1 <= v.ny) {  // the face above the tile
        const T py = kc[3] * (ens_mu(FL, lam, i, j + 1) - muc);
        tDu = py * adj_tape(v, sb, kGY)(i, j + 1, 0);
        tSu = (dc + D(i, j + 1, 0)) * (py * -v.idy);
    }
    const T tDr = __shfl_down_sync(FULL, tDx, 1), tSr = __shfl_down_sync(FULL, tSx, 1);
    __syncthreads();
    if (row < 7) {
        tDu = fdy[row + 1][lane];
        tSu = fsy[row + 1][lane];
    }
    double sdt = 0.0;
    if (own) {
        T pD = T(0), pS = T(0);
        if (i >= 2) {
            pD += tDx;
            pS += -tSx;
        }
        if (i + 1 <= v.nx) {
            pD += tDr;
            pS += tSr;
        }
        if (j >= 2) {
            pD += tDy;
            pS += -tSy;
        }
        if (j + 1 <= v.ny) {
            pD += tDu;
            pS += tSu;
        }
        // the mass balance's direct terms: d H'/d H = 1 + dt beta and d H'/d ela = -dt beta
        // where it is not capped (the step's constants, once per thread)
        const bool mM = (flc & 2) != 0;
        v.lo(i, j, 0) = fma(pD, cdh, mM ? muc * kc[1] : muc) + pS;
        v.pax(i, j, 0) = pD * cex;
        v.pay(i, j, 0) = pD * cey;
        sdt = (double)(muc * cw);
        v.aG(i, j, 0) += (double)(pD * cgf);
        if (mM) v.aE(i, j, 0) -= (double)(muc * kc[0]);
    }
    // the tile's sum of dJ/ddt in a fixed order: down the rows in one warp, then across its lanes
    // (a shuffle tree in every warp would cost each five FP64 instructions)
    sd[row][lane] = sdt;
    __syncthreads();
    if (row == 0) {
        double x = sd[0][lane];
#pragma unroll
        for (int r = 1; r < 8; ++r) x += sd[r][lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(FULL, x, o);
        if (lane == 0) part[blk] = x;
    }
}

// End of the sweep: per 32 x 8 tile, the sums of the per-cell dJ/dGamma and dJ/dela arrays,
// then (one block per member) their ordered sums into acc[2m], acc[2m + 1].
template <class T>
__global__ void __launch_bounds__(256) ens_adj_tile_sums_kernel(const AdjMember<T>* am, const int* prefix, int nm,
                                                                double* part, int ntot) {
    const int blk = blockIdx.x;
    const int m = find_member(prefix, nm, blk);
    const AdjMember<T>& v = adj_member_of(am, m);
    const int t = blk - (m ? prefix[m - 1] : 0);
    const int tx = (v.nx + 31) / 32;
    const int i = (t % tx) * 32 + threadIdx.x + 1;
    const int j = (t / tx) * 8 + threadIdx.y + 1;
    const bool in = i <= v.nx && j <= v.ny;
    const double g = cgsia::block_sum(in ? v.aG(i, j, 0) : 0.0);
    const double e = cgsia::block_sum(in ? v.aE(i, j, 0) : 0.0);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        part[blk] = g;
        part[ntot + blk] = e;
    }
}

__global__ void __launch_bounds__(1024) ens_adj_final_kernel(const int* prefix, const double* part, int ntot, double* acc) {
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ double red[2][32];
    const int m = blockIdx.x;
    const int b0 = m ? prefix[m - 1] : 0, b1 = prefix[m];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double x[2] = {0.0, 0.0};
    for (int b = b0 + tid; b < b1; b += blockDim.x)
        for (int k = 0; k < 2; ++k) x[k] += part[(size_t)k * ntot + b];
    for (int k = 0; k < 2; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x[k] += __shfl_xor_sync(FULL, x[k], o);
        if (lane == 0) red[k][warp] = x[k];
    }
    __syncthreads();
    if (warp != 0) return;
    for (int k = 0; k < 2; ++k) {
        double y = lane < (int)(blockDim.x >> 5) ? red[k][lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(FULL, y, o);
        if (lane == 0) acc[2 * m + k] = y;
    }
}

// lambda_n of every member from lo and the neighbours' pax, pay (the ghost cells' terms folded
// into the interior cells they copy); parity 0 writes Wk, 1 writes L. copy: L = Wk instead.
//
// The dt term (when dt was not capped) adds pD dD/dh, pD dD/dax, pD dD/day to lo, pax, pay of the one
// cell where D attains its maximum, with pD = -dJ/ddt dt/Dmax, and pD dD/dGamma to its dJ/dGamma sum.
// Only the tiles that read that cell need dJ/ddt: they sum the member's tile partials of the cell
// kernel (cprefix its tile prefix) in a fixed order and add the terms as they read; the tile that owns
// the cell updates the dJ/dGamma sum.
template <class T>
__global__ void __launch_bounds__(256) ens_adj_out_kernel(const AdjMember<T>* am, const int* prefix, const int* cprefix, int nm,
                                                          const char* sb, const double* part, int parity, int copy) {
    using namespace cgsia;
    __shared__ double red[8];
    cg_dep_release();
    const int blk = blockIdx.x;
    const int m = find_member(prefix, nm, blk);
    const AdjMember<T>& v = adj_member_of(am, m);
    const int t = blk - (m ? prefix[m - 1] : 0);
    const int tx = (v.nx + 31) / 32;
    const int it = (t % tx) * 32 + 1, jt = (t / tx) * 8 + 1;
    const int i = it + threadIdx.x, j = jt + threadIdx.y;
    int ai = -9, aj = -9;  // the argmax cell, where it matters to this tile
    double pd = 0.0;
    const TapeWords* w = reinterpret_cast<const TapeWords*>(sb + v.toff);
    bool near = false;
    if (!copy && w->capped == 0.0 && w->arg != ~0ull) {
        const int ci = (int)(w->arg % (unsigned long long)(v.nx + 2)), cj = (int)(w->arg / (unsigned long long)(v.nx + 2));
        near = ci >= it - 1 && ci <= it + 32 && cj >= jt - 1 && cj <= jt + 8;
        if (near) {
            ai = ci;
            aj = cj;
        }
    }
    cg_dep_wait();
    if (near) {  // the whole block
        const int b0 = m ? cprefix[m - 1] : 0, b1 = cprefix[m];
        const int tid = threadIdx.x + 32 * threadIdx.y;
        double x = 0.0;
        for (int b = b0 + tid; b < b1; b += 256) x += part[b];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (threadIdx.x == 0) red[threadIdx.y] = x;
        __syncthreads();
        x = 0.0;
#pragma unroll
        for (int r = 0; r < 8; ++r) x += red[r];
        const unsigned long long bb = w->dmax;
        const double dmax = sizeof(T) == 8 ? __longlong_as_double((long long)bb) : (double)__int_as_float((int)(unsigned)bb);
        pd = (double)(T)(-x * w->dt / dmax);
    }
    if (i > v.nx || j > v.ny) return;
    if (copy) {
        v.L(i, j, 0) = v.Wk(i, j, 0);
        return;
    }
    const T hx = T(0.5) * v.idx, hy = T(0.5) * v.idy, pD = (T)pd;
    auto at = [&](const DF<T>& f, int k, int a, int b) {  // f's value, with the dt term's at the argmax cell
        const T x = f(a, b, 0);
        return a == ai && b == aj ? x + pD * adj_tape(v, sb, k)(a, b, 0) : x;
    };
    auto PX = [&](int a, int b) { return (a >= 1 && a <= v.nx) ? at(v.pax, kEX, a, b) : T(0); };
    auto PY = [&](int a, int b) { return (b >= 1 && b <= v.ny) ? at(v.pay, kEY, a, b) : T(0); };
    T r = at(v.lo, kDH, i, j) + hx * (PX(i - 1, j) - PX(i + 1, j)) + hy * (PY(i, j - 1) - PY(i, j + 1));
    if (i == 1) r += -hx * PX(1, j);
    if (i == v.nx) r += hx * PX(v.nx, j);
    if (j == 1) r += -hy * PY(i, 1);
    if (j == v.ny) r += hy * PY(i, v.ny);
    if (i == ai && j == aj) v.aG(i, j, 0) += (double)(pD * adj_tape(v, sb, kGF)(i, j, 0));
    (parity ? v.L : v.Wk)(i, j, 0) = r;
}

template <class T>
int adjoint_run_t(cg_ctx* ctx, int nm, const cg_sia_member* ms, const cg_sia_params* ps, int N, const char* tape,
                  const cg_field* lam, const cg_field* work, double* dJ) {
    const EnsTape et = ens_tape_layout(nm, ms, sizeof(T));
    std::vector<int> pI(nm), pC(nm);
    std::vector<size_t> aoff(nm);
    int totI = 0, totC = 0;
    // scratch slot 7: [members][prefix][partials 3 x tiles][acc 2 x members][lo, pax, pay per member]
    size_t off = 0;
    const size_t mem_off = off;
    off += ((size_t)nm * sizeof(AdjMember<T>) + 255) & ~(size_t)255;
    const size_t p_off = off;
    off += ((size_t)nm * sizeof(int) + 255) & ~(size_t)255;
    const size_t pc_off = off;
    off += ((size_t)nm * sizeof(int) + 255) & ~(size_t)255;
    for (int m = 0; m < nm; ++m) {
        totI += cg_div_up(ms[m].grid.n[0], 32) * cg_div_up(ms[m].grid.n[1], 8);
        totC += cg_div_up(ms[m].grid.n[0], kCW) * cg_div_up(ms[m].grid.n[1], 8);
        pI[m] = totI;
        pC[m] = totC;
    }
    const size_t part_off = off;
    off += ((size_t)std::max(totC, 2 * totI) * sizeof(double) + 255) & ~(size_t)255;
    const size_t acc_off = off;
    off += ((size_t)2 * nm * sizeof(double) + 255) & ~(size_t)255;
    for (int m = 0; m < nm; ++m) {
        aoff[m] = off;
        off += 3 * (size_t)et.tab[m];
    }
    // the per-cell FP64 sums of every member, in one region (zeroed once per sweep)
    std::vector<size_t> doff(nm);
    const size_t sums_off = off;
    for (int m = 0; m < nm; ++m) {
        doff[m] = off;
        off += 2 * cgsia::tape_geom(ms[m].H, sizeof(double)).abytes;
    }
    const size_t sums_bytes = off - sums_off;
    int rc = CG_OK;
    char* base = static_cast<char*>(cg_scratch(ctx, 7, off, &rc));
    if (rc) return rc;
    std::vector<AdjMember<T>> hm(nm);
    for (int m = 0; m < nm; ++m) {
        AdjMember<T>& v = hm[m];
        std::memset(&v, 0, sizeof(v));
        v.L = cg_view<T>(lam[m]);
        v.Wk = cg_view<T>(work[m]);
        DF<T>* sc[3] = {&v.lo, &v.pax, &v.pay};
        for (int a = 0; a < 3; ++a) {
            *sc[a] = v.L;
            sc[a]->p = reinterpret_cast<T*>(base + aoff[m] + (size_t)a * et.tab[m]) + cg_origin_offset(lam[m]);
        }
        const size_t dab = cgsia::tape_geom(ms[m].H, sizeof(double)).abytes;
        DF<double>* sd[2] = {&v.aG, &v.aE};
        for (int a = 0; a < 2; ++a) {
            sd[a]->p = reinterpret_cast<double*>(base + doff[m] + (size_t)a * dab) + cg_origin_offset(lam[m]);
            sd[a]->s1 = v.L.s1;
            sd[a]->s2 = v.L.s2;
        }
        v.beta = (T)ps[m].beta;
        v.idx = (T)ms[m].grid.inv_spacing[0];
        v.idy = (T)ms[m].grid.inv_spacing[1];
        v.nx = ms[m].grid.n[0];
        v.ny = ms[m].grid.n[1];
        v.toff = et.toff[m];
        v.tab = et.tab[m];
        v.orig = et.orig[m];
    }
    AdjMember<T>* dmem = reinterpret_cast<AdjMember<T>*>(base + mem_off);
    int* dp = reinterpret_cast<int*>(base + p_off);
    int* dpc = reinterpret_cast<int*>(base + pc_off);
    double* part = reinterpret_cast<double*>(base + part_off);
    double* acc = reinterpret_cast<double*>(base + acc_off);
    CG_CUDA(ctx, cudaMemcpyAsync(dmem, hm.data(), nm * sizeof(AdjMember<T>), cudaMemcpyHostToDevice, ctx->stream));
    CG_CUDA(ctx, cudaMemcpyAsync(dp, pI.data(), nm * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
    CG_CUDA(ctx, cudaMemcpyAsync(dpc, pC.data(), nm * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
    std::string key = "sia_ensemble_adjoint";
    cg_key_add(key, nm);
    cg_key_add(key, N);
    cg_key_add(key, base);
    cg_key_add(key, tape);
    key.append(reinterpret_cast<const char*>(hm.data()), nm * sizeof(AdjMember<T>));
    const dim3 block(32, 8);
    rc = cg_graph_run(ctx, key, [&](cudaStream_t st) {
        CG_CUDA(ctx, cudaMemsetAsync(base + sums_off, 0, sums_bytes, st));
        for (int r = 0; r < N; ++r) {
            const char* sb = tape + 256 + (size_t)(N - 1 - r) * et.step_bytes;
            const AdjMember<T>* cm = dmem;
            const int *ci = dp, *cc = dpc;
            const double* cpart = part;
            CG_CUDA(ctx, cg_launch(ens_adj_cell_kernel<T>, dim3(totC), block, 0, st, r > 0, cm, cc, nm, sb, r & 1, part));
            CG_CUDA(ctx, cg_launch(ens_adj_out_kernel<T>, dim3(totI), block, 0, st, true, cm, ci, cc, nm, sb, cpart, r & 1, 0));
        }
        if (N & 1) ens_adj_out_kernel<T><<<totI, block, 0, st>>>(dmem, dp, dpc, nm, tape + 256, part, 0, 1);
        ens_adj_tile_sums_kernel<T><<<totI, block, 0, st>>>(dmem, dp, nm, part, totI);
        ens_adj_final_kernel<<<nm, 1024, 0, st>>>(dp, part, totI, acc);
        CG_CHECK_LAUNCH(ctx);
        return (int)CG_OK;
    });
    if (rc) return rc;
    std::vector<double> h(2 * (size_t)nm);
    CG_CUDA(ctx, cudaMemcpyAsync(h.data(), acc, h.size() * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    CG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (dJ)
        for (size_t k = 0; k < h.size(); ++k) dJ[k] += h[k];
    return CG_OK;
}

int check_ensemble(cg_ctx* ctx, int nmembers, const cg_sia_member* members, const cg_sia_params* params,
                   const char* who) {
    if (!ctx) return cg_fail(nullptr, CG_ERR_ARG, "%s: ctx is NULL", who);
    if (nmembers < 1 || !members || !params) return cg_fail(ctx, CG_ERR_ARG, "%s: no members", who);
    const int dtype = members[0].H.dtype;
    for (int m = 0; m < nmembers; ++m) {
        const cg_sia_member& s = members[m];
        int rc = cg_check_grid(ctx, &s.grid);
        if (rc) return rc;
        if (s.grid.ndim != 2) return cg_fail(ctx, CG_ERR_UNSUPPORTED, "%s: member %d is not 2D", who, m);
        if ((rc = cg_check_field(ctx, &s.grid, s.H, dtype, 0, "H"))) return rc;
        if ((rc = cg_check_field(ctx, &s.grid, s.B, dtype, 0, "B"))) return rc;
        if ((rc = cg_check_field(ctx, &s.grid, s.q[0], dtype, 1, "q.x"))) return rc;
        if ((rc = cg_check_field(ctx, &s.grid, s.q[1], dtype, 2, "q.y"))) return rc;
        if (params[m].n < 1 || params[m].n > 16 || params[m].cfl <= 0 || params[m].dt_max <= 0)
            return cg_fail(ctx, CG_ERR_ARG, "%s: bad parameters for member %d", who, m);
    }
    return CG_OK;
}

}  // namespace

// The reverse sweep over `nsteps` taped steps whose blocks start at tape + 256, every member in
// each launch; cg_sia_adjoint_run calls it with one member (a single-member tape has the same
// step blocks). Only the members' grids and H layouts are read.
int cg_sia_reverse_impl(cg_ctx* ctx, int nm, const cg_sia_member* ms, const cg_sia_params* ps, int nsteps,
                        const char* tape, const cg_field* lam, const cg_field* work, double* dJ) {
    return ms[0].H.dtype == CG_F64 ? adjoint_run_t<double>(ctx, nm, ms, ps, nsteps, tape, lam, work, dJ)
                                   : adjoint_run_t<float>(ctx, nm, ms, ps, nsteps, tape, lam, work, dJ);
}

extern "C" int cg_sia_ensemble_run(cg_ctx* ctx, int nmembers, const cg_sia_member* members,
                                   const cg_sia_params* params, int nsteps, double* t_host) {
    int rc = check_ensemble(ctx, nmembers, members, params, "sia_ensemble_run");
    if (rc) return rc;
    if (nsteps < 0) return cg_fail(ctx, CG_ERR_ARG, "sia_ensemble_run: nsteps < 0");
    cudaSetDevice(ctx->device);
    if (nsteps == 0) {
        if (t_host)
            for (int m = 0; m < nmembers; ++m) t_host[m] = 0.0;
        return CG_OK;
    }
    return members[0].H.dtype == CG_F64 ? run_t<double>(ctx, nmembers, members, params, nsteps, t_host)
                                        : run_t<float>(ctx, nmembers, members, params, nsteps, t_host);
}

extern "C" int cg_sia_ensemble_tape_bytes(int nmembers, const cg_sia_member* members, int nsteps, size_t* bytes) {
    if (nmembers < 1 || !members || !bytes || nsteps < 0) return CG_ERR_ARG;
    const int dt = members[0].H.dtype;
    if (dt != CG_F32 && dt != CG_F64) return CG_ERR_ARG;
    const EnsTape et = ens_tape_layout(nmembers, members, dt == CG_F64 ? 8 : 4);
    *bytes = 256 + (size_t)nsteps * et.step_bytes;
    return CG_OK;
}

extern "C" int cg_sia_ensemble_run_taped(cg_ctx* ctx, int nmembers, const cg_sia_member* members,
                                         const cg_sia_params* params, int nsteps, void* tape, size_t tape_bytes,
                                         double* t_host) {
    int rc = check_ensemble(ctx, nmembers, members, params, "sia_ensemble_run_taped");
    if (rc) return rc;
    if (nsteps < 1) return cg_fail(ctx, CG_ERR_ARG, "sia_ensemble_run_taped: nsteps < 1");
    size_t need = 0;
    cg_sia_ensemble_tape_bytes(nmembers, members, nsteps, &need);
    if (!tape || tape_bytes < need)
        return cg_fail(ctx, CG_ERR_ARG, "sia_ensemble_run_taped: the tape holds %zu bytes, %d steps need %zu", tape_bytes,
                       nsteps, need);
    if (reinterpret_cast<uintptr_t>(tape) & 255)
        return cg_fail(ctx, CG_ERR_ARG, "sia_ensemble_run_taped: the tape is not 256-byte aligned");
    cudaSetDevice(ctx->device);
    const int dt = members[0].H.dtype;
    EnsTapeHeader hd;
    std::memset(&hd, 0, sizeof(hd));
    hd.magic = kEnsTapeMagic;
    hd.dtype = dt;
    hd.nm = nmembers;
    hd.nsteps = nsteps;
    hd.step_bytes = ens_tape_layout(nmembers, members, dt == CG_F64 ? 8 : 4).step_bytes;
    hd.hash = ens_tape_hash(nmembers, members, params);
    CG_CUDA(ctx, cudaMemcpyAsync(tape, &hd, sizeof(hd), cudaMemcpyHostToDevice, ctx->stream));
    char* tp = static_cast<char*>(tape);
    return dt == CG_F64 ? run_t<double>(ctx, nmembers, members, params, nsteps, t_host, tp)
                        : run_t<float>(ctx, nmembers, members, params, nsteps, t_host, tp);
}

extern "C" int cg_sia_ensemble_adjoint_run(cg_ctx* ctx, int nmembers, const cg_sia_member* members,
                                           const cg_sia_params* params, const void* tape, size_t tape_bytes,
                                           const cg_field* lam, const cg_field* work, double* dJ) {
    int rc = check_ensemble(ctx, nmembers, members, params, "sia_ensemble_adjoint_run");
    if (rc) return rc;
    if (!tape || !lam || !work) return cg_fail(ctx, CG_ERR_ARG, "sia_ensemble_adjoint_run: NULL argument");
    const int dt = members[0].H.dtype;
    for (int m = 0; m < nmembers; ++m) {
        const cg_field& H = members[m].H;
        if ((rc = cg_check_field(ctx, &members[m].grid, lam[m], dt, 0, "lambda"))) return rc;
        if ((rc = cg_check_field(ctx, &members[m].grid, work[m], dt, 0, "work"))) return rc;
        if (lam[m].data == work[m].data) return cg_fail(ctx, CG_ERR_ARG, "sia_ensemble_adjoint_run: lambda and work alias (member %d)", m);
        for (const cg_field* f : {&lam[m], &work[m]})
            if (f->stride[1] != H.stride[1] || f->halo[0] != H.halo[0] || f->halo[1] != H.halo[1] || f->n[0] != H.n[0] ||
                f->n[1] != H.n[1])
                return cg_fail(ctx, CG_ERR_ARG, "sia_ensemble_adjoint_run: lambda and work need H's layout (member %d)", m);
    }
    if (tape_bytes < sizeof(EnsTapeHeader)) return cg_fail(ctx, CG_ERR_ARG, "sia_ensemble_adjoint_run: the tape is too small");
    cudaSetDevice(ctx->device);
    EnsTapeHeader hd;
    CG_CUDA(ctx, cudaMemcpyAsync(&hd, tape, sizeof(hd), cudaMemcpyDeviceToHost, ctx->stream));
    CG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (hd.magic != kEnsTapeMagic)
        return cg_fail(ctx, CG_ERR_ARG, "sia_ensemble_adjoint_run: no tape of cg_sia_ensemble_run_taped at this address");
    const EnsTape et = ens_tape_layout(nmembers, members, dt == CG_F64 ? 8 : 4);
    if (hd.dtype != dt || hd.nm != nmembers || hd.step_bytes != et.step_bytes ||
        hd.hash != ens_tape_hash(nmembers, members, params))
        return cg_fail(ctx, CG_ERR_ARG, "sia_ensemble_adjoint_run: the tape was recorded for other members or parameters");
    if (hd.nsteps < 1 || tape_bytes < 256 + (size_t)hd.nsteps * et.step_bytes)
        return cg_fail(ctx, CG_ERR_ARG, "sia_ensemble_adjoint_run: the tape is shorter than its %d steps", hd.nsteps);
    return cg_sia_reverse_impl(ctx, nmembers, members, params, hd.nsteps, static_cast<const char*>(tape), lam, work, dJ);
}
