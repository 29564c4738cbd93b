// adjoint.cu - discrete adjoint (reverse mode) of the FP64 RK3 step, with checkpointing.
//
// The reference has no adjoint; this is the derivative of exactly the map the forward kernels
// compute (src/step.cpp:114-257 with FLUXES, BCON and the dt reduction).  A trajectory of N
// steps is recorded by the ordinary forward path, keeping the state every K steps on the
// device and every step's limit minima (32 bytes).  The backward sweep walks the segments in
// reverse: it recomputes the states of a segment from its checkpoint, each step's third stage
// writing straight into the next state's buffer, then for each step (last first) recomputes the
// three stages once more - now also storing the right-hand sides F_s (stage kernels with EMIT) -
// and runs
//
//   for s = 2, 1, 0:   lambda_Y   = BCON^T lambda_X_{s+1}                       (adj_bcon_kernel)
//                      lambda_F_s = gam_s dt lambda_Y + zeta_{s+1} dt lambda_Y(s+1)  (adj_pass1_kernel)
//                      lambda_X_s = F'(X_s)^T lambda_F_s + lambda_Y             (adj_pass2_kernel)
//   lambda_dt = sum_s <F_s, lambda_F_s> / dt                                    (deterministic sum)
//   lambda_X_0 += lambda_dt * sff * d(limit)/dX at the cell that set dt (dt_argmin_kernel, adj_dt_apply)
//
// Each recomputed step is compared bit for bit with the recorded state that follows it; a
// mismatch (a non-reproducible forward) is reported as R3D_ENUMERIC instead of a silently wrong
// gradient.  Limits: FP64 only; a time-independent top boundary (tc == 0), since the plume
// relaxation clock would otherwise couple every step to the sum of all earlier dt.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "adjoint_cell.cuh"
#include "r3d_gpu_impl.hpp"
#include "stage_common.cuh"
#include "tma.cuh"

using namespace r3db;
using r3dk::AdjArgs;

namespace {

constexpr int BX = 32, BY = 8;       // cells per block of the passes
constexpr int kPassBlocks = 2;      // blocks of pass 2 resident per SM
constexpr int kDotBlocks = 32;        // partial sums of the dt dot products

struct AdjScalars {
    unsigned long long wkey[4];  // the step's four limit minima (ordered keys), saved before dt
    unsigned long long argmin;   // smallest cell index holding the winning limit
    unsigned long long mismatch; // recompute vs recorded state: differing values
    double part[kDotBlocks];     // partial sums of <F_s, lambda_F_s> over the three stages
};

__device__ __forceinline__ int block_linear() {
    return blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
}

// Deterministic block sum of v (all threads call); thread 0 stores it to out[block].
__device__ void block_sum_store(double v, double* out) {
    __shared__ double red[BX * BY / 32];
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    if (tid == 0) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x * blockDim.y) / 32; ++w) s += red[w];
        out[block_linear()] = s;
    }
}

struct FieldPtrs {
    const double* x[r3dk::kMaxFields];
    double* lam[r3dk::kMaxFields];
};

__global__ void __launch_bounds__(BX* BY) adj_bcon_kernel(r3dk::Geometry g, r3dk::Physics ph,
                                                           r3dk::Boundary bd, FieldPtrs A, int nf) {
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    if (i > g.npx || j > g.npy) return;
    // one side per thread, or (npz < 6: the two sides share planes) both in turn
    const int z = blockIdx.z;
    r3dk::adj_bcon_column(g, ph, bd, A.x, A.lam, nf, z, i, j);
    if (gridDim.z == 1) r3dk::adj_bcon_column(g, ph, bd, A.x, A.lam, nf, 1, i, j);
}

// Bound by the latency of the gathers, so by how many loads the warps of an SM keep in flight: two
// 256-thread blocks per SM (three for hydro pass 1) with every load of a cell free to go out at once.
// B200, us per stage: 128x128x128 hydro pass 1 145 (two blocks: 173), pass 2 160 (three blocks, 80
// registers and spills: 210); 64x64x128 MHD pass 1 65 (three: 77), pass 2 91 (three: 116).  Both
// together, with every Lambda stored and lambda_F folded separately: 577 and 222.
template <bool MHD>
__global__ void __launch_bounds__(BX* BY, MHD ? 2 : 3) adj_pass1_kernel(const __grid_constant__ AdjArgs A, double* dots) {
    const int i = 1 + blockIdx.x * BX + threadIdx.x;
    const int j = 1 + blockIdx.y * BY + threadIdx.y;
    const int k = 1 + blockIdx.z;
    double dot = 0.0;
    if (i <= A.g.npx && j <= A.g.npy) dot = r3dk::adj_pass1_cell<MHD>(A, i, j, k);
    block_sum_store(dot, dots);
}

// The cell of this thread in the block `ahead` places later in launch order (-1: none): with as many
// places as blocks run at once, its lines are in L2 by the time that block gathers them.  B200, 128x128x128
// hydro pass 2 181 -> 160 us (twice as far ahead 181); a whole step of the sweep 1674 -> 1616 us, at
// 200x200x100 3137 -> 2975.  Not with MHD (64x64x128 pass 2 82 -> 91 us, a step 820 -> 837; 126x126x128 2577
// -> 2553) nor in pass 1, whose gathers are fewer (5% slower).
__device__ __forceinline__ int cell_ahead(const r3dk::Geometry& g, int ahead) {
    const int b = block_linear() + ahead, row = b / (int)gridDim.x;
    const int i = 1 + (b % (int)gridDim.x) * BX + threadIdx.x;
    const int j = 1 + (row % (int)gridDim.y) * BY + threadIdx.y, k = 1 + row / (int)gridDim.y;
    if (i > g.npx || j > g.npy || k > g.npz) return -1;
    return k * (int)g.plane + j * (int)g.pitch + i;
}

template <bool MHD>
__global__ void __launch_bounds__(BX* BY, 2) adj_pass2_kernel(const __grid_constant__ AdjArgs A) {
    if constexpr (!MHD) {
        if (const int n = cell_ahead(A.g, A.ahead); n >= 0) {
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                r3dk::prefetch_l2(A.x + f * A.fe + n);
                r3dk::prefetch_l2(A.a + f * A.fe + n);
                r3dk::prefetch_l2(A.out + f * A.fe + n);
                r3dk::prefetch_l2(A.lam + f * A.fe + n);
            }
#pragma unroll
            for (int q = 0; q < r3dk::kMidHydro; ++q) r3dk::prefetch_l2(A.mid + q * A.fe + n);
        }
    }
    const int i = 1 + blockIdx.x * BX + threadIdx.x;
    const int j = 1 + blockIdx.y * BY + threadIdx.y;
    const int k = 1 + blockIdx.z;
    if (i <= A.g.npx && j <= A.g.npy) r3dk::adj_pass2_cell<MHD>(A, i, j, k);
}

// Interior cells of lam from a cotangent in the reference layout: the cell's own entry and those of
// its periodic ghost images, added in (j, i) order.
__global__ void __launch_bounds__(BX* BY) adj_seed_fold_kernel(r3dk::Geometry g, const double* seed, double* lam) {
    const int i = 1 + blockIdx.x * BX + threadIdx.x;
    const int j = 1 + blockIdx.y * BY + threadIdx.y;
    const int k = 1 + blockIdx.z;
    if (i > g.npx || j > g.npy) return;
    const int64_t nx = g.npx + 2, ny = g.npy + 2;
    auto row = [&](int64_t jj) {  // entries at i = 0 (the image of npx), i, npx + 1 (of 1)
        const double* s = seed + (k * ny + jj) * nx;
        double v = i == g.npx ? s[0] + s[i] : s[i];
        if (i == 1) v += s[g.npx + 1];
        return v;
    };
    double v = j == g.npy ? row(0) + row(j) : row(j);
    if (j == 1) v += row(g.npy + 1);
    lam[(int64_t)k * g.plane + (int64_t)j * g.pitch + i] = v;
}

// Start of a recomputed step: its dt from the limit minima it started with (as step_begin_kernel
// forms it), and bounds under which the third stage skips every cell's limits - the recompute
// needs none.
__global__ void adj_begin_kernel(r3dk::Physics ph, const unsigned long long* key, r3dk::Scalars* sc, AdjScalars* aux) {
    for (int q = 0; q < 4; ++q) aux->wkey[q] = key[q];
    aux->argmin = ~0ull;
    double m;
    r3dk::winning_limit(aux->wkey, ph.lmag, m);
    sc->dt = ph.sff * m;
    sc->bnd = r3dk::DtBounds{};
    sc->bnd.u = __int_as_float(0x7f800000);
}

// The n dot-product partials of the step's passes to kDotBlocks sums, each over a fixed share in
// a fixed order (deterministic).  One block summing all of them took 41 us at 128x128x128.
constexpr int kSumThreads = 256;
__global__ void __launch_bounds__(kSumThreads) adj_dots_kernel(const double* dots, int n, AdjScalars* aux) {
    __shared__ double red[kSumThreads];
    double s = 0.0;
    for (int b = blockIdx.x * kSumThreads + threadIdx.x; b < n; b += kDotBlocks * kSumThreads) s += dots[b];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kSumThreads / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) aux->part[blockIdx.x] = red[0];
}

// lambda_X_0 += lambda_dt * sff * d(limit)/dX at the cell that set dt.
__global__ void adj_dt_apply_kernel(r3dk::Geometry g, r3dk::Physics ph, r3dk::Lines L, const double* x, double* lam,
                                    int64_t fe, int nf, const r3dk::Scalars* sc, const AdjScalars* aux) {
    const unsigned long long an = aux->argmin;
    double mstar;
    const int term = r3dk::winning_limit(aux->wkey, ph.lmag, mstar);
    // sff == 0: dt is 0 whatever the state (and nothing to divide the sums by)
    if (term == 3 || an == ~0ull || ph.sff == 0.0) return;
    double lam_dt = 0.0;
    for (int b = 0; b < kDotBlocks; ++b) lam_dt += aux->part[b];
    lam_dt /= sc->dt;
    const int n = (int)an;
    const int k = n / (int)g.plane, j = (n % (int)g.plane) / (int)g.pitch, i = n % (int)g.pitch;
    const double dxy = (L.ddy[j] < L.ddx[i]) ? L.ddy[j] : L.ddx[i];
    const double dd = (L.ddz[k] < dxy) ? L.ddz[k] : dxy;
    double xv[r3dk::kMaxFields], gv[r3dk::kMaxFields];
    for (int f = 0; f < nf; ++f) xv[f] = x[f * fe + n];
    r3dk::adj_dt_cell(ph, term, dd, L.rkapa[k], xv, nf, lam_dt * ph.sff, gv);
    for (int f = 0; f < nf; ++f) lam[f * fe + n] += gv[f];
}

// Count interior values that differ (bitwise) between a recomputed and a recorded state.
__global__ void __launch_bounds__(BX* BY) adj_compare_kernel(r3dk::Geometry g, const double* a, const double* b,
                                                              int64_t field_elems, int nf, AdjScalars* aux) {
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    const int k = 1 + blockIdx.z;
    if (i > g.npx || j > g.npy) return;
    const int64_t n = (int64_t)k * g.plane + (int64_t)j * g.pitch + i;
    unsigned long long bad = 0;
    for (int f = 0; f < nf; ++f)
        bad += (__double_as_longlong(a[f * field_elems + n]) != __double_as_longlong(b[f * field_elems + n]));
    if (bad) atomicAdd(&aux->mismatch, bad);
}

}  // namespace

namespace r3dg {

// A state is nf fields stored back to back, field f at base + f*field_elems (padded layout).
struct Adjoint {
    int nf = 5;
    int64_t field_elems = 0;
    double* S[4] = {};              // X_1 .. X_3 of the step being recomputed; S[0]: the start state of adjoint_step
    double* Zb = nullptr;           // accumulator Z (nf fields)
    double* F[3] = {};              // F_0 .. F_2 (nf fields each)
    double* lam[2] = {};            // lambda_X / lambda_Y of a stage and of the one after it
    int cur = 0;                    // lam[cur] is the current one
    double* a = nullptr;            // lambda_F (nf fields)
    double* mid = nullptr;          // pass-1 arrays
    int nmid = 0;
    double* dots = nullptr;
    int nblocks = 0;
    r3dk::Scalars* asc = nullptr;   // scalars of the recompute
    unsigned int* edge_cnt = nullptr;  // the recompute's own BCON counters: a stage it abandons leaves the
                                       // forward steps' ones alone
    AdjScalars* aux = nullptr;
    AdjScalars* haux = nullptr;     // pinned mirror
    std::vector<double*> ckpt;      // recorded checkpoints
    std::vector<double*> seg;       // states of the segment being reversed (its first is the checkpoint)
    unsigned long long* lim = nullptr;  // recorded limit minima, four keys per step
    int lim_steps = 0;
    int nsteps = 0, every = 0;
    bool recorded = false;
    int64_t bytes = 0;
};

namespace impl {

double* dalloc(Adjoint* A, size_t n) {
    double* p = nullptr;
    cuda_ok(cudaMalloc(&p, n * sizeof(double)), "cudaMalloc(adjoint)");
    A->bytes += (int64_t)(n * sizeof(double));
    return p;
}

double* state_field(double* base, const Adjoint* A, int f) { return base + (size_t)f * A->field_elems; }

dim3 cell_grid(const r3d_gpu* g) {
    return dim3((g->geo.npx + BX - 1) / BX, (g->geo.npy + BY - 1) / BY, (unsigned)g->geo.npz);
}

Adjoint* workspace(r3d_gpu* g) {
    if (g->adj) return g->adj;
    if (g->fp32) throw Error(R3D_EINVAL, "the adjoint is available for precision fp64 only");
    if (g->p.id != 0) throw Error(R3D_EINVAL, "the adjoint does not include the density diffusion (ID)");
    if (g->p.itcon == 2 || g->p.itcon == 3)
        throw Error(R3D_EINVAL, "the adjoint covers itcon 0, 1 and 4 (not the embedded heat loss or a free top T)");
    if (g->nloc != g->p.npz || g->halo) throw Error(R3D_EINVAL, "the adjoint needs the whole domain on one handle");
    if (g->p.tp != 0.0 && g->p.tc != 0.0 && (g->p.itcon == 0 || g->p.itcon == 1))
        throw Error(R3D_EINVAL, "the adjoint needs a time-independent top boundary (tc == 0)");
    if (g->geo.npz > 65535) throw Error(R3D_EINVAL, "the adjoint supports npz <= 65535");
    auto A = new Adjoint();
    try {
        A->nf = g->nfields;
        A->field_elems = g->geo.plane * (g->geo.npz + 2);
        const size_t st = (size_t)A->nf * A->field_elems;
        for (int s = 1; s < 4; ++s) A->S[s] = dalloc(A, st);
        A->Zb = dalloc(A, st);
        for (int s = 0; s < 3; ++s) A->F[s] = dalloc(A, st);
        for (int s = 0; s < 2; ++s) A->lam[s] = dalloc(A, st);
        A->a = dalloc(A, st);
        A->nmid = A->nf == 8 ? r3dk::kMidMax : r3dk::kMidHydro;
        A->mid = dalloc(A, (size_t)A->nmid * A->field_elems);
        const dim3 gr = cell_grid(g);
        A->nblocks = (int)(gr.x * gr.y * gr.z);
        A->dots = dalloc(A, (size_t)3 * A->nblocks);
        cuda_ok(cudaMalloc(&A->asc, sizeof(r3dk::Scalars)), "cudaMalloc(adjoint scalars)");
        if (g->tail) {
            cuda_ok(cudaMalloc(&A->edge_cnt, g->edge_bytes), "cudaMalloc(counters)");
            A->bytes += (int64_t)g->edge_bytes;
        }
        cuda_ok(cudaMalloc(&A->aux, sizeof(AdjScalars)), "cudaMalloc(adjoint scalars)");
        cuda_ok(cudaMallocHost(&A->haux, sizeof(AdjScalars)), "cudaMallocHost");
        // the z ghost planes of a and mid are read (with weight 0) and stay zero; keep every
        // other buffer defined as well
        for (double* p : {A->Zb, A->F[0], A->F[1], A->F[2], A->lam[0], A->lam[1], A->a})
            cuda_ok(cudaMemsetAsync(p, 0, st * sizeof(double), g->stream), "cudaMemset");
        cuda_ok(cudaMemsetAsync(A->mid, 0, (size_t)A->nmid * A->field_elems * sizeof(double), g->stream),
                "cudaMemset");
    } catch (...) {
        g->adj = A;
        adjoint_free(g);
        throw;
    }
    g->adj = A;
    return A;
}

void free_states(std::vector<double*>& v) {
    for (double* p : v) cudaFree(p);
    v.clear();
}

// n state buffers, keeping those that are there (the excess is given back).
void resize_states(const Adjoint* A, std::vector<double*>& v, int n) {
    while ((int)v.size() > n) {
        cudaFree(v.back());
        v.pop_back();
    }
    while ((int)v.size() < n) {
        double* p = nullptr;
        cuda_ok(cudaMalloc(&p, (size_t)A->nf * A->field_elems * sizeof(double)), "cudaMalloc(states)");
        v.push_back(p);
    }
}

// Copy the simulation's current state (separate field arrays) into a contiguous state buffer.
void save_current(r3d_gpu* g, Adjoint* A, double* dst) {
    const size_t nb = (size_t)A->field_elems * sizeof(double);
    for (int f = 0; f < A->nf; ++f)
        cuda_ok(cudaMemcpyAsync(state_field(dst, A, f), g->X[g->cur][f], nb, cudaMemcpyDeviceToDevice, g->stream),
                "checkpoint copy");
}

// The z ghost planes of a state buffer: constants that every stage reads and none writes.
void copy_ghost_planes(r3d_gpu* g, Adjoint* A, double* dst, const double* src) {
    const size_t pitch = (size_t)A->field_elems * sizeof(double), width = (size_t)g->geo.plane * sizeof(double);
    for (int64_t k : {(int64_t)0, (int64_t)g->geo.npz + 1})
        cuda_ok(cudaMemcpy2DAsync(dst + k * g->geo.plane, pitch, src + k * g->geo.plane, pitch, width, A->nf,
                                  cudaMemcpyDeviceToDevice, g->stream),
                "ghost planes");
}

r3dk::FieldSet stage_fields(const Adjoint* A, int s, const double* in, double* out) {
    r3dk::FieldSet fs{};
    for (int f = 0; f < A->nf; ++f) {
        fs.xin[f] = in + (size_t)f * A->field_elems;
        fs.xout[f] = out + (size_t)f * A->field_elems;
        fs.z[f] = state_field(A->Zb, A, f);
        fs.f[f] = state_field(A->F[s], A, f);
    }
    return fs;
}

r3dk::StageMaps state_maps(const r3d_gpu* g, const Adjoint* A, const double* base) {
    r3dk::StageMaps m{};
    unsigned bx = 0, by = 0;
    r3dk::stage_fp64_box(g->geo.tile_rows, &bx, &by);
    for (int f = 0; f < A->nf; ++f)
        m.m[f] = field_map(const_cast<double*>(base) + (size_t)f * A->field_elems, g->d.nx, g->d.ny, g->d.nz,
                           g->geo.pitch, g->geo.plane, bx, by, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, sizeof(double));
    return m;
}

// Start of a sweep: nothing an earlier one left (an error flag, counters of a stage that was abandoned
// mid-way, differing values) counts in this one.
void begin_sweep(r3d_gpu* g, Adjoint* A) {
    cuda_ok(cudaMemsetAsync(A->asc, 0, sizeof(r3dk::Scalars), g->stream), "cudaMemset");
    cuda_ok(cudaMemcpyAsync(&A->asc->tx_extra, &g->dsc->tx_extra, sizeof(g->dsc->tx_extra), cudaMemcpyDeviceToDevice,
                            g->stream),
            "tx_extra");
    cuda_ok(cudaMemsetAsync(A->aux, 0, sizeof(AdjScalars), g->stream), "cudaMemset");
    if (A->edge_cnt) cuda_ok(cudaMemsetAsync(A->edge_cnt, 0, g->edge_bytes, g->stream), "cudaMemset");
}

// One forward step from the state src with the dt of the limit minima key, through S[1] and S[2]
// into dst; emit: F[0..2] stored.
void recompute_step(r3d_gpu* g, Adjoint* A, const unsigned long long* key, const double* src, double* dst, bool emit) {
    adj_begin_kernel<<<1, 1, 0, g->stream>>>(g->ph, key, A->asc, A->aux);
    cuda_ok(cudaGetLastError(), "adjoint begin");
    const double* in[3] = {src, A->S[1], A->S[2]};
    double* out[3] = {A->S[1], A->S[2], dst};
    for (int s = 0; s < 3; ++s) {
        r3dk::FieldSet fs = stage_fields(A, s, in[s], out[s]);
        // (the EMIT stages have no single-wave form)
        r3dk::StageTail tail = emit ? r3dk::StageTail{} : stage_tail(g, r3dk::kTailBcon);
        tail.edge_cnt = A->edge_cnt;
        cuda_ok(r3dk::launch_stage_fp64(s, state_maps(g, A, in[s]), g->geo, g->ph, g->lines, fs, A->asc, g->depth, tail,
                                        g->stream, emit),
                "adjoint recompute stage");
        if (!tail.flags)
            cuda_ok(r3dk::launch_bcon(g->geo, g->ph, g->lines, g->bnd, fs, A->asc, 0, g->stream), "adjoint bcon");
    }
}

// Reverse the step from src whose intermediates recompute_step left in S[1..3] and F: lam[cur]
// holds the adjoint of X_3 on entry and of X_0 = src on exit.
void reverse_step(r3d_gpu* g, Adjoint* A, const double* src) {
    const double* X[4] = {src, A->S[1], A->S[2], A->S[3]};
    const dim3 blk(BX, BY, 1), cg = cell_grid(g);
    const dim3 cols(cg.x, cg.y, g->geo.npz < 6 ? 1 : 2);
    const bool mhd = A->nf == 8;
    for (int s = 2; s >= 0; --s) {
        double* lam = A->lam[A->cur];
        double* other = A->lam[1 - A->cur];  // lambda_Y of stage s + 1, then lambda_X of stage s
        FieldPtrs fp{};
        for (int f = 0; f < A->nf; ++f) {
            fp.x[f] = X[s + 1] + (size_t)f * A->field_elems;
            fp.lam[f] = state_field(lam, A, f);
        }
        adj_bcon_kernel<<<cols, blk, 0, g->stream>>>(g->geo, g->ph, g->bnd, fp, A->nf);
        cuda_ok(cudaGetLastError(), "adj_bcon");
        AdjArgs p{};
        p.g = g->geo;
        p.ph = g->ph;
        p.L = g->lines;
        p.fe = A->field_elems;
        p.x = X[s];
        p.lam = lam;
        p.lprev = s < 2 ? other : nullptr;
        p.a = A->a;
        p.mid = A->mid;
        p.out = other;
        p.F = A->F[s];
        p.sc = A->asc;
        p.ahead = g->num_sms * kPassBlocks;
        p.gam = g->ph.gam[s];
        p.zeta = s < 2 ? g->ph.zeta[s + 1] : 0.0;
        double* dots = A->dots + (size_t)s * A->nblocks;
        if (mhd) adj_pass1_kernel<true><<<cg, blk, 0, g->stream>>>(p, dots);
        else adj_pass1_kernel<false><<<cg, blk, 0, g->stream>>>(p, dots);
        cuda_ok(cudaGetLastError(), "adj_pass1");
        if (mhd) adj_pass2_kernel<true><<<cg, blk, 0, g->stream>>>(p);
        else adj_pass2_kernel<false><<<cg, blk, 0, g->stream>>>(p);
        cuda_ok(cudaGetLastError(), "adj_pass2");
        A->cur = 1 - A->cur;
    }
    adj_dots_kernel<<<kDotBlocks, kSumThreads, 0, g->stream>>>(A->dots, 3 * A->nblocks, A->aux);
    cuda_ok(cudaGetLastError(), "adj_dots");
    cuda_ok(r3dk::launch_dt_argmin(g->geo, g->ph, g->lines, stage_fields(A, 0, src, A->S[1]), A->aux->wkey,
                                   &A->aux->argmin, g->stream),
            "adj_argmin");
    adj_dt_apply_kernel<<<1, 1, 0, g->stream>>>(g->geo, g->ph, g->lines, src, A->lam[A->cur], A->field_elems, A->nf,
                                                A->asc, A->aux);
    cuda_ok(cudaGetLastError(), "adj_dt_apply");
}

void compare_states(r3d_gpu* g, Adjoint* A, const double* a, const double* b) {
    const dim3 blk(BX, BY, 1), cg = cell_grid(g);
    adj_compare_kernel<<<cg, blk, 0, g->stream>>>(g->geo, a, b, A->field_elems, A->nf, A->aux);
    cuda_ok(cudaGetLastError(), "adj_compare");
}

// Host cotangent (NX*NY*NZ per field, ghosts included) -> lam: x/y ghost entries are added to
// the interior cells they image, z ghost planes are constants and dropped.  The fields pass through
// F[0], which holds nothing between steps.
void upload_seed(r3d_gpu* g, Adjoint* A, const double* const* seed) {
    for (int f = 0; f < A->nf; ++f)
        if (!seed[f]) throw std::invalid_argument("null seed field");
    const int64_t NX = g->d.nx, NY = g->d.ny, NZ = g->d.nz;
    const dim3 blk(BX, BY, 1), gr = cell_grid(g);
    for (int f = 0; f < A->nf; ++f) {
        double* stage = state_field(A->F[0], A, f);
        from_host(g, stage, seed[f], (size_t)(NX * NY * NZ) * sizeof(double), "seed upload");
        adj_seed_fold_kernel<<<gr, blk, 0, g->stream>>>(g->geo, stage, state_field(A->lam[A->cur], A, f));
        cuda_ok(cudaGetLastError(), "adj_seed_fold");
    }
    cuda_ok(cudaStreamSynchronize(g->stream), "seed upload");  // the caller's arrays are free again
}

void download_grad(r3d_gpu* g, Adjoint* A, double* const* grad) {
    for (int f = 0; f < A->nf; ++f)
        if (!grad[f]) throw std::invalid_argument("null gradient field");
    // lam's ghost cells are zero: nothing writes them
    for (int f = 0; f < A->nf; ++f)
        to_host(g, grad[f], state_field(A->lam[A->cur], A, f), g->geo.pitch * sizeof(double), g->d.nx * sizeof(double),
                g->d.ny * g->d.nz, "gradient download");
    cuda_ok(cudaStreamSynchronize(g->stream), "gradient download");
}

void check_aux(r3d_gpu* g, Adjoint* A) {
    cuda_ok(cudaMemcpyAsync(A->haux, A->aux, sizeof(AdjScalars), cudaMemcpyDeviceToHost, g->stream), "adjoint scalars");
    r3dk::Scalars sc{};
    cuda_ok(cudaMemcpyAsync(&sc, A->asc, sizeof(sc), cudaMemcpyDeviceToHost, g->stream), "adjoint scalars");
    cuda_ok(cudaStreamSynchronize(g->stream), "adjoint");
    if (sc.err != r3dk::kErrNone)
        throw Error(R3D_ECUDA, "a recompute stage kernel abandoned a bounded TMA wait; the gradient is invalid");
    if (A->haux->mismatch)
        throw Error(R3D_ENUMERIC, "adjoint recompute diverged from the recorded trajectory (" +
                                      std::to_string(A->haux->mismatch) + " values)");
}

}  // namespace impl

void adjoint_free(r3d_gpu* g) {
    Adjoint* A = g->adj;
    if (!A) return;
    for (double* p : A->S) cudaFree(p);
    cudaFree(A->lim);
    cudaFree(A->Zb);
    for (double* p : A->F) cudaFree(p);
    for (double* p : A->lam) cudaFree(p);
    cudaFree(A->a);
    cudaFree(A->mid);
    cudaFree(A->dots);
    cudaFree(A->asc);
    cudaFree(A->edge_cnt);
    cudaFree(A->aux);
    if (A->haux) cudaFreeHost(A->haux);
    impl::free_states(A->ckpt);
    impl::free_states(A->seg);
    delete A;
    g->adj = nullptr;
}

}  // namespace r3dg

using namespace r3dg;
using namespace r3dg::impl;

extern "C" {

int r3d_gpu_adjoint_record(r3d_gpu* g, int nsteps, int checkpoint_every, r3d_scalars* sc) {
    return guarded([&] {
        if (!g) throw std::invalid_argument("null handle");
        if (!g->uploaded) throw Error(R3D_ESTATE, "record before upload");
        if (nsteps < 1 || checkpoint_every < 1) throw std::invalid_argument("nsteps and checkpoint_every must be >= 1");
        DeviceGuard dg(g->device);
        Range r("r3d.adjoint_record");
        Adjoint* A = workspace(g);
        A->recorded = false;
        // checkpoints at steps 0, K, 2K, .. and the final state (compared against in backward)
        const int nck = (nsteps + checkpoint_every - 1) / checkpoint_every + 1;
        resize_states(A, A->ckpt, nck);
        if (nsteps > A->lim_steps) {
            cudaFree(A->lim);
            A->lim = nullptr;
            A->lim_steps = 0;
            cuda_ok(cudaMalloc(&A->lim, (size_t)nsteps * sizeof(g->dsc->wmin)), "cudaMalloc(limits)");
            A->lim_steps = nsteps;
        }
        Timer tm{g, false, nullptr};
        int launches = 0, stage_launches = 0;
        for (int n = 0; n < nsteps; ++n) {
            if (n % checkpoint_every == 0) save_current(g, A, A->ckpt[n / checkpoint_every]);
            cuda_ok(cudaMemcpyAsync(A->lim + 4 * n, g->dsc->wmin, sizeof(g->dsc->wmin), cudaMemcpyDeviceToDevice,
                                    g->stream),
                    "record limits");
            enqueue_step(g, 3, tm, launches, stage_launches);
        }
        save_current(g, A, A->ckpt.back());
        pull_scalars(g, sc);
        A->nsteps = nsteps;
        A->every = checkpoint_every;
        A->recorded = true;
    });
}

int r3d_gpu_adjoint_backward(r3d_gpu* g, const double* const* seed, double* const* grad) {
    return guarded([&] {
        if (!g || !seed || !grad) throw std::invalid_argument("null argument");
        if (!g->adj || !g->adj->recorded) throw Error(R3D_ESTATE, "no recorded trajectory (call r3d_gpu_adjoint_record)");
        DeviceGuard dg(g->device);
        Range r("r3d.adjoint_backward");
        Adjoint* A = g->adj;
        const int K = A->every, N = A->nsteps;
        // states 1 .. K-1 of a segment; the recompute buffers take the constant z ghost planes of X_0
        resize_states(A, A->seg, std::min(K, N) - 1);
        for (int s = 1; s < 4; ++s) copy_ghost_planes(g, A, A->S[s], A->ckpt[0]);
        for (double* p : A->seg) copy_ghost_planes(g, A, p, A->ckpt[0]);
        begin_sweep(g, A);
        upload_seed(g, A, seed);
        const double* final_state = A->ckpt.back();  // the recorded final state
        {
            const int nseg = (N + K - 1) / K;
            for (int sg = nseg - 1; sg >= 0; --sg) {
                const int s0 = sg * K, len = std::min(K, N - s0);
                auto state = [&](int s) -> double* { return s == 0 ? A->ckpt[sg] : A->seg[s - 1]; };
                for (int s = 1; s < len; ++s)
                    recompute_step(g, A, A->lim + 4 * (s0 + s - 1), state(s - 1), state(s), false);
                for (int s = len - 1; s >= 0; --s) {
                    recompute_step(g, A, A->lim + 4 * (s0 + s), state(s), A->S[3], true);
                    const double* next = s + 1 < len ? state(s + 1) : (sg + 1 < nseg ? A->ckpt[sg + 1] : final_state);
                    compare_states(g, A, A->S[3], next);
                    reverse_step(g, A, state(s));
                }
                check_aux(g, A);
            }
            download_grad(g, A, grad);
        }
    });
}

int r3d_gpu_adjoint_step(r3d_gpu* g, const double* const* seed, double* const* grad) {
    return guarded([&] {
        if (!g || !seed || !grad) throw std::invalid_argument("null argument");
        if (!g->uploaded) throw Error(R3D_ESTATE, "adjoint before upload");
        DeviceGuard dg(g->device);
        Adjoint* A = workspace(g);
        if (!A->S[0]) A->S[0] = dalloc(A, (size_t)A->nf * A->field_elems);
        save_current(g, A, A->S[0]);
        for (int s = 1; s < 4; ++s) copy_ghost_planes(g, A, A->S[s], A->S[0]);
        begin_sweep(g, A);
        upload_seed(g, A, seed);
        cuda_ok(r3dk::launch_reset_reduction(A->asc, g->stream), "adjoint reset");
        cuda_ok(r3dk::launch_dt_full(g->geo, g->ph, g->lines, stage_fields(A, 0, A->S[0], A->S[1]), A->asc, g->stream),
                "adjoint dt_full");
        recompute_step(g, A, A->asc->wmin, A->S[0], A->S[3], true);
        reverse_step(g, A, A->S[0]);
        check_aux(g, A);
        download_grad(g, A, grad);
    });
}

int r3d_gpu_adjoint_memory(const r3d_gpu* g, int64_t* bytes) {
    return guarded([&] {
        if (!g || !bytes) throw std::invalid_argument("null argument");
        const Adjoint* A = g->adj;
        int64_t b = 0;
        if (A) {
            const int64_t st = (int64_t)A->nf * A->field_elems * (int64_t)sizeof(double);
            b = A->bytes + st * (int64_t)(A->ckpt.size() + A->seg.size()) + A->lim_steps * (int64_t)sizeof(g->dsc->wmin);
        }
        *bytes = b;
    });
}

}  // extern "C"
