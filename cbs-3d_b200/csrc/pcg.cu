// Pressure PCG on sm_100a.
//
// Operator.  The reference applies the pressure operator element by element,
// colour by colour (src/linalg/MatrixVectorCalc.cpp:125-205).  Here the six
// per-element coefficients gstif = gstifE*dt_e are summed once per step into
// one coefficient per node pair (contributions added in ascending element
// order), stored as SELL-32: slices of 32 consecutive rows, each slice padded
// to its longest row and laid out column-major so a warp reads 32 rows'
// k-th entries in one coalesced 256-byte (FP64) load.  For the Kuhn meshes
// this halves the bytes per matvec against the element-by-element form
// (14 pair entries of 12 B per node instead of ~5.7 tets of 64 B).
//
// Solver.  One persistent cooperative kernel runs the whole Jacobi-PCG of
// ConjugateGradient::solvePressure (src/linalg/ConjugateGradient.cpp:584-869):
// the same masks, constraints, checks, convergence tests and iteration
// count semantics, with two grid-wide barriers per iteration.  The search
// direction update p = z + beta*p of the next iteration is folded into the
// matvec (double-buffered p; neighbours' new p formed on the fly from z and
// the previous p), and every CTA reduces the per-CTA partials in the same
// fixed order, so alpha, beta and the stopping decision are identical in all
// CTAs and reproducible run to run.  That is k_pcg64 with its variants; the
// kernels that solves run by default (k_pcg64c, k_pcg64g, further down) take
// the single-reduction form, one all-reduce per iteration.
#include "pcg.cuh"
#include "mg.cuh"

#include <algorithm>
#include <cstdio>
#include <map>
#include <mutex>
#include <cstring>
#include <type_traits>
#include <vector>

namespace cbs3d {

namespace {

// One 512-thread CTA per SM (128 registers per thread fill the register
// file): half the CTAs of two 256-thread CTAs per SM, so the grid-wide
// all-reduce reads half the partials.
constexpr int PCG_THREADS = 512;
constexpr int PCG_CTAS_PER_SM = 1;
constexpr int PCG_WARPS = PCG_THREADS / 32;

#define CUDA_OK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) throw Error(CBS3D_CUDA_ERROR, std::string(#x) + ": " + cudaGetErrorString(e_)); } while (0)

// The dynamic shared-memory limit is one attribute per kernel and device,
// shared by every engine and batch in the process: it only ever grows, so a
// smaller later request cannot invalidate an earlier engine's launches.
cudaError_t raise_smem_limit(const void* fn, size_t smem)
{
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> limit;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    size_t& cur = limit[{dev, fn}];
    if (smem <= cur) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e == cudaSuccess) cur = smem;
    return e;
}

template <typename T>
T* dalloc(size_t n)
{
    T* p = nullptr;
    if (n == 0) n = 1;
    CUDA_OK(cudaMalloc(&p, n * sizeof(T)));
    return p;
}

// ------------------------------------------------------- ELL assembly
__global__ void k_ell_from_state(DevState S, const long long* cptr, const int* cent, double* val,
                                 float* val32, long long nslots)
{
    const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nslots) return;
    const int E = S.P.E;
    double v = 0.0;
    for (long long c = cptr[s]; c < cptr[s + 1]; ++c) {
        const int ent = cent[c];
        const int e = ent >> 3, g = ent & 7;
        v += S.gstifE[(size_t)g * E + e] * S.delte[e];
    }
    val[s] = v;
    if (val32) val32[s] = (float)v;
}

__global__ void k_ell_from_gstif(const double* gstif, const long long* cptr, const int* cent,
                                 double* val, float* val32, long long nslots)
{
    const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nslots) return;
    double v = 0.0;
    for (long long c = cptr[s]; c < cptr[s + 1]; ++c) {
        const int ent = cent[c];
        v += gstif[(size_t)(ent >> 3) * 6 + (ent & 7)];
    }
    val[s] = v;
    if (val32) val32[s] = (float)v;
}

// impose_pressure_constraints (src/linalg/ConjugateGradient.cpp:188-214) on
// the node-ordered arrays, and the solver's inputs from them in row-position
// order (every node has one position; padding positions get inactive flags
// and zeros).  One launch: on small meshes a step's time outside the solve is
// its launches.
__global__ void k_impose_perm_in(PcgDev D, double* xp, double* bp, double* dp, uint8_t* fp)
{
    const int pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= D.N) return;
    const int i = D.row_node[pos];
    double x = 0.0, b = 0.0, d = 0.0;
    uint8_t f = 0;
    if (i >= 0) {
        f = D.nflag[i] & 5;
        if (!(f & 1)) {
            D.pres[i] = 0.0; D.rhs1[i] = 0.0; D.pdiag[i] = 0.0;
        } else if (f & 4) {
            x = b = D.pfix[i];
            d = 1.0;
            D.pres[i] = x; D.rhs1[i] = b; D.pdiag[i] = d;
        } else {
            x = D.pres[i]; b = D.rhs1[i]; d = D.pdiag[i];
        }
    }
    xp[pos] = x;
    bp[pos] = b;
    dp[pos] = d;
    fp[pos] = f;
}

// The pressure back to node order.
__global__ void k_perm_out(PcgDev D, const double* xp, double* pres)
{
    const int pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= D.N) return;
    const int i = D.row_node[pos];
    if (i >= 0) pres[i] = xp[pos];
}

// y = A x on the assembled operator; identity rows on fixed nodes
__global__ void k_ell_multiply(PcgDev D, const double* x, double* y)
{
    const int pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= D.nslices * 32) return;
    const int i = D.row_node[pos];
    if (i < 0) return;
    const int s = pos >> 5, lane = pos & 31;
    const long long base = D.slice_off[s] + lane;
    const int w = D.slice_w[s];
    double off = 0.0;
    for (int k = 0; k < w; ++k) {
        const int j = D.row_node[D.col[base + 32LL * k]];
        off = fma(D.val[base + 32LL * k], j >= 0 ? x[j] : 0.0, off);
    }
    double v = fma(D.pdiag[i], x[i], off);
    if (D.nflag[i] & 4) v = x[i];
    y[i] = v;
}

// ------------------------------------------------------- solve segments
// One cooperative launch solves one system, or -- for the batched step --
// several independent systems at once: CTAs [cta0, cta0+ncta) of the grid
// then own instance k's slice range [s0, s1), and every reduction, barrier,
// status and result is per instance.  SegView is this CTA's view, with the
// solve's scalars.
struct SegView {
    int G, b;      // CTAs of this CTA's solve; this CTA's index among them
    int s0, s1;    // slice range of the solve
    int k;         // instance, -1 for a single solve
    int precond, conv_test, max_iter;
    double rel_tol, abs_tol;
};

template <bool BATCH>
__device__ __forceinline__ SegView seg_view(const PcgDev& D)
{
    if constexpr (!BATCH)
        return SegView{(int)gridDim.x, (int)blockIdx.x, 0, D.nslices, -1, D.precond, D.conv_test, D.max_iter,
                       D.rel_tol, D.abs_tol};
    else {
    const int k = D.cta_inst[blockIdx.x];
    const PcgInst& I = D.inst[k];
    return SegView{I.ncta, (int)blockIdx.x - I.cta0, I.s0, I.s1, k, I.precond, I.conv_test, I.max_iter,
                   I.rel_tol, I.abs_tol};
    }
}
__device__ __forceinline__ DevStatus* seg_status(const PcgDev& D, const SegView& g) { return g.k < 0 ? D.status : D.inst[g.k].status; }
__device__ __forceinline__ CgOut* seg_out(const PcgDev& D, const SegView& g) { return g.k < 0 ? D.out : D.inst[g.k].out; }

// ------------------------------------------------- deterministic reductions
struct Acc4 {
    double a, b, mx, flag;
};

// Grid-wide all-reduce of (sum a, sum b, max mx, max flag) fused with the
// grid barrier (grid_allreduce_v below).
template <int NV, int NSUM, int NT = PCG_THREADS>
__device__ __forceinline__ bool grid_allreduce_v(double (&v)[NV], const PcgDev& D, const SegView& g, int phase,
                                                 double (&out)[NV]);

__device__ __forceinline__ bool grid_allreduce(Acc4 v, const PcgDev& D, const SegView& g, int phase, Acc4& out)
{
    double a[4] = {v.a, v.b, v.mx, v.flag}, o[4];
    const bool ok = grid_allreduce_v<4, 2>(a, D, g, phase, o);
    out = Acc4{o[0], o[1], o[2], o[3]};
    return ok;
}

__device__ __forceinline__ bool cg_converged(int test, double rel, double mx, double rtol, double atol)
{
    if (test == 1) return mx <= atol;
    if (test == 2) return rel <= rtol;
    return mx <= atol || rel <= rtol;
}

__device__ __forceinline__ void cg_finish(const PcgDev& D, const SegView& g, int it, int conv, double init,
                                          double fin, double rel, double mx)
{
    if (g.b == 0 && threadIdx.x == 0) {
        CgOut* o = seg_out(D, g);
        o->iterations = it;
        o->converged = conv;
        o->initial_l2 = init;
        o->final_l2 = fin;
        o->rel = rel;
        o->max_abs = mx;
    }
}

// ---------------------------------------------------- persistent FP64 PCG
// HALO: the neighbour values of each iteration's product (z and the previous
// direction of every column of the CTA's rows) are staged in shared memory
// once per iteration, and the slots carry 16-bit indices into that halo
// (D.halo_ptr/halo_idx/lcol of this kernel's partition), so the rounds
// stream only coefficients and local columns and read neighbours from shared
// memory.  Same arithmetic in the same order as without.
template <bool HALO>
__global__ void __launch_bounds__(PCG_THREADS, PCG_CTAS_PER_SM) k_pcg64(PcgDev D)
{
    const SegView g = seg_view<false>(D);
    const int G = g.G, b = g.b;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s_beg = g.s0 + (int)((long long)b * (g.s1 - g.s0) / G);
    const int s_end = g.s0 + (int)((long long)(b + 1) * (g.s1 - g.s0) / G);
    int phase = 0;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // HALO: per halo entry (z, previous direction) -- on the first
    // iteration (0, current direction) -- one 16-byte read per neighbour
    double2* hzp = reinterpret_cast<double2*>(smem_raw);
    // HALO: the CTA's slices in KP parts (one unless a CTA's whole halo
    // would not fit), each staged and processed in turn
    const int KP = HALO ? (D.halo_parts > 0 ? D.halo_parts : 1) : 1;

    // ---- r0 = b - A p0, z0, d0 = z0, (r,r), (r,z), max|r|
    Acc4 acc{0.0, 0.0, 0.0, 0.0};
    for (int s = s_beg + warp; s < s_end; s += PCG_WARPS) {
        const int i = s * 32 + lane;
        const long long base = D.slice_off[s] + lane;
        const int w = D.slice_w[s];
        double off = 0.0;
        for (int k = 0; k < w; ++k) off = fma(D.val[base + 32LL * k], D.pres[D.col[base + 32LL * k]], off);
        const uint8_t f = D.nflag[i];
        const bool active = f & 1, freen = (f & 1) && !(f & 4);
        const double y = fma(D.pdiag[i], D.pres[i], off);
        double ri = active ? D.rhs1[i] - y : 0.0;
        if (!freen) ri = 0.0;
        double zi = 0.0;
        if (freen) {
            if (g.precond) {
                const double dg = D.pdiag[i];
                if (!(isfinite(dg) && dg > 1.0e-30)) acc.flag = fmax(acc.flag, 1.0);
                else zi = ri / dg;
            } else {
                zi = ri;
            }
            if (!isfinite(ri)) acc.flag = fmax(acc.flag, 2.0);
            acc.a = fma(ri, ri, acc.a);
            acc.b = fma(ri, zi, acc.b);
            acc.mx = fmax(acc.mx, fabs(ri));
        }
        D.r[i] = ri;
        D.z[i] = zi;
        D.pA[i] = zi;
    }
    Acc4 t = Acc4{0.0, 0.0, 0.0, 0.0};
    if (!grid_allreduce(acc, D, g, phase, t)) return;
    ++phase;
    const double init = sqrt(t.a);
    if (init <= 1.0e-300) { cg_finish(D, g, 0, 1, init, init, 0.0, t.mx); return; }
    if (cg_converged(g.conv_test, 1.0, t.mx, g.rel_tol, g.abs_tol)) { cg_finish(D, g, 0, 1, init, init, 1.0, t.mx); return; }
    if (t.flag >= 2.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, 0, R_PCG_RESID); return; }
    if (t.flag >= 1.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 1, ST_PCG, 0, R_PCG_DIAG); return; }
    double rz = t.b;
    if (rz <= 1.0e-300 || !isfinite(rz)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, 0, R_PCG_RZ0); return; }

    double* pc = D.pA;   // current direction
    double* pp = D.pB;   // previous direction (unused at it=1)
    double beta = 0.0, fin = init, rel = 1.0, mx = t.mx;
    int it = 0, conv = 0;
    for (it = 1; it <= g.max_iter; ++it) {
        // ---- q = A p (p formed here from z and the previous p), (p, q)
        Acc4 pa{0.0, 0.0, 0.0, 0.0};
        const bool upd = it > 1;
        for (int part = 0; part < KP; ++part) {
        const int ps0 = s_beg + (int)((long long)part * (s_end - s_beg) / KP);
        const int ps1 = s_beg + (int)((long long)(part + 1) * (s_end - s_beg) / KP);
        if constexpr (HALO) {
            // z and pp (or pc) were written before the last all-reduce
            __syncthreads();
            const int h0 = D.halo_ptr[b * KP + part], nh = D.halo_ptr[b * KP + part + 1] - h0;
            for (int k = threadIdx.x; k < nh; k += PCG_THREADS) {
                const int j = D.halo_idx[h0 + k];
                hzp[k] = make_double2(upd ? __ldcg(D.z + j) : 0.0, __ldcg((upd ? pp : pc) + j));
            }
            __syncthreads();
        }
        for (int s = ps0 + warp; s < ps1; s += PCG_WARPS) {
            const int i = s * 32 + lane;
            const long long base = D.slice_off[s] + lane;
            const int w = D.slice_w[s];
            const uint8_t f = D.nflag[i];
            const bool freen = (f & 1) && !(f & 4);
            double off = 0.0, pci;
            // Rounds of eight slots; the next round's columns and
            // coefficients (streamed from HBM on large meshes) are requested
            // before this round's neighbour gathers (mostly L2 hits), so the
            // two latencies overlap and each lane keeps more loads in flight.
            // The sum still runs over the slots in order.
            constexpr int CH = 8;
            // columns: global positions, or (HALO) indices into the staged halo
            auto colat = [&](long long t) -> int { return HALO ? (int)__ldcs(D.lcol + t) : D.col[t]; };
            const int cpad = HALO ? 0 : i;   // a valid column for the padding lanes of a round
            int cn[CH];
            double vn[CH];
#pragma unroll
            for (int u = 0; u < CH; ++u) {
                cn[u] = u < w ? colat(base + 32LL * u) : cpad;
                vn[u] = u < w ? __ldcs(D.val + base + 32LL * u) : 0.0;
            }
            for (int k0 = 0; k0 < w; k0 += CH) {
                int c[CH];
                double v[CH];
#pragma unroll
                for (int u = 0; u < CH; ++u) { c[u] = cn[u]; v[u] = vn[u]; }
#pragma unroll
                for (int u = 0; u < CH; ++u) {
                    const int k = k0 + CH + u;
                    cn[u] = k < w ? colat(base + 32LL * k) : cpad;
                    vn[u] = k < w ? __ldcs(D.val + base + 32LL * k) : 0.0;
                }
                double x[CH];
                if constexpr (HALO) {
                    if (upd) {
#pragma unroll
                        for (int u = 0; u < CH; ++u) {
                            const double2 zp = hzp[c[u]];
                            x[u] = fma(beta, zp.y, zp.x);
                        }
                    } else {
#pragma unroll
                        for (int u = 0; u < CH; ++u) x[u] = hzp[c[u]].y;
                    }
                } else if (upd) {
#pragma unroll
                    for (int u = 0; u < CH; ++u) x[u] = fma(beta, __ldcg(pp + c[u]), __ldcg(D.z + c[u]));
                } else {
#pragma unroll
                    for (int u = 0; u < CH; ++u) x[u] = __ldcg(pc + c[u]);
                }
#pragma unroll
                for (int u = 0; u < CH; ++u)
                    if (k0 + u < w) off = fma(v[u], x[u], off);
            }
            if (upd) {
                pci = freen ? fma(beta, pp[i], D.z[i]) : 0.0;
                pc[i] = pci;
            } else {
                pci = pc[i];
            }
            const double qi = freen ? fma(D.pdiag[i], pci, off) : 0.0;
            D.q[i] = qi;
            if (freen) pa.a = fma(pci, qi, pa.a);
        }
        }   // parts
        t = Acc4{0.0, 0.0, 0.0, 0.0};
        if (!grid_allreduce(pa, D, g, phase, t)) return;
        ++phase;
        const double pAp = t.a;
        if (fabs(pAp) <= 1.0e-300 || !isfinite(pAp)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_PAP); return; }
        const double alpha = rz / pAp;

        // ---- p += alpha d, r -= alpha q, z = M^-1 r, (r,r), (r,z), max|r|
        Acc4 rr{0.0, 0.0, 0.0, 0.0};
        for (int s = s_beg + warp; s < s_end; s += PCG_WARPS) {
            const int i = s * 32 + lane;
            const uint8_t f = D.nflag[i];
            if (!((f & 1) && !(f & 4))) continue;
            D.pres[i] = fma(alpha, pc[i], D.pres[i]);
            const double ri = fma(-alpha, D.q[i], D.r[i]);
            D.r[i] = ri;
            const double zi = g.precond ? ri / D.pdiag[i] : ri;
            D.z[i] = zi;
            if (!isfinite(ri)) rr.flag = 1.0;
            rr.a = fma(ri, ri, rr.a);
            rr.b = fma(ri, zi, rr.b);
            rr.mx = fmax(rr.mx, fabs(ri));
        }
        t = Acc4{0.0, 0.0, 0.0, 0.0};
        if (!grid_allreduce(rr, D, g, phase, t)) return;
        ++phase;
        fin = sqrt(t.a);
        mx = t.mx;
        rel = fin / init;
        if (cg_converged(g.conv_test, rel, mx, g.rel_tol, g.abs_tol)) { conv = 1; break; }
        if (t.flag > 0.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, it, R_PCG_RESID); return; }
        const double rzn = t.b;
        if (rzn <= 1.0e-300 || !isfinite(rzn)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_RZ); return; }
        beta = rzn / rz;
        rz = rzn;
        double* tmp = pp; pp = pc; pc = tmp;
    }
    if (it > g.max_iter) it = g.max_iter;
    cg_finish(D, g, it, conv, init, fin, rel, mx);
    if (!conv && b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 2, ST_PCG, it, R_PCG_MAXIT);
}

// ------------------------------------------- register-resident FP64 PCG
// Same algorithm as k_pcg64, for meshes where every thread owns at most RMAX
// rows (slices s_beg + warp + 8r, lane = row within the slice).  The row
// state -- residual, search direction, q, diagonal and flags -- stays in
// registers for the whole solve; each iteration writes the new direction
// (double-buffered, for the neighbours' on-the-fly update), z and the
// pressure to global memory.  Each row's pair entries are fetched eight at a time before
// the neighbour gathers are issued, so a lane keeps many loads in flight.
template <int RMAX>
__global__ void __launch_bounds__(PCG_THREADS, PCG_CTAS_PER_SM) k_pcg64r(PcgDev D)
{
    const SegView g = seg_view<false>(D);
    const int G = g.G, b = g.b;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s_beg = g.s0 + (int)((long long)b * (g.s1 - g.s0) / G);
    const int s_end = g.s0 + (int)((long long)(b + 1) * (g.s1 - g.s0) / G);
    int phase = 0;
    

    double r[RMAX], p[RMAX], q[RMAX], dg[RMAX];
    bool fr[RMAX];
    int row[RMAX];
#pragma unroll
    for (int k = 0; k < RMAX; ++k) {
        const int s = s_beg + warp + PCG_WARPS * k;
        row[k] = (s < s_end) ? s * 32 + lane : -1;
        r[k] = p[k] = q[k] = dg[k] = 0.0;
        fr[k] = false;
    }

    // off[k] = sum_j A_ij v_j over row k's pair entries, v_j = beta*pp_j + zz_j
    // (v = zz when pp is null).  All of the thread's rows advance chunk by
    // chunk together, so RMAX*CH coefficient loads and then RMAX*CH gathers
    // are in flight at once; each row still accumulates in ascending k.
    constexpr int CH = (RMAX >= 8) ? 1 : (RMAX >= 4) ? 2 : 8;
    long long base[RMAX];
    int wr[RMAX];
    int wmax = 0;
#pragma unroll
    for (int k = 0; k < RMAX; ++k) {
        base[k] = 0;
        wr[k] = 0;
        if (row[k] >= 0) {
            const int s = row[k] >> 5;
            base[k] = D.slice_off[s] + lane;
            wr[k] = D.slice_w[s];
            wmax = wr[k] > wmax ? wr[k] : wmax;
        }
    }
    auto offdiag_all = [&](double beta, const double* pp, const double* zz, double* off) {
#pragma unroll
        for (int k = 0; k < RMAX; ++k) off[k] = 0.0;
        for (int k0 = 0; k0 < wmax; k0 += CH) {
            int c[RMAX][CH];
            double v[RMAX][CH], g[RMAX][CH];
#pragma unroll
            for (int k = 0; k < RMAX; ++k)
#pragma unroll
                for (int u = 0; u < CH; ++u) {
                    const bool ok = k0 + u < wr[k];
                    c[k][u] = ok ? D.col[base[k] + 32LL * (k0 + u)] : 0;
                    v[k][u] = ok ? D.val[base[k] + 32LL * (k0 + u)] : 0.0;
                }
#pragma unroll
            for (int k = 0; k < RMAX; ++k)
#pragma unroll
                for (int u = 0; u < CH; ++u) {
                    const bool ok = k0 + u < wr[k];
                    g[k][u] = ok ? (pp ? fma(beta, __ldcg(pp + c[k][u]), __ldcg(zz + c[k][u])) : __ldcg(zz + c[k][u])) : 0.0;
                }
#pragma unroll
            for (int k = 0; k < RMAX; ++k)
#pragma unroll
                for (int u = 0; u < CH; ++u) off[k] = fma(v[k][u], g[k][u], off[k]);
        }
    };

    // ---- r0 = b - A p0, z0; direction buffer 0 cleared for iteration 1
    Acc4 acc{0.0, 0.0, 0.0, 0.0};
    double off[RMAX];
    offdiag_all(0.0, nullptr, D.pres, off);
#pragma unroll
    for (int k = 0; k < RMAX; ++k) {
        const int i = row[k];
        if (i < 0) continue;
        const uint8_t f = D.nflag[i];
        const bool active = f & 1;
        fr[k] = (f & 1) && !(f & 4);
        dg[k] = D.pdiag[i];
        const double y = fma(dg[k], D.pres[i], off[k]);
        double ri = active ? D.rhs1[i] - y : 0.0;
        if (!fr[k]) ri = 0.0;
        double zi = 0.0;
        if (fr[k]) {
            if (g.precond) {
                if (!(isfinite(dg[k]) && dg[k] > 1.0e-30)) acc.flag = fmax(acc.flag, 1.0);
                else zi = ri / dg[k];
            } else {
                zi = ri;
            }
            if (!isfinite(ri)) acc.flag = fmax(acc.flag, 2.0);
            acc.a = fma(ri, ri, acc.a);
            acc.b = fma(ri, zi, acc.b);
            acc.mx = fmax(acc.mx, fabs(ri));
        }
        r[k] = ri;
        D.z[i] = zi;
        D.pA[i] = 0.0;
    }
    Acc4 t = Acc4{0.0, 0.0, 0.0, 0.0};
    if (!grid_allreduce(acc, D, g, phase, t)) return;
    ++phase;
    const double init = sqrt(t.a);
    if (init <= 1.0e-300) { cg_finish(D, g, 0, 1, init, init, 0.0, t.mx); return; }
    if (cg_converged(g.conv_test, 1.0, t.mx, g.rel_tol, g.abs_tol)) { cg_finish(D, g, 0, 1, init, init, 1.0, t.mx); return; }
    if (t.flag >= 2.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, 0, R_PCG_RESID); return; }
    if (t.flag >= 1.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 1, ST_PCG, 0, R_PCG_DIAG); return; }
    double rz = t.b;
    if (rz <= 1.0e-300 || !isfinite(rz)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, 0, R_PCG_RZ0); return; }

    double beta = 0.0, fin = init, rel = 1.0, mx = t.mx;
    int it = 0, conv = 0;
    for (it = 1; it <= g.max_iter; ++it) {
        const double* pprev = (it & 1) ? D.pA : D.pB;
        double* pnew = (it & 1) ? D.pB : D.pA;
        // ---- p = z + beta p (own rows), q = A p with neighbours' p formed on the fly
        Acc4 pa{0.0, 0.0, 0.0, 0.0};
        offdiag_all(beta, pprev, D.z, off);
#pragma unroll
        for (int k = 0; k < RMAX; ++k) {
            const int i = row[k];
            if (i < 0) continue;
            p[k] = fr[k] ? fma(beta, p[k], D.z[i]) : 0.0;
            pnew[i] = p[k];
            q[k] = fr[k] ? fma(dg[k], p[k], off[k]) : 0.0;
            if (fr[k]) pa.a = fma(p[k], q[k], pa.a);
        }
        t = Acc4{0.0, 0.0, 0.0, 0.0};
        if (!grid_allreduce(pa, D, g, phase, t)) return;
        ++phase;
        const double pAp = t.a;
        if (fabs(pAp) <= 1.0e-300 || !isfinite(pAp)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_PAP); return; }
        const double alpha = rz / pAp;

        // ---- x += alpha p, r -= alpha q, z = M^-1 r
        Acc4 rr{0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < RMAX; ++k) {
            const int i = row[k];
            if (i < 0 || !fr[k]) continue;
            D.pres[i] = fma(alpha, p[k], D.pres[i]);
            r[k] = fma(-alpha, q[k], r[k]);
            const double zk = g.precond ? r[k] / dg[k] : r[k];
            D.z[i] = zk;
            if (!isfinite(r[k])) rr.flag = 1.0;
            rr.a = fma(r[k], r[k], rr.a);
            rr.b = fma(r[k], zk, rr.b);
            rr.mx = fmax(rr.mx, fabs(r[k]));
        }
        t = Acc4{0.0, 0.0, 0.0, 0.0};
        if (!grid_allreduce(rr, D, g, phase, t)) return;
        ++phase;
        fin = sqrt(t.a);
        mx = t.mx;
        rel = fin / init;
        if (cg_converged(g.conv_test, rel, mx, g.rel_tol, g.abs_tol)) { conv = 1; break; }
        if (t.flag > 0.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, it, R_PCG_RESID); return; }
        const double rzn = t.b;
        if (rzn <= 1.0e-300 || !isfinite(rzn)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_RZ); return; }
        beta = rzn / rz;
        rz = rzn;
    }
    if (it > g.max_iter) it = g.max_iter;
    cg_finish(D, g, it, conv, init, fin, rel, mx);
    if (!conv && b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 2, ST_PCG, it, R_PCG_MAXIT);
}

// --------------------------------------- halo-staged FP64 PCG (choice 3)
// The register-resident algorithm of k_pcg64r with the neighbour gathers
// served from shared memory.  Each persistent CTA owns a contiguous block of
// slices; the host lists, per CTA, the distinct nodes its rows reference (its
// halo, own rows included) and rewrites every pair entry's column as a 16-bit
// index into that list.  Each phase the CTA stages the values it needs
// (v = beta*p_prev + z, or the pressure in phase 0) for its halo into shared
// memory with one cooperative, mostly contiguous load, and the matvec then
// reads only the streamed coefficients from global memory.  The local column
// indices stay in shared memory for the whole solve.
template <int RMAX>
__global__ void __launch_bounds__(PCG_THREADS, PCG_CTAS_PER_SM) k_pcg64h(PcgDev D)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const SegView g = seg_view<false>(D);
    const int G = g.G, b = g.b;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s_beg = g.s0 + (int)((long long)b * (g.s1 - g.s0) / G);
    const int s_end = g.s0 + (int)((long long)(b + 1) * (g.s1 - g.s0) / G);
    const long long S0 = D.slice_off[s_beg];
    const int nsl = (int)(D.slice_off[s_end] - S0);
    const int h0 = D.halo_ptr[blockIdx.x];
    const int nh = D.halo_ptr[blockIdx.x + 1] - h0;
    double* vh = reinterpret_cast<double*>(smem_raw);
    int* hidx = reinterpret_cast<int*>(vh + D.halo_max);
    unsigned short* lcs = reinterpret_cast<unsigned short*>(hidx + D.halo_max);
    for (int k = threadIdx.x; k < nh; k += PCG_THREADS) hidx[k] = D.halo_idx[h0 + k];
    for (int k = threadIdx.x; k < nsl; k += PCG_THREADS) lcs[k] = D.lcol[S0 + k];
    int phase = 0;
    

    double r[RMAX], p[RMAX], q[RMAX], dg[RMAX];
    bool fr[RMAX];
    int row[RMAX], lbase[RMAX], wr[RMAX];
    int wmax = 0;
#pragma unroll
    for (int k = 0; k < RMAX; ++k) {
        const int s = s_beg + warp + PCG_WARPS * k;
        row[k] = (s < s_end) ? s * 32 + lane : -1;
        lbase[k] = 0;
        wr[k] = 0;
        if (s < s_end) {
            lbase[k] = (int)(D.slice_off[s] - S0) + lane;
            wr[k] = D.slice_w[s];
            wmax = wr[k] > wmax ? wr[k] : wmax;
        }
        r[k] = p[k] = q[k] = dg[k] = 0.0;
        fr[k] = false;
    }

    // stage v_j = beta*pp_j + zz_j (v = zz when pp is null) for the halo
    auto stage = [&](double beta, const double* pp, const double* zz) {
        __syncthreads();
        for (int k = threadIdx.x; k < nh; k += PCG_THREADS) {
            const int j = hidx[k];
            vh[k] = pp ? fma(beta, __ldcg(pp + j), __ldcg(zz + j)) : __ldcg(zz + j);
        }
        __syncthreads();
    };
    constexpr int CH = (RMAX >= 8) ? 2 : (RMAX >= 4) ? 4 : 8;
    auto offdiag_all = [&](double* off) {
#pragma unroll
        for (int k = 0; k < RMAX; ++k) off[k] = 0.0;
        for (int k0 = 0; k0 < wmax; k0 += CH) {
            double v[RMAX][CH];
#pragma unroll
            for (int k = 0; k < RMAX; ++k)
#pragma unroll
                for (int u = 0; u < CH; ++u)
                    v[k][u] = (k0 + u < wr[k]) ? __ldcg(D.val + S0 + lbase[k] + 32 * (k0 + u)) : 0.0;
#pragma unroll
            for (int k = 0; k < RMAX; ++k)
#pragma unroll
                for (int u = 0; u < CH; ++u) {
                    const double g = (k0 + u < wr[k]) ? vh[lcs[lbase[k] + 32 * (k0 + u)]] : 0.0;
                    off[k] = fma(v[k][u], g, off[k]);
                }
        }
    };

    // ---- r0 = b - A p0, z0; direction buffer 0 cleared for iteration 1
    Acc4 acc{0.0, 0.0, 0.0, 0.0};
    double off[RMAX];
    stage(0.0, nullptr, D.pres);
    offdiag_all(off);
#pragma unroll
    for (int k = 0; k < RMAX; ++k) {
        const int i = row[k];
        if (i < 0) continue;
        const uint8_t f = D.nflag[i];
        const bool active = f & 1;
        fr[k] = (f & 1) && !(f & 4);
        dg[k] = D.pdiag[i];
        const double y = fma(dg[k], D.pres[i], off[k]);
        double ri = active ? D.rhs1[i] - y : 0.0;
        if (!fr[k]) ri = 0.0;
        double zi = 0.0;
        if (fr[k]) {
            if (g.precond) {
                if (!(isfinite(dg[k]) && dg[k] > 1.0e-30)) acc.flag = fmax(acc.flag, 1.0);
                else zi = ri / dg[k];
            } else {
                zi = ri;
            }
            if (!isfinite(ri)) acc.flag = fmax(acc.flag, 2.0);
            acc.a = fma(ri, ri, acc.a);
            acc.b = fma(ri, zi, acc.b);
            acc.mx = fmax(acc.mx, fabs(ri));
        }
        r[k] = ri;
        D.z[i] = zi;
        D.pA[i] = 0.0;
    }
    Acc4 t = Acc4{0.0, 0.0, 0.0, 0.0};
    if (!grid_allreduce(acc, D, g, phase, t)) return;
    ++phase;
    const double init = sqrt(t.a);
    if (init <= 1.0e-300) { cg_finish(D, g, 0, 1, init, init, 0.0, t.mx); return; }
    if (cg_converged(g.conv_test, 1.0, t.mx, g.rel_tol, g.abs_tol)) { cg_finish(D, g, 0, 1, init, init, 1.0, t.mx); return; }
    if (t.flag >= 2.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, 0, R_PCG_RESID); return; }
    if (t.flag >= 1.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 1, ST_PCG, 0, R_PCG_DIAG); return; }
    double rz = t.b;
    if (rz <= 1.0e-300 || !isfinite(rz)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, 0, R_PCG_RZ0); return; }

    double beta = 0.0, fin = init, rel = 1.0, mx = t.mx;
    int it = 0, conv = 0;
    for (it = 1; it <= g.max_iter; ++it) {
        const double* pprev = (it & 1) ? D.pA : D.pB;
        double* pnew = (it & 1) ? D.pB : D.pA;
        Acc4 pa{0.0, 0.0, 0.0, 0.0};
        stage(beta, pprev, D.z);
        offdiag_all(off);
#pragma unroll
        for (int k = 0; k < RMAX; ++k) {
            const int i = row[k];
            if (i < 0) continue;
            p[k] = fr[k] ? fma(beta, p[k], D.z[i]) : 0.0;
            pnew[i] = p[k];
            q[k] = fr[k] ? fma(dg[k], p[k], off[k]) : 0.0;
            if (fr[k]) pa.a = fma(p[k], q[k], pa.a);
        }
        t = Acc4{0.0, 0.0, 0.0, 0.0};
        if (!grid_allreduce(pa, D, g, phase, t)) return;
        ++phase;
        const double pAp = t.a;
        if (fabs(pAp) <= 1.0e-300 || !isfinite(pAp)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_PAP); return; }
        const double alpha = rz / pAp;

        Acc4 rr{0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < RMAX; ++k) {
            const int i = row[k];
            if (i < 0 || !fr[k]) continue;
            D.pres[i] = fma(alpha, p[k], D.pres[i]);
            r[k] = fma(-alpha, q[k], r[k]);
            const double zk = g.precond ? r[k] / dg[k] : r[k];
            D.z[i] = zk;
            if (!isfinite(r[k])) rr.flag = 1.0;
            rr.a = fma(r[k], r[k], rr.a);
            rr.b = fma(r[k], zk, rr.b);
            rr.mx = fmax(rr.mx, fabs(r[k]));
        }
        t = Acc4{0.0, 0.0, 0.0, 0.0};
        if (!grid_allreduce(rr, D, g, phase, t)) return;
        ++phase;
        fin = sqrt(t.a);
        mx = t.mx;
        rel = fin / init;
        if (cg_converged(g.conv_test, rel, mx, g.rel_tol, g.abs_tol)) { conv = 1; break; }
        if (t.flag > 0.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, it, R_PCG_RESID); return; }
        const double rzn = t.b;
        if (rzn <= 1.0e-300 || !isfinite(rzn)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_RZ); return; }
        beta = rzn / rz;
        rz = rzn;
    }
    if (it > g.max_iter) it = g.max_iter;
    cg_finish(D, g, it, conv, init, fin, rel, mx);
    if (!conv && b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 2, ST_PCG, it, R_PCG_MAXIT);
}

// ------------------------------------------- single-synchronisation PCG
// Chronopoulos-Gear form of the same Jacobi-PCG: the matvec is applied to z
// (w = A z) and the direction's product s = A p follows the recurrence
// s = w + beta*s, so alpha and beta come from one grid reduction of
// (r.z, z.w, r.r, max|r|) per iteration instead of two.  Residuals, stopping
// test, iteration count and breakdown checks keep the reference's meaning
// (src/linalg/ConjugateGradient.cpp:725-853); in exact arithmetic the iterates
// equal the standard PCG's.  k_pcg64c (the default), k_pcg64g, k_pcg64d and
// k_pcg32m are this iteration.
struct Acc6 {
    double a, b, c, mx, flag;
};

// Grid-wide all-reduce of NV values per thread: the first NSUM summed, the
// rest max-reduced.  Every CTA publishes its partials (double-buffered by
// phase parity), arrives on a 64-bit counter that only grows, waits until
// all G CTAs of this phase have arrived, and then reduces the G partials
// itself in a fixed order (thread t takes CTAs t, t+T, ...; warp shuffles;
// warps in order).  The partials are stored value-major (value q of CTA b at
// q*G + b), so a warp reading one value of 32 CTAs touches two L2 lines.  Every CTA therefore computes bit-identical totals without
// a second round trip through a last-arriving CTA.  The caller passes the
// number of all-reduces this launch has completed as `phase`.  Returns false
// when the wait gave up (status TIMEOUT) or another CTA raised a status.
template <int NV, int NSUM, int NT>
__device__ __forceinline__ bool grid_allreduce_v(double (&v)[NV], const PcgDev& D, const SegView& g, int phase,
                                                 double (&out)[NV])
{
    static_assert(NV <= 8, "partials hold 8 doubles per CTA");
    __shared__ double sm[(NT / 32)][NV];
    __shared__ int s_ok;
    const int G = g.G;
    DevStatus* status = seg_status(D, g);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            const double x = __shfl_down_sync(0xffffffffu, v[q], o);
            v[q] = q < NSUM ? v[q] + x : fmax(v[q], x);
        }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) sm[w][q] = v[q];
    __syncthreads();
    unsigned long long* cnt = reinterpret_cast<unsigned long long*>(D.bar);
    double* part = D.part + (size_t)(phase & 1) * G * 8;
    if (threadIdx.x == 0) {
        double t[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) t[q] = 0.0;
        for (int k = 0; k < (NT / 32); ++k)
#pragma unroll
            for (int q = 0; q < NV; ++q) t[q] = q < NSUM ? t[q] + sm[k][q] : fmax(t[q], sm[k][q]);
#pragma unroll
        for (int q = 0; q < NV; ++q) __stcg(part + (q * G + g.b), t[q]);
        const unsigned long long target = (unsigned long long)(phase + 1) * (unsigned long long)G;
        unsigned long long arrived;
        asm volatile("atom.add.acq_rel.gpu.global.u64 %0, [%1], 1;" : "=l"(arrived) : "l"(cnt) : "memory");
        int ok = 1;
        if (arrived + 1 < target) {
            const long long t0 = clock64();
            for (;;) {
                unsigned long long c;
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(cnt) : "memory");
                if (c >= target) break;
                if (ld_relaxed_int(&status->code) != 0) { ok = 0; break; }
                if (clock64() - t0 > (1LL << 31)) {
                    set_status(status, 5 /*CBS3D_TIMEOUT*/, ST_PCG, 0, R_PCG_BARRIER);
                    ok = 0;
                    break;
                }
            }
        }
        if (ok && ld_relaxed_int(&status->code) != 0) ok = 0;
        s_ok = ok;
    }
    __syncthreads();
    const bool ok = s_ok != 0;
    double t[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) t[q] = 0.0;
    if (ok) {
        for (int k = threadIdx.x; k < G; k += NT) {
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                const double x = __ldcg(part + (q * G + k));
                t[q] = q < NSUM ? t[q] + x : fmax(t[q], x);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            const double x = __shfl_down_sync(0xffffffffu, t[q], o);
            t[q] = q < NSUM ? t[q] + x : fmax(t[q], x);
        }
    // sm was last read by thread 0 before the barrier that published s_ok,
    // so the warps' totals can overwrite it now.  Thread q folds value q
    // over the warps in warp order (the same sums as every thread folding
    // all of them) and the warps read the NV results: NV shared-memory
    // reads per warp instead of NV * warps broadcasts, which at 16 warps
    // kept the shared-memory pipe busy for ~1,300 cycles per all-reduce.
    __shared__ double so[NV];
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) sm[w][q] = t[q];
    __syncthreads();
    if (threadIdx.x < NV) {
        const int q = threadIdx.x;
        double x = 0.0;
        for (int k = 0; k < (NT / 32); ++k) x = q < NSUM ? x + sm[k][q] : fmax(x, sm[k][q]);
        so[q] = x;
    }
    __syncthreads();
    // no barrier after these reads: so is rewritten only after the next
    // call's third barrier, and every thread reads it before it arrives at
    // that call's first
#pragma unroll
    for (int q = 0; q < NV; ++q) out[q] = so[q];
    return ok;
}

// Grid all-reduce of (sum a, sum b, sum c, max mx, max flag) that also
// gathers one per-CTA sum: every CTA's block sum of `x` lands in cvec[CTA]
// of every CTA (the aggregated vectors of the two-level preconditioner).
template <int NT>
__device__ __forceinline__ bool grid_allreduce3g(Acc6 v, double x, const PcgDev& D, const SegView& g, int phase,
                                                 Acc6& out, double* cvec)
{
    constexpr int NW = NT / 32;
    __shared__ double sm[NW][6];
    __shared__ int s_ok;
    const int G = g.G;
    DevStatus* status = seg_status(D, g);
    double vv[6] = {v.a, v.b, v.c, v.mx, v.flag, x};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const double y = __shfl_down_sync(0xffffffffu, vv[q], o);
            vv[q] = (q < 3 || q == 5) ? vv[q] + y : fmax(vv[q], y);
        }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 6; ++q) sm[w][q] = vv[q];
    __syncthreads();
    unsigned long long* cnt = reinterpret_cast<unsigned long long*>(D.bar);
    double* part = D.part + (size_t)(phase & 1) * G * 8;
    if (threadIdx.x == 0) {
        double t[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int k = 0; k < NW; ++k)
#pragma unroll
            for (int q = 0; q < 6; ++q) t[q] = (q < 3 || q == 5) ? t[q] + sm[k][q] : fmax(t[q], sm[k][q]);
#pragma unroll
        for (int q = 0; q < 6; ++q) __stcg(part + (q * G + g.b), t[q]);
        const unsigned long long target = (unsigned long long)(phase + 1) * (unsigned long long)G;
        unsigned long long arrived;
        asm volatile("atom.add.acq_rel.gpu.global.u64 %0, [%1], 1;" : "=l"(arrived) : "l"(cnt) : "memory");
        int ok = 1;
        if (arrived + 1 < target) {
            const long long t0 = clock64();
            for (;;) {
                unsigned long long c;
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(cnt) : "memory");
                if (c >= target) break;
                if (ld_relaxed_int(&status->code) != 0) { ok = 0; break; }
                if (clock64() - t0 > (1LL << 31)) {
                    set_status(status, 5 /*CBS3D_TIMEOUT*/, ST_PCG, 0, R_PCG_BARRIER);
                    ok = 0;
                    break;
                }
            }
        }
        if (ok && ld_relaxed_int(&status->code) != 0) ok = 0;
        s_ok = ok;
    }
    __syncthreads();
    const bool ok = s_ok != 0;
    double t[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (ok) {
        for (int k = threadIdx.x; k < G; k += NT) {
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                const double y = __ldcg(part + (q * G + k));
                t[q] = q < 3 ? t[q] + y : fmax(t[q], y);
            }
            cvec[k] = __ldcg(part + (5 * G + k));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            const double y = __shfl_down_sync(0xffffffffu, t[q], o);
            t[q] = q < 3 ? t[q] + y : fmax(t[q], y);
        }
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 5; ++q) sm[w][q] = t[q];
    __syncthreads();
    double o5[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int k = 0; k < NW; ++k)
#pragma unroll
        for (int q = 0; q < 5; ++q) o5[q] = q < 3 ? o5[q] + sm[k][q] : fmax(o5[q], sm[k][q]);
    out = Acc6{o5[0], o5[1], o5[2], o5[3], o5[4]};
    __syncthreads();
    return ok;
}

// ------------------------------------------------------ tagged exchange
// The single-reduction kernels (k_pcg64c, k_pcg64g) exchange values between
// CTAs as 16-byte records {value, tag} that are written and read whole
// (.b128 accesses are single-copy atomic), so a reader that finds the tag it
// waits for holds the value of that exchange: no counter, and for the values
// themselves no fence.  The tag is the solve's epoch (a counter in device
// memory, one more per solve) in the high word and the exchange's number in
// the solve in the low word, so nothing has to be cleared between solves.
// Two buffers alternate by the exchange's parity.  A CTA writes exchange k+2
// over exchange k only after all-reduce k+1, to which every CTA contributes
// after it has read its records of exchange k.
__device__ __forceinline__ void st_tag(TagVal* p, double v, unsigned long long tag)
{
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"(tag)
                 : "memory");
}
template <bool ACQ = false>
__device__ __forceinline__ void ld_tag(const TagVal* p, double& v, unsigned long long& tag)
{
    long long b;
    if constexpr (ACQ)
        asm volatile("{ .reg .b128 t; ld.acquire.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                     : "=l"(b), "=l"(tag)
                     : "l"(p)
                     : "memory");
    else
    asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                 : "=l"(b), "=l"(tag)
                 : "l"(p)
                 : "memory");
    v = __longlong_as_double(b);
}

// Slots per round of k_pcg64c's products: every row of a thread at once (at
// four rows 2 measured as fast as 4; at two rows 2 instead of 8 took 48^3 from 4.46 to 4.12 us).
constexpr int CGCG_ROUND = 2;

// One solve's side of the exchange, for this CTA.
struct TagComm {
    TagVal* rec;                 // 2 x G all-reduce records of REC_STRIDE
    int G, b;
    unsigned long long epoch;    // the solve's epoch in the high word
    DevStatus* status;
    __device__ __forceinline__ unsigned long long tag(int phase) const { return epoch | (unsigned)(phase + 1); }
};
__device__ __forceinline__ TagComm tag_comm(const PcgDev& D, const SegView& g, unsigned long long epoch)
{
    return TagComm{g.k < 0 ? D.rec : D.inst[g.k].rec, g.G, g.b, epoch, seg_status(D, g)};
}
__device__ __forceinline__ unsigned long long* seg_epoch(const PcgDev& D, const SegView& g) { return g.k < 0 ? D.epoch : D.inst[g.k].epoch; }

// A wait's slow path: every 64 unsuccessful polls look for a status raised
// elsewhere, and give up (TIMEOUT) after about a second.
struct SpinLimit {
    int spins = 0;
    long long t0 = 0;
    __device__ __forceinline__ bool expired(DevStatus* status)
    {
        if ((++spins & 63) != 0) return false;
        if (ld_relaxed_int(&status->code) != 0) return true;
        const long long t = clock64();
        if (t0 == 0) t0 = t;
        else if (t - t0 > (1LL << 31)) {
            set_status(status, 5 /*CBS3D_TIMEOUT*/, ST_PCG, 0, R_PCG_BARRIER);
            return true;
        }
        return false;
    }
};

// Waits for the record tagged `want` (v, t: what the last poll returned).
__device__ __forceinline__ bool tag_wait(const TagVal* p, unsigned long long want, double& v, unsigned long long& t,
                                         SpinLimit& lim, DevStatus* status)
{
    while (t != want) {
        if (lim.expired(status)) return false;
        ld_tag(p, v, t);
    }
    return true;
}

// The maximum is taken over the bits of magnitudes, whose order is that of
// the values with infinities and NaN above every finite one: a non-finite
// entry anywhere shows in the total.
__device__ __forceinline__ double max_bits(double a, double b)
{
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    return __longlong_as_double(x > y ? x : y);
}
template <bool MX>
__device__ __forceinline__ double red4(int q, double a, double b)
{
    if constexpr (MX) return q == 3 ? max_bits(a, b) : a + b;
    else return a + b;
}

// All-reduce of three sums and, with MX, a maximum of magnitudes, in two
// halves so that a kernel can put work between them.  The all-reduce is a
// serial chain (shuffles, a store, a poll, shuffles), so its instructions
// count: the maximum, whose comparisons double them, is left out of the
// iterations that need none.  Publish: a warp halves its values with its
// lanes (6 exchanges for four values instead of 20), one warp folds the
// CTA's warps, and four of its lanes write the CTA's record with one store.
// Every CTA's record has a 128-byte line of its own: a line that other SMs
// poll costs a store to it about 0.4 us on B200 (each poll leaves a copy
// that the store has to recall), so with eight CTAs' values to a line a
// 148-CTA all-reduce took 4-6 us, with one 2.0 us (against 2.4 us for a
// counter and separate partials).
// ORDERED: the CTA's earlier plain stores are made visible before the record
// (a fence) and the polls acquire, for kernels that exchange vectors by plain
// stores.
constexpr int REC_STRIDE = 8;    // TagVals per record: one 128-byte line
// Sums (and with MX the maximum) of the CTA: every lane of warp 0 returns
// value lane/8; send() is called there.
template <int NT, bool MX, typename F>
__device__ __forceinline__ void cta_reduce4(const double (&v)[4], F&& send)
{
    constexpr int NW = NT / 32;
    static_assert(NW == 8 || NW == 16, "warps per CTA");
    __shared__ double sm[4][NW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool h = lane & 16, e = lane & 8;
    const int q = lane >> 3;     // the value this lane ends up with
    const double v3 = MX ? v[3] : 0.0;
    double k0 = h ? v[2] : v[0], k1 = h ? v3 : v[1];
    const double x0 = __shfl_xor_sync(0xffffffffu, h ? v[0] : v[2], 16);
    const double x1 = __shfl_xor_sync(0xffffffffu, h ? v[1] : v3, 16);
    k0 += x0;
    k1 = red4<MX>(h ? 3 : 1, k1, x1);
    double k = e ? k1 : k0;
    k = red4<MX>(q, k, __shfl_xor_sync(0xffffffffu, e ? k0 : k1, 8));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) k = red4<MX>(q, k, __shfl_xor_sync(0xffffffffu, k, o));
    if ((lane & 7) == 0) sm[q][warp] = k;
    __syncthreads();
    if (warp == 0) {
        double x = sm[q][lane & 7];
        if (NW == 16) x = red4<MX>(q, x, sm[q][(lane & 7) + 8]);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) x = red4<MX>(q, x, __shfl_xor_sync(0xffffffffu, x, o));
        send(q, lane & 7, x);
    }
}
template <int NT, bool ORDERED, bool MX>
__device__ __forceinline__ void tag_allreduce_publish(const TagComm& c, int phase, const double (&v)[4])
{
    cta_reduce4<NT, MX>(v, [&](int q, int j, double x) {
        if (ORDERED) __threadfence();
        if (j == 0) st_tag(c.rec + ((phase & 1) * c.G + c.b) * REC_STRIDE + q, x, c.tag(phase));
    });
}

// Wait: thread t polls value t%4 of CTAs t/4, t/4 + NT/4, ...; lanes, then
// warps in a fixed order, so every CTA computes the same totals bit for bit.
// all_in() runs when every record has come in, before the last fold.  `ok`:
// false when an earlier wait of this thread gave up; the result is false for
// the whole CTA then, when this wait gives up, or when another CTA raised a
// status.
// A poll that comes before its record costs the record's writer a recall and
// the reader another round trip (24 CTAs: 4,150 cycles from the publish to
// the totals, 3,180 with the first poll held back by 1,200), so each warp
// holds its first poll back by `hold` cycles, adapted to the last exchanges:
// a little longer after a miss, a little shorter after a hit.
struct PollHold {
    unsigned cycles = 0;
    __device__ __forceinline__ void wait() const
    {
        const unsigned t0 = clock_lo();
        while (clock_lo() - t0 < cycles) {}
    }
    __device__ __forceinline__ void learn(bool missed)
    {
        if (__any_sync(0xffffffffu, missed)) cycles = cycles < 4096u ? cycles + 64u : cycles;
        else cycles = cycles > 16u ? cycles - 16u : 0u;
    }
    static __device__ __forceinline__ unsigned clock_lo()
    {
        unsigned t;
        asm volatile("mov.u32 %0, %%clock;" : "=r"(t));
        return t;
    }
};

// Records polled per thread, and the largest grid that covers: 256 CTAs of 512
// threads, 320 of 256.  A record past it would be left out of every sum, so the
// host keeps the grids of these kernels within it.
constexpr int tag_records(int nt) { return nt >= 512 ? 2 : 5; }
constexpr int tag_grid_max(int nt) { return tag_records(nt) * (nt / 4); }

template <int NT, bool ORDERED, bool MX, typename F>
__device__ __forceinline__ bool tag_allreduce_wait(const TagComm& c, int phase, double (&out)[4], bool ok, PollHold& hold,
                                                   F&& all_in)
{
    constexpr int NW = NT / 32, STEP = NT / 4;
    constexpr int MP = tag_records(NT);
    __shared__ double sm[NW][4];
    const int lane = threadIdx.x & 31, q = threadIdx.x & 3, j = threadIdx.x >> 2;
    const TagVal* r = c.rec + ((phase & 1) * c.G + j) * REC_STRIDE + q;
    const unsigned long long want = c.tag(phase);
    double a = 0.0;
    if ((j & ~7) < c.G) {        // this warp has records to poll
        double x[MP];
        unsigned long long t[MP];
        hold.wait();
        // every record requested before the first is looked at
        bool missed = false;
#pragma unroll
        for (int u = 0; u < MP; ++u) {
            x[u] = 0.0;
            t[u] = want;
            if (j + u * STEP < c.G) ld_tag<ORDERED>(r + u * STEP * REC_STRIDE, x[u], t[u]);
        }
#pragma unroll
        for (int u = 0; u < MP; ++u) missed = missed || t[u] != want;
        hold.learn(missed);
        if (missed) {
            SpinLimit lim;
#pragma unroll
            for (int u = 0; u < MP; ++u)
                while (t[u] != want) {
                    if (lim.expired(c.status)) { ok = false; break; }
                    ld_tag<ORDERED>(r + u * STEP * REC_STRIDE, x[u], t[u]);
                }
        }
        __syncwarp();
        a = x[0];
#pragma unroll
        for (int u = 1; u < MP; ++u) a = red4<MX>(q, a, x[u]);
#pragma unroll
        for (int o = 16; o >= 4; o >>= 1) a = red4<MX>(q, a, __shfl_xor_sync(0xffffffffu, a, o));
    }
    if (lane < 4) sm[threadIdx.x >> 5][lane] = a;
    ok = __syncthreads_and(ok);
    all_in();
    a = sm[lane >> 2][q];
    if (NW == 16) a = red4<MX>(q, a, sm[(lane >> 2) + 8][q]);
#pragma unroll
    for (int o = 16; o >= 4; o >>= 1) a = red4<MX>(q, a, __shfl_xor_sync(0xffffffffu, a, o));
#pragma unroll
    for (int p = 0; p < (MX ? 4 : 3); ++p) out[p] = __shfl_sync(0xffffffffu, a, p);
    if (!MX) out[3] = 0.0;
    return ok;
}

// Stopping test of the single-reduction kernels.  The exact test (a square
// root, a division, max|r|) is made only where it may hold: with test 2 not
// while (r,r) is above the square of rtol*||r0|| with a margin of 1e-12.
struct StopTest {
    int test;
    double rtol, atol, init, bound;
    __device__ __forceinline__ StopTest(const SegView& g, double init_)
        : test(g.conv_test), rtol(g.rel_tol), atol(g.abs_tol), init(init_)
    {
        const double x = g.rel_tol * init_;
        bound = x * x * (1.0 + 1.0e-12);
        // near underflow, or with a test on max|r|: always the exact test
        if (test != 2 || !(bound > 1.0e-280)) bound = __longlong_as_double(0x7ff0000000000000LL);
    }
    // the maximum is part of every iteration's all-reduce
    __device__ __forceinline__ bool needs_max() const { return test != 2; }
    // the iteration can go on without the exact test (a NaN or an infinite
    // (r,r) is not above the bound, or not below infinity)
    __device__ __forceinline__ bool clear(double rr) const { return rr > bound && rr < __longlong_as_double(0x7ff0000000000000LL); }
    __device__ __forceinline__ bool exact(double rr, double mx) const
    {
        return cg_converged(test, sqrt(rr) / init, mx, rtol, atol);
    }
};

// ------------------------------------------------------ cluster exchange
// Meshes whose rows fit one thread-block cluster exchange through the SMs'
// shared memory instead of L2: st.async writes a value into another CTA and
// counts its bytes on that CTA's mbarrier, so one wait on the CTA's own
// mbarrier covers the partial sums of every CTA and every neighbour value.
// Two mbarriers and two sets of buffers alternate by the exchange's parity,
// under the same rule as the tagged records.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, int rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_async_f64(uint32_t addr, double v, uint32_t bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, DevStatus* status)
{
    SpinLimit lim;
    while (!mbar_try_wait(bar, parity))
        if (lim.expired(status)) return false;
    return true;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// This CTA's side of a cluster's exchange.  In shared memory: two mbarriers
// and 2 x 16 x 4 partial sums.
constexpr int CLUSTER_MAX = 16;
struct ClusterShared {
    unsigned long long bar[2];
    double part[2][CLUSTER_MAX][4];
};

// ---------------------------------------------- tensor memory as storage
// The SM's 256 KB tensor memory (TMEM: 128 lanes x 512 columns of 32 bits)
// holds, for the whole solve, coefficients that would otherwise stream from
// L2 in every iteration.  No MMA touches it: it is read with tcgen05.ld into
// registers.  With the 32x32b access shape, warp w reads and writes lanes
// 32*(w%4) .. 32*(w%4)+31, one lane per thread, so the four warps that share
// a lane quarter split the 512 columns into four ranges of 128.  One warp
// allocates all 512 columns (one CTA per SM, nothing else in this library
// uses TMEM) and frees them before the CTA exits, on every path.
__device__ __forceinline__ void tmem_alloc_all(uint32_t* slot)
{
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(slot));
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(a) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free_all(uint32_t base)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(base) : "memory");
}
__device__ __forceinline__ void tmem_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// one double into two consecutive columns of this thread's lane (low word first)
__device__ __forceinline__ void tmem_st_f64(uint32_t addr, double v)
{
    const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v));
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(addr),
                 "r"(static_cast<uint32_t>(b)), "r"(static_cast<uint32_t>(b >> 32))
                 : "memory");
}
__device__ __forceinline__ void tmem_st_b32(uint32_t addr, uint32_t v)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// N consecutive 32-bit columns of this thread's lane; the registers are
// undefined until tmem_wait_ld, after which tmem_hold pins their uses
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t addr, uint32_t (&r)[N]);
template <>
__device__ __forceinline__ void tmem_ld<4>(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
template <>
__device__ __forceinline__ void tmem_ld<16>(uint32_t addr, uint32_t (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
                   "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// after tmem_wait_ld: an empty statement that "rewrites" the loaded registers,
// so no use of them can be scheduled before the wait
template <int N>
__device__ __forceinline__ void tmem_hold(uint32_t (&r)[N])
{
#pragma unroll
    for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]));
}

// ------------------------------------ global-vector single-reduction PCG
// The Chronopoulos-Gear iteration of k_pcg64c for meshes whose rows do not
// fit the register tiling: the rows' r, s, w (double-buffered by iteration
// parity), direction p and pressure stay in global memory, and every CTA
// stages, per part of its slices, the new z of its halo into shared memory
// from the previous iteration's r, w, s and the inverse diagonal -- the same
// operations the owner applies to its rows.  One grid all-reduce per
// iteration (k_pcg64 takes two) and no separate vector-update pass.  The
// search direction lives in the engine's permuted right-hand side, which is
// dead once r0 is formed.  Where the whole halo fits (one part) the inverse
// diagonal of the halo stays in shared memory for the solve.
//
// Bound by memory traffic (96^3: 248 MB per iteration, more than L2 holds)
// and, with one row per lane at a time, by the latency of a row's loads: so a
// warp requests the first 16 slots of its next streamed row while it works on
// the present one (into the registers just consumed), and the SM's tensor
// memory keeps the coefficients and local columns of D.tm_rows of its rows
// (three of Kuhn meshes' 14 slots) for the solve.  Those alternate with the
// streamed ones, so that memory stays busy while they are processed: four of
// them ahead of the streamed rows took 88^3 from 31.5 to 33.7 us.
__device__ __forceinline__ void pcg64g_body(const PcgDev& D, uint32_t tm, unsigned long long epoch)
{
    constexpr int NT = PCG_THREADS;
    const SegView g = seg_view<false>(D);
    const int G = g.G, b = g.b;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s_beg = g.s0 + (int)((long long)b * (g.s1 - g.s0) / G);
    const int s_end = g.s0 + (int)((long long)(b + 1) * (g.s1 - g.s0) / G);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int KP = D.halo_parts > 0 ? D.halo_parts : 1;
    const bool dzres = KP == 1;   // the halo's inverse diagonal resident in shared memory
    double* vh = reinterpret_cast<double*>(smem_raw);
    double* dzh = vh + D.halo_max;
    const TagComm comm = tag_comm(D, g, epoch);
    PollHold hold;
    int phase = 0;
    const int N = D.N;
    double* rb[2] = {D.r, D.r + N};
    double* wb[2] = {D.q, D.q + N};
    double* sb[2] = {D.pA, D.pB};
    double* dz = D.z;     // free ? 1/diagonal : 0  (z = r * dz)
    double* pv = D.rhs1;  // search direction (after r0)

    // halo of part q: h0, nh
    auto halo_of = [&](int q, int& h0, int& nh) {
        h0 = D.halo_ptr[b * KP + q];
        nh = D.halo_ptr[b * KP + q + 1] - h0;
    };
    // first slot (from the CTA's first) and width of the CTA's slices
    int2* meta = reinterpret_cast<int2*>(smem_raw + D.lcs_off);
    const long long S0 = D.slice_off[s_beg];
    for (int k = threadIdx.x; k < s_end - s_beg; k += NT) meta[k] = make_int2((int)(D.slice_off[s_beg + k] - S0), D.slice_w[s_beg + k]);
    __syncthreads();
    const double* vbase = D.val + S0 + lane;
    const unsigned short* cbase = D.lcol + S0 + lane;
    // The warp's rows of part q are slices ps0 + warp + 16*i; row i is in
    // tensor memory when i is even and fewer than tm_rows rows came before.
    // The t-th row there: columns TC*t .. of lane 32*(warp%4)+lane, from
    // 128*(warp/4) on: tm_w doubles, then tm_w/2 words of two local columns.
    const uint32_t tm0 = tm + (static_cast<uint32_t>(32 * (warp & 3)) << 16) + static_cast<uint32_t>(128 * (warp >> 2));
    const int TC = 2 * D.tm_w + D.tm_w / 2;
    auto part_slices = [&](int part, int& ps0, int& n) {
        ps0 = s_beg + (int)((long long)part * (s_end - s_beg) / KP) + warp;
        const int ps1 = s_beg + (int)((long long)(part + 1) * (s_end - s_beg) / KP);
        n = ps1 > ps0 ? (ps1 - ps0 + PCG_WARPS - 1) / PCG_WARPS : 0;
    };
    auto tm_used = [&](int t0, int n) { const int e = (n + 1) / 2, f = D.tm_rows - t0; return e < f ? e : f; };
    for (int part = 0, t0 = 0; part < KP; ++part) {
        int ps0, n;
        part_slices(part, ps0, n);
        const int nt = tm_used(t0, n);
        for (int t = 0; t < nt; ++t) {
            const int2 m = meta[ps0 + 2 * t * PCG_WARPS - s_beg];
            const uint32_t at = tm0 + TC * (t0 + t);
            for (int u = 0; u < D.tm_w; u += 2) {
                const bool h0 = u < m.y, h1 = u + 1 < m.y;
                tmem_st_f64(at + 2 * u, h0 ? __ldcs(vbase + m.x + 32 * u) : 0.0);
                tmem_st_f64(at + 2 * u + 2, h1 ? __ldcs(vbase + m.x + 32 * u + 32) : 0.0);
                const unsigned lo = h0 ? __ldcs(cbase + m.x + 32 * u) : 0, hi = h1 ? __ldcs(cbase + m.x + 32 * u + 32) : 0;
                tmem_st_b32(at + 2 * D.tm_w + u / 2, lo | hi << 16);
            }
        }
        t0 += nt;
    }
    if (D.tm_rows) tmem_wait_st();
    // Every row of a part, in order: pre(i) (loads the row's vectors), the
    // off-diagonal sum over the staged halo (the slots in order), post(i, sum)
    auto rows = [&](int part, int t0, auto&& pre, auto&& post) {
        constexpr int CH = 8, PH = 2;    // slots per round, rounds requested ahead
        int ps0, n;
        part_slices(part, ps0, n);
        auto in_tm = [&](int i) { return !(i & 1) && t0 + (i >> 1) < D.tm_rows; };
        double v[PH][CH];
        int c[PH][CH];
        auto request = [&](int h, const int2& m) {
#pragma unroll
            for (int u = 0; u < CH; ++u) {
                const int k = CH * h + u;
                v[h][u] = k < m.y ? __ldcs(vbase + m.x + 32 * k) : 0.0;
                c[h][u] = k < m.y ? (int)__ldcs(cbase + m.x + 32 * k) : 0;
            }
        };
        int nx = in_tm(0) ? 1 : 0;       // next streamed row
        if (nx < n) {
            const int2 m = meta[ps0 + nx * PCG_WARPS - s_beg];
#pragma unroll
            for (int h = 0; h < PH; ++h) request(h, m);
        }
        for (int i = 0; i < n; ++i) {
            const int s = ps0 + i * PCG_WARPS;
            const int2 m = meta[s - s_beg];
            pre(s * 32 + lane);
            double off = 0.0;
            if (i == nx) {
                nx = in_tm(i + 1) ? i + 2 : i + 1;
                const int2 mn = nx < n ? meta[ps0 + nx * PCG_WARPS - s_beg] : make_int2(0, 0);
#pragma unroll
                for (int h = 0; h < PH; ++h) {
                    double x[CH];
#pragma unroll
                    for (int u = 0; u < CH; ++u) x[u] = vh[c[h][u]];
#pragma unroll
                    for (int u = 0; u < CH; ++u)
                        if (CH * h + u < m.y) off = fma(v[h][u], x[u], off);
                    request(h, mn);
                }
                for (int k = PH * CH; k < m.y; ++k)
                    off = fma(__ldcs(vbase + m.x + 32 * k), vh[__ldcs(cbase + m.x + 32 * k)], off);
            } else {
                const uint32_t at = tm0 + TC * (t0 + (i >> 1));
                for (int k0 = 0; k0 < m.y; k0 += CH) {
                    uint32_t tv[2 * CH], tc[CH / 2];
                    tmem_ld<CH / 2>(at + 2 * D.tm_w + k0 / 2, tc);
                    tmem_ld<2 * CH>(at + 2 * k0, tv);
                    tmem_wait_ld();
                    tmem_hold<CH / 2>(tc);
                    tmem_hold<2 * CH>(tv);
                    double x[CH];
#pragma unroll
                    for (int u = 0; u < CH; ++u) x[u] = vh[u & 1 ? tc[u / 2] >> 16 : tc[u / 2] & 0xffffu];
#pragma unroll
                    for (int u = 0; u < CH; ++u)
                        if (k0 + u < m.y)
                            off = fma(__hiloint2double(static_cast<int>(tv[2 * u + 1]), static_cast<int>(tv[2 * u])), x[u], off);
                }
            }
            post(s * 32 + lane, off);
        }
        return t0 + tm_used(t0, n);
    };

    double t[4];
    auto allreduce = [&](const double (&v)[4], bool with_max) {
        bool ok;
        if (with_max) {
            tag_allreduce_publish<NT, true, true>(comm, phase, v);
            ok = tag_allreduce_wait<NT, true, true>(comm, phase, t, true, hold, [] {});
        } else {
            tag_allreduce_publish<NT, true, false>(comm, phase, v);
            ok = tag_allreduce_wait<NT, true, false>(comm, phase, t, true, hold, [] {});
        }
        ++phase;
        return ok;
    };
    // ---- phase 0a: r0 = b - A x0 (constraints as the reference), dz, p = s = 0;
    // partials: invalid diagonals, non-finite residuals, (r,r), max|r|
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int part = 0, q = 0; part < KP; ++part) {
        int h0, nh;
        halo_of(part, h0, nh);
        __syncthreads();
        for (int k = threadIdx.x; k < nh; k += NT) vh[k] = __ldcg(D.pres + D.halo_idx[h0 + k]);
        __syncthreads();
        q = rows(part, q, [](int) {}, [&](int i, double off) {
            const uint8_t f = D.nflag[i];
            const bool active = f & 1, fr = (f & 1) && !(f & 4);
            const double pd = D.pdiag[i];
            const double y = fma(pd, D.pres[i], off);
            double ri = active ? D.rhs1[i] - y : 0.0;
            double dd = 0.0;
            if (!fr) ri = 0.0;
            if (fr) {
                if (g.precond) {
                    if (!(isfinite(pd) && pd > 1.0e-30)) acc[0] += 1.0;
                    dd = 1.0 / pd;
                } else {
                    dd = 1.0;
                }
                if (!isfinite(ri)) acc[1] += 1.0;
                acc[2] = fma(ri, ri, acc[2]);
                acc[3] = max_bits(acc[3], fabs(ri));
            }
            rb[0][i] = ri;
            dz[i] = dd;
            sb[0][i] = 0.0;
        });
    }
    if (!allreduce(acc, true)) return;
    const double init = sqrt(t[2]);
    if (init <= 1.0e-300) { cg_finish(D, g, 0, 1, init, init, 0.0, t[3]); return; }
    if (cg_converged(g.conv_test, 1.0, t[3], g.rel_tol, g.abs_tol)) { cg_finish(D, g, 0, 1, init, init, 1.0, t[3]); return; }
    if (t[1] > 0.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, 0, R_PCG_RESID); return; }
    if (t[0] > 0.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 1, ST_PCG, 0, R_PCG_DIAG); return; }
    const StopTest stop(g, init);

    // ---- phase 0b: z0 = M^-1 r0, w0 = A z0, gamma0 = (r0,z0), delta0 = (z0,w0);
    // the right-hand side is no longer needed: p = 0 from here
    acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
    for (int part = 0, q = 0; part < KP; ++part) {
        int h0, nh;
        halo_of(part, h0, nh);
        __syncthreads();
        for (int k = threadIdx.x; k < nh; k += NT) {
            const int j = D.halo_idx[h0 + k];
            const double dj = __ldcg(dz + j);
            if (dzres) dzh[k] = dj;
            vh[k] = __ldcg(rb[0] + j) * dj;
        }
        __syncthreads();
        q = rows(part, q, [](int) {}, [&](int i, double off) {
            const uint8_t f = D.nflag[i];
            const bool fr = (f & 1) && !(f & 4);
            const double ri = rb[0][i];
            const double zi = ri * dz[i];
            const double wi = fr ? fma(D.pdiag[i], zi, off) : 0.0;
            wb[0][i] = wi;
            pv[i] = 0.0;
            if (fr) {
                acc[0] = fma(ri, zi, acc[0]);
                acc[1] = fma(zi, wi, acc[1]);
            }
        });
    }
    if (!allreduce(acc, false)) return;
    double gam = t[0];
    if (gam <= 1.0e-300 || !isfinite(gam)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, 0, R_PCG_RZ0); return; }
    double den = t[1];
    double beta = 0.0, rr = t[2], mx = 0.0, alpha = 0.0;
    int it = 0, conv = 0;
    for (it = 1; it <= g.max_iter; ++it) {
        if (fabs(den) <= 1.0e-300 || !isfinite(den)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_PAP); return; }
        alpha = gam / den;
        const int po = (it - 1) & 1, pn = it & 1;
        const double* so = sb[po];
        const double* wo = wb[po];
        const double* ro = rb[po];
        acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
        for (int part = 0, q = 0; part < KP; ++part) {
            int h0, nh;
            halo_of(part, h0, nh);
            // stage z_it of the halo: s = w_o + beta*s_o, r = r_o - alpha*s,
            // z = r * dz (SU nodes per thread per round, all loads first); the
            // all-reduce (or the previous part) ended with a barrier
            {
                constexpr int SU = 4;
                __syncthreads();
                for (int k0 = threadIdx.x; k0 < nh; k0 += SU * NT) {
                    double a[SU], c[SU], e[SU], d[SU];
#pragma unroll
                    for (int u = 0; u < SU; ++u) {
                        const int k = k0 + u * NT;
                        const int j = k < nh ? D.halo_idx[h0 + k] : 0;
                        a[u] = __ldcg(so + j);
                        c[u] = __ldcg(wo + j);
                        e[u] = __ldcg(ro + j);
                        d[u] = dzres ? 0.0 : __ldcg(dz + j);
                    }
#pragma unroll
                    for (int u = 0; u < SU; ++u) {
                        const int k = k0 + u * NT;
                        if (k < nh) {
                            const double sj = fma(beta, a[u], c[u]);
                            const double rj = fma(-alpha, sj, e[u]);
                            vh[k] = rj * (dzres ? dzh[k] : d[u]);
                        }
                    }
                }
                __syncthreads();
            }
            // own rows: p = z_o + beta*p, s = w_o + beta*s_o, x += alpha*p,
            // r = r_o - alpha*s; then w = A z, the partials
            uint8_t f;
            double r_o, s_o, w_o, dd, p_o, x_o, pd;
            q = rows(part, q, [&](int i) {
                f = D.nflag[i];
                r_o = ro[i], s_o = so[i], w_o = wo[i], dd = dz[i];
                p_o = pv[i], x_o = D.pres[i], pd = D.pdiag[i];
            }, [&](int i, double off) {
                const bool fr = (f & 1) && !(f & 4);
                const double zo = r_o * dd;
                const double pi = fr ? fma(beta, p_o, zo) : 0.0;
                const double si = fma(beta, s_o, w_o);
                if (fr) D.pres[i] = fma(alpha, pi, x_o);
                const double ri = fma(-alpha, si, r_o);
                pv[i] = pi;
                rb[pn][i] = ri;
                sb[pn][i] = si;
                const double zi = ri * dd;
                const double wi = fr ? fma(pd, zi, off) : 0.0;
                wb[pn][i] = wi;
                if (fr) {
                    acc[0] = fma(ri, zi, acc[0]);
                    acc[1] = fma(zi, wi, acc[1]);
                    acc[2] = fma(ri, ri, acc[2]);
                    acc[3] = max_bits(acc[3], fabs(ri));
                }
            });
        }
        if (!allreduce(acc, stop.needs_max())) return;
        rr = t[2];
        mx = t[3];
        const double gn = t[0], delta = t[1];
        if (!stop.clear(rr) || gn <= 1.0e-300 || !isfinite(gn)) {
            if (!stop.needs_max()) {
                acc[0] = acc[1] = acc[2] = 0.0;
                if (!allreduce(acc, true)) return;
                mx = t[3];
            }
            if (stop.exact(rr, mx)) { conv = 1; break; }
            if (!isfinite(mx)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, it, R_PCG_RESID); return; }
            if (gn <= 1.0e-300 || !isfinite(gn)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_RZ); return; }
        }
        beta = gn / gam;
        den = fma(-beta * beta, den, delta);
        gam = gn;
    }
    if (!conv && !stop.needs_max()) {
        acc[0] = acc[1] = acc[2] = 0.0;
        if (!allreduce(acc, true)) return;
        mx = t[3];
    }
    if (it > g.max_iter) it = g.max_iter;
    cg_finish(D, g, it, conv, init, sqrt(rr), sqrt(rr) / init, mx);
    if (!conv && b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 2, ST_PCG, it, R_PCG_MAXIT);
}

// The epoch of this solve, and whether an earlier stage has already failed
// (then no CTA starts); after the solve the next one's epoch.  CTA 0 cannot
// get past its first all-reduce, let alone here, before every CTA has read
// the epoch.
template <bool BATCH>
__device__ __forceinline__ bool tag_begin(const PcgDev& D, unsigned long long& epoch)
{
    const SegView g = seg_view<BATCH>(D);
    epoch = *seg_epoch(D, g) << 32;
    return !__syncthreads_or(threadIdx.x == 0 && ld_relaxed_int(&seg_status(D, g)->code) != 0);
}
template <bool BATCH>
__device__ __forceinline__ void tag_end(const PcgDev& D, unsigned long long epoch)
{
    const SegView g = seg_view<BATCH>(D);
    if (g.b == 0 && threadIdx.x == 0) *seg_epoch(D, g) = (epoch >> 32) + 1;
}

// one CTA per SM: with rows in tensor memory warp 0 takes all of it before
// the solve and returns it after, every exit of the body being CTA-uniform
__global__ void __launch_bounds__(PCG_THREADS, PCG_CTAS_PER_SM) k_pcg64g(PcgDev D)
{
    unsigned long long epoch;
    if (!tag_begin<false>(D, epoch)) return;
    __shared__ uint32_t s_tm;
    const bool w0 = (threadIdx.x >> 5) == 0;
    if (w0 && D.tm_rows) tmem_alloc_all(&s_tm);
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    const uint32_t tm = D.tm_rows ? s_tm : 0u;
    pcg64g_body(D, tm, epoch);
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    if (w0 && D.tm_rows) tmem_free_all(tm);
    tag_end<false>(D, epoch);
}

// The single-reduction iteration with the rows' vectors in registers.  Row by
// row it performs the operations of pcg64g_body in the same order.
//
// Exchange.  A CTA keeps the neighbour values that other CTAs own ("remote"
// entries of its halo) up to date itself: r and s of those rows follow the
// same recurrences from the same alpha, beta as at their owners, so the only
// vector that crosses CTAs is w, one tagged record per row and iteration
// (staging r, s and w cost three values and a second trip to L2 after the
// all-reduce).  The records are requested when the other CTAs' partials have
// come in -- a CTA stores its w before its partials, so they are there, and
// polling them earlier would slow their stores -- and travel while the
// partials are folded; neither exchange needs a fence.  The own rows' new z go
// from registers into the halo.
//
// Bound at 64^3 (13,700 cycles per iteration): instruction issue (44% of the
// cycles), the shared-memory wavefronts (5,630 per CTA and iteration, about
// 3,280 of them the gathers) and the latency of the all-reduce.
//
// KT > 0: the coefficients of each thread's rows KS .. KS+KT-1 live in TMEM
// for the solve (D.tm_w slots per row, zero-padded past the slice's width);
// `tm` is the CTA's TMEM base address (0 when KT = 0).
//
// RG: for CTAs whose halo is mostly remote (thin meshes, orders without
// coordinates) the 30 bytes per remote entry do not fit beside the halo.
// Their positions, places and inverse diagonals are then read from global
// memory as one 16-byte record each, r and s stay in shared memory where those
// fit (else in global memory too, always touched by the same thread), the
// local columns are places instead of byte offsets (halos up to 65,534), and
// slots past tm_w stream from L2, so that every mesh the halo itself fits for
// has this kernel.
template <int RMAX, bool BATCH, int NT, int KS, int KT, bool CL, bool RG>
__device__ __forceinline__ void pcg64c_body(const PcgDev& D, uint32_t tm, unsigned long long epoch)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const SegView g = seg_view<BATCH>(D);
    const TagComm comm = tag_comm(D, g, epoch);
    PollHold hold;
    const int G = g.G, b = g.b;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s_beg = g.s0 + (int)((long long)b * (g.s1 - g.s0) / G);
    const int s_end = g.s0 + (int)((long long)(b + 1) * (g.s1 - g.s0) / G);
    const long long S0 = D.slice_off[s_beg];
    const int h0 = D.halo_ptr[blockIdx.x];
    const int nh = D.halo_ptr[blockIdx.x + 1] - h0;
    const int q0 = D.rem_ptr[blockIdx.x];
    const int nr = D.rem_ptr[blockIdx.x + 1] - q0;
    double* vh = reinterpret_cast<double*>(smem_raw);          // halo_max: z of every column, and one spare
    double* rh = vh + D.halo_max;                              // rem_max: r, s, inverse diagonal of the remote ones
    double* sh = rh + D.rem_max;
    double* dzh = sh + D.rem_max;
    int* rgi = reinterpret_cast<int*>(dzh + D.rem_max);        // rem_max: their row positions
    unsigned short* rhp = reinterpret_cast<unsigned short*>(rgi + D.rem_max);   // ... and places in vh
    RemoteState* rst = nullptr;
    if constexpr (RG) {
        rst = D.rem_state + q0;
        rh = D.rs_off ? reinterpret_cast<double*>(smem_raw + D.rs_off) : D.rem_rs + 2 * (size_t)q0;
        sh = rh + (D.rs_off ? D.rem_max : nr);
    }
    // the own rows' diagonal, kept in shared memory for the solve where the
    // engine sized it so
    double* pds = NT == 512 && D.pds_off ? reinterpret_cast<double*>(smem_raw + D.pds_off) : nullptr;
    for (int k = threadIdx.x; k < nr; k += NT) {
        const int2 e = D.rem[q0 + k];
        const uint8_t f = D.nflag[e.x];
        const double dj = (f & 1) && !(f & 4) ? (g.precond ? 1.0 / D.pdiag[e.x] : 1.0) : 0.0;
        if constexpr (RG) {
            rst[k].dz = dj;
        } else {
            if (!CL) rgi[k] = e.x;
            rhp[k] = (unsigned short)e.y;
            dzh[k] = dj;
        }
        sh[k] = 0.0;
    }
    // place and inverse diagonal of remote entry e
    auto remote = [&](int e, int& place, double& dj) {
        if constexpr (RG) {
            const RemoteState x = rst[e];
            place = x.place;
            dj = x.dz;
        } else {
            place = rhp[e];
            dj = dzh[e];
        }
    };
    // CL: the exchange through the cluster's shared memory.  cwx: 2 x rem_max
    // values of the remote entries, as their owners push them; cwo: the own
    // rows' value; cpu, cpl: where each pushed value goes (in the consumer's
    // first buffer) and consumer << 12 | own row.
    static_assert(!CL || RMAX * NT <= 4096, "own rows in 12 bits");
    __shared__ ClusterShared cs;
    double* cwx = reinterpret_cast<double*>(smem_raw + D.cl_off);
    double* cwo = cwx + 2 * D.rem_max;
    uint32_t* cpu = reinterpret_cast<uint32_t*>(cwo + RMAX * NT);
    unsigned short* cpl = reinterpret_cast<unsigned short*>(cpu + D.push_max);
    int npush = 0;
    if constexpr (CL) {
        const int p0 = D.push_ptr[b];
        npush = D.push_ptr[b + 1] - p0;
        for (int k = threadIdx.x; k < npush; k += NT) {
            const int2 e = D.push[p0 + k];     // own row, consumer << 16 | entry
            cpu[k] = cluster_addr(smem_addr(cwx + (e.y & 0xffff)), e.y >> 16);
            cpl[k] = (unsigned short)(e.x | (e.y >> 16) << 12);
        }
        for (int k = threadIdx.x; k < 2 * CLUSTER_MAX * 4; k += NT) (&cs.part[0][0][0])[k] = 0.0;
        if (threadIdx.x < 2) mbar_init(smem_addr(&cs.bar[threadIdx.x]));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        cluster_sync();          // every CTA is there, its mbarriers ready
    }
    // KS = 1: the coefficients of every warp's first row (the CTA's first
    // NT/32 slices, its leading slots) copied once into shared memory and
    // read from there in every iteration instead of from L2
    double* cvs = reinterpret_cast<double*>(smem_raw + D.coef_off);
    if constexpr (KS > 0) {
        const int sc = s_beg + (NT / 32) * KS < s_end ? s_beg + (NT / 32) * KS : s_end;
        const int c0 = (int)(D.slice_off[sc] - S0);
        for (int k = threadIdx.x; k < c0; k += NT) cvs[k] = __ldcg(D.val + S0 + k);
    }
    int phase = 0;

    // the own rows (row k of this thread is row0 + k*NT): r, p, s, w and the
    // reciprocal of the Jacobi diagonal (0 off the free rows) in registers
    // for the solve.  Rows off the free ones, and the empty rows of a short
    // warp, have r = dd = 0 and stay 0 without branches.
    double r[RMAX], p[RMAX], s[RMAX], w[RMAX], dd[RMAX];
    // Registers bound the kernel (128 at 512 threads).  Past four rows per
    // thread p and the pressure live in memory: the pressure in shared memory
    // where that has room (else global; both at the rows' distance NT),
    // updated once the CTA's partials are on their way, and p in global
    // memory except from there to the next update.  At three rows the
    // pressure in shared memory measured faster (56^3: 4.82 us per iteration
    // against 4.99), at four slower (64^3: 7.45 against 7.16).
    constexpr bool XM = RMAX == 3 || RMAX > 4, PM = RMAX > 4;
    double xr[XM ? 1 : RMAX];
    const int row0 = (s_beg + warp) * 32 + lane;
    // per row: place of its z in vh (the last, unused one where it is no
    // column of this CTA), whether other CTAs read it, whether it is free
    constexpr int PLACE = 0xffff, PUB = 1 << 16, FREE = 1 << 17;
    int own[RMAX], lbase[RMAX], wr[RMAX];
    int wmax = 0, nk = 0;        // the warp's widest row and its rows (uniform)
#pragma unroll
    for (int k = 0; k < RMAX; ++k) {
        const int sl = s_beg + warp + (NT / 32) * k;
        lbase[k] = 0;
        wr[k] = 0;
        own[k] = D.halo_max - 1;
        if (sl < s_end) {
            ++nk;
            lbase[k] = (int)(D.slice_off[sl] - S0) + lane;
            wr[k] = D.slice_w[sl];
            wmax = wr[k] > wmax ? wr[k] : wmax;
            const int o = D.own[row0 + k * NT];
            own[k] = (o & PUB) | ((o & PLACE) == PLACE ? D.halo_max - 1 : (o & PLACE));
        }
        r[k] = p[k] = s[k] = w[k] = 0.0;
        dd[k] = 0.0;
    }
    double* xs = !XM ? nullptr
               : D.xs_off ? reinterpret_cast<double*>(smem_raw + D.xs_off) + threadIdx.x : D.pres + row0;
    double* ps = PM ? D.pA + row0 : nullptr;
    // slots per round
    constexpr int CH = CGCG_ROUND;
    // one row per thread: the first RW slots' coefficients and local columns
    // in registers for the solve
    constexpr int RW = RMAX == 1 ? 16 : 0;
    static_assert(RMAX > 1 || (KS == 0 && KT == 0), "one row needs no other place for its coefficients");
    static_assert(KT == 0 || KS + KT <= RMAX, "TMEM rows follow the shared-memory rows");
    // rows past the tensor memory's: their coefficients stream from L2, the
    // first XW slots of one row requested together (one row's before the
    // barrier ahead of the products)
    constexpr int KX = KT > 0 ? RMAX - KS - KT : 0, XW = 16;
    // The warp's local columns, as byte offsets into vh, two slots to a word:
    // word j of row k is at lcp[(k * wmax/2 + j) * 32].  Every row of a warp
    // is padded to the warp's widest (rounded up to CH) with a column whose
    // coefficient is zero, so the rounds carry no guards.  (A non-finite z in
    // such a column can only come with a non-finite residual or r.z, which
    // end the solve in the same iteration.)
    wmax = (wmax + CH - 1) / CH * CH;
    const unsigned* lcp;
    {
        __shared__ int s_words[NT / 32];
        if (lane == 0) s_words[warp] = nk * (wmax / 2) * 32;
        __syncthreads();
        int o = 0;
        for (int q = 0; q < warp; ++q) o += s_words[q];
        unsigned* mine = reinterpret_cast<unsigned*>(smem_raw + D.lcs_off) + o + lane;
        for (int k = 0; k < nk; ++k) {
            const unsigned short* src = D.lcol + S0 + lbase[k];
            const unsigned pad = wr[k] > 0 ? src[0] : 0;
            for (int j = 0; j < wmax / 2; ++j) {
                const unsigned lo = 2 * j < wr[k] ? src[64 * j] : pad, hi = 2 * j + 1 < wr[k] ? src[64 * j + 32] : pad;
                mine[(k * (wmax / 2) + j) * 32] = RG ? lo | hi << 16 : lo * 8 | hi * 8 << 16;
            }
        }
        lcp = mine;
    }
    // TMEM rows: row KS+q of this thread starts at column
    // 128*(warp/4) + 2*tm_w*q of lane 32*(warp%4)+lane; slot u of the row is
    // the double in columns 2u, 2u+1.  Every warp runs the same (uniform)
    // loops here, as the .sync.aligned forms require.
    uint32_t tmr[KT > 0 ? KT : 1];
    if constexpr (KT > 0) {
        const int tw = D.tm_w;
        const uint32_t wb0 = tm + (static_cast<uint32_t>(32 * (warp & 3)) << 16) + static_cast<uint32_t>(128 * (warp >> 2));
#pragma unroll
        for (int q = 0; q < KT; ++q) {
            tmr[q] = wb0 + static_cast<uint32_t>(2 * tw * q);
            const int k = KS + q;
            for (int u = 0; u < tw; ++u) {
                const double c = (u < wr[k]) ? __ldcg(D.val + S0 + lbase[k] + 32 * u) : 0.0;
                tmem_st_f64(tmr[q] + 2 * u, c);
            }
        }
        tmem_wait_st();
    }
    double vrow[RW > 0 ? RW : 1];
    unsigned crow[RW > 0 ? RW / 2 : 1];
    if constexpr (RW > 0) {
#pragma unroll
        for (int u = 0; u < RW; ++u) vrow[u] = u < wr[0] ? __ldcg(D.val + S0 + lbase[0] + 32 * u) : 0.0;
#pragma unroll
        for (int j = 0; j < RW / 2; ++j) crow[j] = 2 * j < wmax ? lcp[j * 32] : 0;
    }
    double vx[KX > 0 ? XW : 1];
    auto extra_load = [&](int k) {
#pragma unroll
        for (int u = 0; u < XW; ++u) vx[u] = u < wr[k] ? __ldcg(D.val + S0 + lbase[k] + 32 * u) : 0.0;
    };
    // z at a local column
    auto zcol = [&](unsigned c) -> double {
        if constexpr (RG) return vh[c];
        else return *reinterpret_cast<const double*>(smem_raw + c);
    };
    auto offdiag_all = [&](double* off) {
#pragma unroll
        for (int k = 0; k < RMAX; ++k) off[k] = 0.0;
        if constexpr (RW > 0) {
#pragma unroll
            for (int j = 0; j < RW / 2; ++j)
                if (2 * j < wmax) {
                    const double x0 = zcol(crow[j] & 0xffffu);
                    const double x1 = zcol(crow[j] >> 16);
                    off[0] = fma(vrow[2 * j], x0, off[0]);
                    off[0] = fma(vrow[2 * j + 1], x1, off[0]);
                }
            for (int u = RW; u < wr[0]; ++u) {
                const unsigned c = lcp[(u >> 1) * 32] >> (16 * (u & 1));
                off[0] = fma(__ldcg(D.val + S0 + lbase[0] + 32 * u),
                             zcol(c & 0xffffu), off[0]);
            }
            return;
        }
        const unsigned* lc = lcp;
        const int wt = RG && KT > 0 ? min(wmax, D.tm_w) : wmax;
        for (int k0 = 0; k0 < wt; k0 += CH, lc += CH / 2 * 32) {
            double v[RMAX][CH], x[RMAX][CH];
            uint32_t tv[KT > 0 ? KT : 1][2 * CH];
            if constexpr (KT > 0) {
#pragma unroll
                for (int q = 0; q < KT; ++q) tmem_ld<2 * CH>(tmr[q] + 2 * k0, tv[q]);
            }
#pragma unroll
            for (int k = 0; k < RMAX; ++k) {
                if (k >= KS && (KT > 0 || k < KS + KT)) continue;
#pragma unroll
                for (int u = 0; u < CH; ++u)
                    v[k][u] = (k0 + u < wr[k]) ? (k < KS ? cvs[lbase[k] + 32 * (k0 + u)]
                                                         : __ldcg(D.val + S0 + lbase[k] + 32 * (k0 + u)))
                                               : 0.0;
            }
#pragma unroll
            for (int k = 0; k < RMAX - KX; ++k)
                if (k < nk) {
#pragma unroll
                    for (int j = 0; j < CH / 2; ++j) {
                        const unsigned c = lc[(k * (wmax / 2) + j) * 32];
                        x[k][2 * j] = zcol(c & 0xffffu);
                        x[k][2 * j + 1] = zcol(c >> 16);
                    }
                }
            if constexpr (KT > 0) {
                tmem_wait_ld();
#pragma unroll
                for (int q = 0; q < KT; ++q) {
                    tmem_hold<2 * CH>(tv[q]);
#pragma unroll
                    for (int u = 0; u < CH; ++u)
                        v[KS + q][u] = __hiloint2double(static_cast<int>(tv[q][2 * u + 1]), static_cast<int>(tv[q][2 * u]));
                }
            }
#pragma unroll
            for (int k = 0; k < RMAX - KX; ++k)
                if (k < nk) {
#pragma unroll
                    for (int u = 0; u < CH; ++u) off[k] = fma(v[k][u], x[k][u], off[k]);
                }
        }
        if constexpr (RG && KT > 0) {
            for (int k0 = wt; k0 < wmax; k0 += CH, lc += CH / 2 * 32)
#pragma unroll
                for (int k = 0; k < RMAX - KX; ++k)
                    if (k < nk) {
                        double v[CH];
#pragma unroll
                        for (int u = 0; u < CH; ++u)
                            v[u] = k0 + u < wr[k] ? __ldcg(D.val + S0 + lbase[k] + 32 * (k0 + u)) : 0.0;
#pragma unroll
                        for (int j = 0; j < CH / 2; ++j) {
                            const unsigned c = lc[(k * (wmax / 2) + j) * 32];
                            off[k] = fma(v[2 * j], zcol(c & 0xffffu), off[k]);
                            off[k] = fma(v[2 * j + 1], zcol(c >> 16), off[k]);
                        }
                    }
        }
        if constexpr (KX > 0) {
#pragma unroll
            for (int k = RMAX - KX; k < RMAX; ++k)
                if (k < nk) {
                    if (k > RMAX - KX) extra_load(k);
                    const unsigned* lx = lcp + k * (wmax / 2) * 32;
#pragma unroll
                    for (int j = 0; j < XW / 2; ++j)
                        if (2 * j < wmax) {
                            const unsigned c = lx[j * 32];
                            off[k] = fma(vx[2 * j], zcol(c & 0xffffu), off[k]);
                            off[k] = fma(vx[2 * j + 1], zcol(c >> 16), off[k]);
                        }
                    for (int u = XW; u < wr[k]; ++u) {
                        const unsigned c = lx[(u >> 1) * 32] >> (16 * (u & 1));
                        off[k] = fma(__ldcg(D.val + S0 + lbase[k] + 32 * u),
                                     zcol(c & 0xffffu), off[k]);
                    }
                }
        }
    };
    auto extra_first = [&]() {
        if constexpr (KX > 0)
            if (RMAX - KX < nk) extra_load(RMAX - KX);
    };

    auto diag = [&](int k) -> double {
        return pds ? pds[k * NT + threadIdx.x] : (k < nk ? D.pdiag[row0 + k * NT] : 0.0);
    };

    // exchange of one value per row (exchange number `phase`): the rows that
    // other CTAs read are stored as records; the first RP remote entries of
    // this thread are requested with request() and all are waited for and
    // handed to use(entry, value) by collect()
    constexpr int RP = RMAX >= 8 ? 2 : RMAX;
    auto row_of = [&](int e) -> int {
        if constexpr (RG) return rst[e].row;
        else return rgi[e];
    };
    auto store = [&](const double (&v)[RMAX]) {
        if constexpr (CL) {
#pragma unroll
            for (int k = 0; k < RMAX; ++k) cwo[k * NT + threadIdx.x] = v[k];
            return;
        }
        TagVal* o = D.xw + (size_t)(phase & 1) * D.N;
        const unsigned long long tg = comm.tag(phase);
#pragma unroll
        for (int k = 0; k < RMAX; ++k)
            if (own[k] & PUB) st_tag(o + row0 + k * NT, v[k], tg);
    };
    double xv[RP];
    unsigned long long xt[RP];
    auto request = [&](int ph) {
        if constexpr (CL) return;
        const TagVal* o = D.xw + (size_t)(ph & 1) * D.N;
#pragma unroll
        for (int u = 0; u < RP; ++u) {
            const int e = threadIdx.x + u * NT;
            xt[u] = 0;
            if (e < nr) ld_tag(o + row_of(e), xv[u], xt[u]);
        }
    };
    auto collect = [&](int ph, auto&& use) -> bool {
        if constexpr (CL) {
            for (int e = threadIdx.x; e < nr; e += NT) use(e, cwx[(ph & 1) * D.rem_max + e]);
            return true;
        }
        const TagVal* o = D.xw + (size_t)(ph & 1) * D.N;
        const unsigned long long want = comm.tag(ph);
        bool ok = true;
        SpinLimit lim;
        for (int e0 = threadIdx.x; e0 < nr && ok; e0 += RP * NT) {
            if (e0 != threadIdx.x) {
#pragma unroll
                for (int u = 0; u < RP; ++u) {
                    const int e = e0 + u * NT;
                    xt[u] = 0;
                    if (e < nr) ld_tag(o + row_of(e), xv[u], xt[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < RP; ++u) {
                const int e = e0 + u * NT;
                if (e < nr) {
                    if (xt[u] != want && !tag_wait(o + row_of(e), want, xv[u], xt[u], lim, comm.status)) ok = false;
                    use(e, xv[u]);
                }
            }
        }
        return ok;
    };

    // the all-reduce's two halves; MX (a tag) also takes the maximum
    auto publish = [&](const double (&v)[4], auto mx_tag, bool values = true) {
        constexpr bool MX = decltype(mx_tag)::value;
        if constexpr (CL) {
            const int par = phase & 1;
            const uint32_t bar = smem_addr(&cs.bar[par]);
            if (threadIdx.x == NT - 1) mbar_expect(bar, 32u * G + (values ? 8u * nr : 0u));
            cta_reduce4<NT, MX>(v, [&](int q, int j, double x) {
                const uint32_t at = smem_addr(&cs.part[par][b][q]);
                for (int c = j; c < G; c += 8) st_async_f64(cluster_addr(at, c), x, cluster_addr(bar, c));
            });
            // the own rows' values (visible since the reduction's barrier)
            if (values) {
                const uint32_t shift = 8u * par * D.rem_max;
                for (int k = threadIdx.x; k < npush; k += NT) {
                    const uint32_t e = cpl[k];
                    st_async_f64(cpu[k] + shift, cwo[e & 0xfffu], cluster_addr(bar, e >> 12));
                }
            }
        } else {
            tag_allreduce_publish<NT, false, MX>(comm, phase, v);
        }
    };
    auto wait = [&](double (&o)[4], bool ok, auto mx_tag, auto&& all_in) -> bool {
        constexpr bool MX = decltype(mx_tag)::value;
        if constexpr (CL) {
            const int par = phase & 1;
            const uint32_t bar = smem_addr(&cs.bar[par]);
            if (!mbar_wait(bar, (phase >> 1) & 1, comm.status)) ok = false;
            const int q = lane & 3;
            double a0 = cs.part[par][lane >> 2][q], a1 = cs.part[par][(lane >> 2) + 8][q];
#pragma unroll
            for (int d = 16; d >= 4; d >>= 1) {
                a0 = red4<MX>(q, a0, __shfl_xor_sync(0xffffffffu, a0, d));
                a1 = red4<MX>(q, a1, __shfl_xor_sync(0xffffffffu, a1, d));
            }
            a0 = red4<MX>(q, a0, a1);
#pragma unroll
            for (int p = 0; p < (MX ? 4 : 3); ++p) o[p] = __shfl_sync(0xffffffffu, a0, p);
            if (!MX) o[3] = 0.0;
            return __syncthreads_and(ok);
        } else {
            return tag_allreduce_wait<NT, false, MX>(comm, phase, o, ok, hold, all_in);
        }
    };
    using Max = std::true_type;
    using Sums = std::false_type;

    // ---- phase 0a: r0 = b - A x0 (constraints as the reference); partials:
    // invalid diagonals, non-finite residuals, (r,r), max|r|
    double off[RMAX], acc[4] = {0.0, 0.0, 0.0, 0.0}, t[4];
    for (int k = threadIdx.x; k < nh; k += NT) vh[k] = __ldcg(D.pres + D.halo_idx[h0 + k]);
    extra_first();
    __syncthreads();
    offdiag_all(off);
#pragma unroll
    for (int k = 0; k < RMAX; ++k) {
        if (k >= nk) continue;
        const int i = row0 + k * NT;
        const uint8_t f = D.nflag[i];
        const bool active = f & 1, fr = (f & 1) && !(f & 4);
        if (fr) own[k] |= FREE;
        const double pd = D.pdiag[i];
        const double xi = D.pres[i];
        if (pds) pds[k * NT + threadIdx.x] = pd;
        if (!XM) xr[XM ? 0 : k] = xi;
        else if (D.xs_off) xs[k * NT] = xi;
        if (PM) ps[k * NT] = 0.0;
        const double y = fma(pd, xi, off[k]);
        double ri = active ? D.rhs1[i] - y : 0.0;
        if (!fr) ri = 0.0;
        if (fr) {
            if (g.precond) {
                if (!(isfinite(pd) && pd > 1.0e-30)) acc[0] += 1.0;
                dd[k] = 1.0 / pd;
            } else {
                dd[k] = 1.0;
            }
            if (!isfinite(ri)) acc[1] += 1.0;
            acc[2] = fma(ri, ri, acc[2]);
            acc[3] = max_bits(acc[3], fabs(ri));
        }
        r[k] = ri;
    }
    // the pressure of the free own rows back to global memory
    auto store_x = [&]() {
        if (XM && !D.xs_off) return;
#pragma unroll
        for (int k = 0; k < RMAX; ++k)
            if (own[k] & FREE) D.pres[row0 + k * NT] = XM ? xs[k * NT] : xr[XM ? 0 : k];
    };
    store(r);
    publish(acc, Max());
    if (!wait(t, true, Max(), [&] { request(phase); })) return;
    const double init = sqrt(t[2]);
    if (init <= 1.0e-300) { cg_finish(D, g, 0, 1, init, init, 0.0, t[3]); return; }
    if (cg_converged(g.conv_test, 1.0, t[3], g.rel_tol, g.abs_tol)) { cg_finish(D, g, 0, 1, init, init, 1.0, t[3]); return; }
    if (t[1] > 0.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, 0, R_PCG_RESID); return; }
    if (t[0] > 0.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 1, ST_PCG, 0, R_PCG_DIAG); return; }
    const StopTest stop(g, init);

    // ---- phase 0b: z0 = M^-1 r0, w0 = A z0, gamma0 = (r0,z0), delta0 = (z0,w0)
    bool got = collect(phase, [&](int e, double v) {
        int place;
        double dj;
        remote(e, place, dj);
        rh[e] = v;
        vh[place] = v * dj;
    });
#pragma unroll
    for (int k = 0; k < RMAX; ++k)
        vh[own[k] & PLACE] = r[k] * dd[k];
    ++phase;
    extra_first();
    __syncthreads();
    offdiag_all(off);
    acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
#pragma unroll
    for (int k = 0; k < RMAX; ++k) {
        const double zi = r[k] * dd[k];
        w[k] = (own[k] & FREE) ? fma(diag(k), zi, off[k]) : 0.0;
        acc[0] = fma(r[k], zi, acc[0]);
        acc[1] = fma(zi, w[k], acc[1]);
    }
    store(w);
    publish(acc, Sums());
    if (!wait(t, got, Sums(), [&] { request(phase); })) return;
    double gam = t[0];
    if (gam <= 1.0e-300 || !isfinite(gam)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, 0, R_PCG_RZ0); return; }
    double den = t[1], alpha = gam / den, beta = 0.0, rr = init * init, mx = 0.0;
    int it = 0, conv = 0;
    int wph = phase;             // exchange that carries the w to collect
    // max|r| where the iterations carry none: an all-reduce of its own
    auto final_max = [&]() {
        double m[4] = {0.0, 0.0, 0.0, 0.0}, o[4];
#pragma unroll
        for (int k = 0; k < RMAX; ++k)
            if (own[k] & FREE) m[3] = max_bits(m[3], fabs(r[k]));
        ++phase;
        publish(m, Max(), false);
        const bool ok = wait(o, true, Max(), [] {});
        mx = o[3];
        return ok;
    };
    for (it = 1; it <= g.max_iter; ++it) {
        if (fabs(den) <= 1.0e-300 || !isfinite(den)) { store_x(); if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_PAP); return; }
        // z_it of the halo: s = w + beta*s, r -= alpha*s, z = r * dz, for the
        // remote entries from their owners' w and for the own rows
        got = collect(wph, [&](int e, double v) {
            int place;
            double dj;
            remote(e, place, dj);
            const double sj = fma(beta, sh[e], v);
            const double rj = fma(-alpha, sj, rh[e]);
            sh[e] = sj;
            rh[e] = rj;
            vh[place] = rj * dj;
        });
        // own rows: p = z_o + beta*p, s = w + beta*s, r -= alpha*s
#pragma unroll
        for (int k = 0; k < RMAX; ++k) {
            p[k] = fma(beta, p[k], r[k] * dd[k]);
            if (PM && (own[k] & FREE)) ps[k * NT] = p[k];
            s[k] = fma(beta, s[k], w[k]);
            r[k] = fma(-alpha, s[k], r[k]);
            vh[own[k] & PLACE] = r[k] * dd[k];
        }
        ++phase;
        extra_first();
        __syncthreads();
        offdiag_all(off);
        acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
#pragma unroll
        for (int k = 0; k < RMAX; ++k) {
            const double zi = r[k] * dd[k];
            w[k] = (own[k] & FREE) ? fma(diag(k), zi, off[k]) : 0.0;
            acc[0] = fma(r[k], zi, acc[0]);
            acc[1] = fma(zi, w[k], acc[1]);
            acc[2] = fma(r[k], r[k], acc[2]);
            if (stop.needs_max()) acc[3] = max_bits(acc[3], fabs(r[k]));
        }
        store(w);
        wph = phase;
        // x after the CTA's partials are on their way
        auto update_x = [&]() {
#pragma unroll
            for (int k = 0; k < RMAX; ++k) {
                if (!XM) xr[XM ? 0 : k] = fma(alpha, p[k], xr[XM ? 0 : k]);
                else if (own[k] & FREE) {
                    if (PM) p[k] = ps[k * NT];
                    xs[k * NT] = fma(alpha, p[k], xs[k * NT]);
                }
            }
        };
        if (!stop.needs_max()) {
            publish(acc, Sums());
            update_x();
            got = wait(t, got, Sums(), [&] { request(phase); });
        } else {
            publish(acc, Max());
            update_x();
            got = wait(t, got, Max(), [&] { request(phase); });
        }
        if (!got) { store_x(); return; }
        rr = t[2];
        mx = t[3];
        const double gn = t[0];
        // (p, Ap) of the next direction: delta - beta*gn/alpha, where
        // gn/alpha = beta*den; the rare exits beside the two divisions
        beta = gn / gam;
        den = fma(-beta * beta, den, t[1]);
        alpha = gn / den;
        gam = gn;
        if (!stop.clear(rr) || gn <= 1.0e-300 || !isfinite(gn)) {
            if (!stop.needs_max() && !final_max()) { store_x(); return; }
            if (stop.exact(rr, mx)) { conv = 1; break; }
            // a non-finite residual shows as a non-finite max |r|
            if (!isfinite(mx)) { store_x(); if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, it, R_PCG_RESID); return; }
            if (gn <= 1.0e-300 || !isfinite(gn)) { store_x(); if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_RZ); return; }
            // rounding put (r,r) inside the margin: on, after one more
            // all-reduce that keeps the records' two buffers apart (the next
            // w may not overwrite the last one before every CTA has read it)
            if (!stop.needs_max() && !final_max()) { store_x(); return; }
        }
    }
    if (!conv && !stop.needs_max() && !final_max()) { store_x(); return; }
    store_x();
    if (it > g.max_iter) it = g.max_iter;
    cg_finish(D, g, it, conv, init, sqrt(rr), sqrt(rr) / init, mx);
    if (!conv && b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 2, ST_PCG, it, R_PCG_MAXIT);
}

// The single-reduction (Chronopoulos-Gear) Jacobi-PCG with its rows in
// registers.  KT > 0 (one 512-thread CTA per SM): warp 0 takes the SM's
// tensor memory before the solve and returns it after; every exit of the
// body (converged, an error status, a timed-out wait) is CTA-uniform and
// comes back here, so the memory is freed on every path.
template <int RMAX, bool BATCH, int NT, int KS = 0, int KT = 0, bool CL = false, bool RG = false>
__global__ void __launch_bounds__(NT, NT >= 512 ? 1 : 2) k_pcg64c(PcgDev D)
{
    unsigned long long epoch;
    if (!tag_begin<BATCH>(D, epoch)) return;
    if constexpr (KT == 0) {
        pcg64c_body<RMAX, BATCH, NT, KS, 0, CL, RG>(D, 0u, epoch);
    } else {
        static_assert(NT == 512, "TMEM rows: one CTA per SM");
        __shared__ uint32_t s_tm;
        const bool w0 = (threadIdx.x >> 5) == 0;
        if (w0) tmem_alloc_all(&s_tm);
        tmem_fence_before_sync();
        __syncthreads();
        tmem_fence_after_sync();
        const uint32_t tm = s_tm;
        pcg64c_body<RMAX, BATCH, NT, KS, KT, CL, RG>(D, tm, epoch);
        tmem_fence_before_sync();
        __syncthreads();
        tmem_fence_after_sync();
        if (w0) tmem_free_all(tm);
    }
    // no CTA leaves while another may still write into its shared memory
    // (every wait before this one is bounded, so all of them get here)
    if constexpr (CL) cluster_sync();
    tag_end<BATCH>(D, epoch);
}

template <int RMAX>
__global__ void __launch_bounds__(512, 1) k_pcg64d(PcgDev D, CoarseDev C)
{
    constexpr bool BATCH = false;
    constexpr int NT = 512;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const SegView g = seg_view<BATCH>(D);
    const int G = g.G, b = g.b;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s_beg = g.s0 + (int)((long long)b * (g.s1 - g.s0) / G);
    const int s_end = g.s0 + (int)((long long)(b + 1) * (g.s1 - g.s0) / G);
    const long long S0 = D.slice_off[s_beg];
    const int nsl = (int)(D.slice_off[s_end] - S0);
    const int h0 = D.halo_ptr[blockIdx.x];
    const int nh = D.halo_ptr[blockIdx.x + 1] - h0;
    const TwoLevelLayout L(D.halo_max, D.slot_max, C.nbr_max, C.G);
    double* vh = reinterpret_cast<double*>(smem_raw);
    double* dzh = vh + D.halo_max;
    int* hidx = reinterpret_cast<int*>(smem_raw + L.hidx);
    unsigned short* lcs = reinterpret_cast<unsigned short*>(smem_raw + L.lcs);
    for (int k = threadIdx.x; k < nh; k += NT) hidx[k] = D.halo_idx[h0 + k];
    for (int k = threadIdx.x; k < nsl; k += NT) lcs[k] = D.lcol[S0 + k];
    // coarse space: this CTA's rows of the coarse inverse (its own and its
    // halo's owners), the coarse vectors P^T r, P^T s, P^T w, the coarse
    // correction of each neighbour and the owner of every halo entry
    const int GC = C.G;
    const int nb0 = C.nbr_ptr[blockIdx.x];
    const int nn = C.nbr_ptr[blockIdx.x + 1] - nb0;
    double* ainv = reinterpret_cast<double*>(smem_raw + L.ainv);
    double* cr = ainv + (size_t)C.nbr_max * GC;
    double* cs = cr + GC;
    double* cw = cs + GC;
    double* ec = cw + GC;
    unsigned char* hown = smem_raw + L.hown;
    __shared__ int s_own;
    __shared__ double s_ecp;   // this CTA's coarse correction of the previous iteration's z
    if (threadIdx.x == 0)
        for (int j = 0; j < nn; ++j)
            if (C.nbr_ids[nb0 + j] == (int)blockIdx.x) s_own = j;
    for (int t = threadIdx.x; t < nn * GC; t += NT)
        ainv[t] = C.ainv[(size_t)C.nbr_ids[nb0 + t / GC] * GC + t % GC];
    for (int k = threadIdx.x; k < nh; k += NT) hown[k] = C.hown[h0 + k];
    for (int t = threadIdx.x; t < GC; t += NT) cs[t] = 0.0;
    // ec[j] = (A_c^-1 P^T r)[neighbour j]: one warp per neighbour, fixed order
    auto coarse_correction = [&]() {
        __syncthreads();
        for (int j = warp; j < nn; j += NT / 32) {
            double acc = 0.0;
            for (int t = lane; t < GC; t += 32) acc = fma(ainv[(size_t)j * GC + t], cr[t], acc);
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
            if (lane == 0) ec[j] = acc;
        }
        __syncthreads();
    };
    int phase = 0;
    const int N = D.N;
    // parity buffers: r in r/pA, w in q/pB, s in z/dz(+N)... laid out by the engine
    double* rb[2] = {D.r, D.r + N};
    double* wb[2] = {D.q, D.q + N};
    double* sb[2] = {D.pA, D.pB};
    double* dz = D.z;   // free ? 1/diagonal : 0  (z = r * dz)

    // rows of this thread: slice s_beg + warp + NW*k, lane; their slot base
    // and width are re-read where needed (registers go to the coarse state)
    double r[RMAX], p[RMAX], s[RMAX], w[RMAX], dd[RMAX];
    bool fr[RMAX];
    int wmax = 0;
    auto slice_of = [&](int k) { return s_beg + warp + (NT / 32) * k; };
    auto row_of = [&](int k) { const int sl = slice_of(k); return sl < s_end ? sl * 32 + lane : -1; };
    auto width_of = [&](int k) { const int sl = slice_of(k); return sl < s_end ? D.slice_w[sl] : 0; };
    auto base_of = [&](int k) { const int sl = slice_of(k); return sl < s_end ? (int)(D.slice_off[sl] - S0) + lane : 0; };
#pragma unroll
    for (int k = 0; k < RMAX; ++k) {
        const int wk = width_of(k);
        wmax = wk > wmax ? wk : wmax;
        r[k] = p[k] = s[k] = w[k] = 0.0;
        dd[k] = 0.0;   // reciprocal of the Jacobi diagonal; 0 off the free rows
        fr[k] = false;
    }
    constexpr int CH = (RMAX >= 8) ? 2 : (RMAX >= 4) ? 4 : 8;
    auto offdiag_all = [&](double* off) {
        int lbase[RMAX], wr[RMAX];
#pragma unroll
        for (int k = 0; k < RMAX; ++k) { off[k] = 0.0; lbase[k] = base_of(k); wr[k] = width_of(k); }
        for (int k0 = 0; k0 < wmax; k0 += CH) {
            double v[RMAX][CH];
#pragma unroll
            for (int k = 0; k < RMAX; ++k)
#pragma unroll
                for (int u = 0; u < CH; ++u)
                    v[k][u] = (k0 + u < wr[k]) ? __ldcg(D.val + S0 + lbase[k] + 32 * (k0 + u)) : 0.0;
#pragma unroll
            for (int k = 0; k < RMAX; ++k)
#pragma unroll
                for (int u = 0; u < CH; ++u) {
                    const double g = (k0 + u < wr[k]) ? vh[lcs[lbase[k] + 32 * (k0 + u)]] : 0.0;
                    off[k] = fma(v[k][u], g, off[k]);
                }
        }
    };

    // ---- phase 0a: r0 = b - A x0 (constraints as the reference), dz
    double off[RMAX];
    __syncthreads();
    for (int k0 = threadIdx.x; k0 < nh; k0 += 4 * NT) {
        double a[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + u * NT;
            a[u] = __ldcg(D.pres + (k < nh ? hidx[k] : 0));
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k0 + u * NT < nh) vh[k0 + u * NT] = a[u];
    }
    __syncthreads();
    offdiag_all(off);
    Acc6 acc{0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < RMAX; ++k) {
        const int i = row_of(k);
        if (i < 0) continue;
        const uint8_t f = D.nflag[i];
        const bool active = f & 1;
        fr[k] = (f & 1) && !(f & 4);
        const double pd = D.pdiag[i];
        const double y = fma(pd, D.pres[i], off[k]);
        double ri = active ? D.rhs1[i] - y : 0.0;
        if (!fr[k]) ri = 0.0;
        if (fr[k]) {
            if (g.precond) {
                if (!(isfinite(pd) && pd > 1.0e-30)) acc.flag = fmax(acc.flag, 1.0);
                dd[k] = 1.0 / pd;
            } else {
                dd[k] = 1.0;
            }
            if (!isfinite(ri)) acc.flag = fmax(acc.flag, 2.0);
            acc.c = fma(ri, ri, acc.c);
            acc.mx = fmax(acc.mx, fabs(ri));
        }
        r[k] = ri;
        rb[0][i] = ri;
        dz[i] = dd[k];
        sb[0][i] = 0.0;
    }
    double xs = 0.0;
#pragma unroll
    for (int k = 0; k < RMAX; ++k) xs += r[k];
    Acc6 t{0.0, 0.0, 0.0, 0.0, 0.0};
    if (!grid_allreduce3g<NT>(acc, xs, D, g, phase, t, cr)) return;
    ++phase;
    const double init = sqrt(t.c);
    if (init <= 1.0e-300) { cg_finish(D, g, 0, 1, init, init, 0.0, t.mx); return; }
    if (cg_converged(g.conv_test, 1.0, t.mx, g.rel_tol, g.abs_tol)) { cg_finish(D, g, 0, 1, init, init, 1.0, t.mx); return; }
    if (t.flag >= 2.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, 0, R_PCG_RESID); return; }
    if (t.flag >= 1.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 1, ST_PCG, 0, R_PCG_DIAG); return; }

    // ---- phase 0b: z0 = M^-1 r0, w0 = A z0, gamma0 = (r0,z0), delta0 = (z0,w0)
    coarse_correction();
    for (int k0 = threadIdx.x; k0 < nh; k0 += 4 * NT) {
        double a[4], c[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + u * NT;
            const int j = k < nh ? hidx[k] : 0;
            a[u] = __ldcg(dz + j);
            c[u] = __ldcg(rb[0] + j);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + u * NT;
            if (k < nh) { dzh[k] = a[u]; vh[k] = a[u] != 0.0 ? fma(c[u], a[u], ec[hown[k]]) : 0.0; }
        }
    }
    __syncthreads();
    offdiag_all(off);
    acc = Acc6{0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < RMAX; ++k) {
        const int i = row_of(k);
        if (i < 0) continue;
        const double zi = fr[k] ? fma(r[k], dd[k], ec[s_own]) : 0.0;
        w[k] = fr[k] ? fma(D.pdiag[i], zi, off[k]) : 0.0;
        wb[0][i] = w[k];
        if (fr[k]) {
            acc.a = fma(r[k], zi, acc.a);
            acc.b = fma(zi, w[k], acc.b);
        }
    }
    xs = 0.0;
#pragma unroll
    for (int k = 0; k < RMAX; ++k) xs += w[k];
    t = Acc6{0.0, 0.0, 0.0, 0.0, 0.0};
    if (!grid_allreduce3g<NT>(acc, xs, D, g, phase, t, cw)) return;
    ++phase;
    if (threadIdx.x == 0) s_ecp = ec[s_own];
    double gam = t.a;
    if (gam <= 1.0e-300 || !isfinite(gam)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, 0, R_PCG_RZ0); return; }
    double den = t.b;
    double beta = 0.0, fin = init, rel = 1.0, mx = 0.0, alpha = 0.0;
    int it = 0, conv = 0;
    for (it = 1; it <= g.max_iter; ++it) {
        if (fabs(den) <= 1.0e-300 || !isfinite(den)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_PAP); return; }
        alpha = gam / den;
        const int po = (it - 1) & 1, pn = it & 1;
        // P^T s = P^T w_o + beta P^T s_o, P^T r = P^T r_o - alpha P^T s (the
        // recurrences of s and r, aggregated), then the new coarse correction
        for (int c = threadIdx.x; c < GC; c += NT) {
            cs[c] = fma(beta, cs[c], cw[c]);
            cr[c] = fma(-alpha, cs[c], cr[c]);
        }
        coarse_correction();
        // stage z_it of the halo: s = w_o + beta*s_o, r = r_o - alpha*s, z = r / dz
        // (SU halo nodes per thread per round, all their loads issued first)
        __syncthreads();
        {
            constexpr int SU = 8;   // halo nodes per thread per round (measured: 8 beats 4 and 2)
            const double* so = sb[po];
            const double* wo = wb[po];
            const double* ro = rb[po];
            for (int k0 = threadIdx.x; k0 < nh; k0 += SU * NT) {
                double a[SU], c[SU], e[SU];
#pragma unroll
                for (int u = 0; u < SU; ++u) {
                    const int k = k0 + u * NT;
                    const int j = k < nh ? hidx[k] : 0;
                    a[u] = __ldcg(so + j);
                    c[u] = __ldcg(wo + j);
                    e[u] = __ldcg(ro + j);
                }
#pragma unroll
                for (int u = 0; u < SU; ++u) {
                    const int k = k0 + u * NT;
                    if (k < nh) {
                        const double sj = fma(beta, a[u], c[u]);
                        const double rj = fma(-alpha, sj, e[u]);
                        vh[k] = dzh[k] != 0.0 ? fma(rj, dzh[k], ec[hown[k]]) : 0.0;
                    }
                }
            }
        }
        __syncthreads();
        // own rows: p = z_o + beta*p, s = w + beta*s, x += alpha*p, r -= alpha*s
#pragma unroll
        for (int k = 0; k < RMAX; ++k) {
            const int i = row_of(k);
            if (i < 0) continue;
            const double zo = fma(r[k], dd[k], s_ecp);
            p[k] = fr[k] ? fma(beta, p[k], zo) : 0.0;
            s[k] = fma(beta, s[k], w[k]);
            if (fr[k]) D.pres[i] = fma(alpha, p[k], D.pres[i]);
            r[k] = fma(-alpha, s[k], r[k]);
            rb[pn][i] = r[k];
            sb[pn][i] = s[k];
        }
        offdiag_all(off);
        Acc6 a6{0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < RMAX; ++k) {
            const int i = row_of(k);
            if (i < 0) continue;
            const double zi = fr[k] ? fma(r[k], dd[k], ec[s_own]) : 0.0;
            w[k] = fr[k] ? fma(D.pdiag[i], zi, off[k]) : 0.0;
            wb[pn][i] = w[k];
            if (fr[k]) {
                if (!isfinite(r[k])) a6.flag = 1.0;
                a6.a = fma(r[k], zi, a6.a);
                a6.b = fma(zi, w[k], a6.b);
                a6.c = fma(r[k], r[k], a6.c);
                a6.mx = fmax(a6.mx, fabs(r[k]));
            }
        }
        xs = 0.0;
#pragma unroll
        for (int k = 0; k < RMAX; ++k) xs += w[k];
        t = Acc6{0.0, 0.0, 0.0, 0.0, 0.0};
        if (!grid_allreduce3g<NT>(a6, xs, D, g, phase, t, cw)) return;
        ++phase;
        if (threadIdx.x == 0) s_ecp = ec[s_own];
        fin = sqrt(t.c);
        mx = t.mx;
        rel = fin / init;
        if (cg_converged(g.conv_test, rel, mx, g.rel_tol, g.abs_tol)) { conv = 1; break; }
        if (t.flag > 0.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, it, R_PCG_RESID); return; }
        const double gn = t.a;
        if (gn <= 1.0e-300 || !isfinite(gn)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_RZ); return; }
        beta = gn / gam;
        den = t.b - beta * gn / alpha;
        gam = gn;
    }
    if (it > g.max_iter) it = g.max_iter;
    cg_finish(D, g, it, conv, init, fin, rel, mx);
    if (!conv && b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 2, ST_PCG, it, R_PCG_MAXIT);
}

// ------------------------------------------- mixed-precision PCG (FP32)
// The Chronopoulos-Gear iteration of k_pcg64c in FP32 -- r, z, w, s, p and
// the assembled coefficients are single precision, the coefficients and local
// column indices resident in shared memory for the whole solve -- with the
// reductions, alpha/beta and the pressure in FP64, and FP64 defect
// correction by residual replacement: whenever the recursive residual has
// fallen by the inner tolerance since the last correction, and whenever it meets the
// stopping test, the true residual r = b - A x is recomputed from the FP64
// coefficients and FP64 pressure, and w = A z, s = A p are recomputed, so the
// FP32 recurrences restart from exact data without discarding the search
// direction; the curvature of the next direction is then computed from
// fresh products rather than recurred, and a correction that finds no
// progress since the previous one also drops the direction.  The solve
// stops only when the FP64 true residual meets the reference's stopping
// test.
constexpr int RU_STALL = 256;   // iterations without a correction before one is forced

template <int RMAX, bool BATCH, int NT>
__device__ __forceinline__ void pcg32m_body(const PcgDev& D, unsigned long long epoch)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const SegView g = seg_view<BATCH>(D);
    const int G = g.G, b = g.b;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s_beg = g.s0 + (int)((long long)b * (g.s1 - g.s0) / G);
    const int s_end = g.s0 + (int)((long long)(b + 1) * (g.s1 - g.s0) / G);
    const long long S0 = D.slice_off[s_beg];
    const int nsl = (int)(D.slice_off[s_end] - S0);
    const int h0 = D.halo_ptr[blockIdx.x];
    const int nh = D.halo_ptr[blockIdx.x + 1] - h0;
    const int HM = D.halo_max;
    double* vh64 = reinterpret_cast<double*>(smem_raw);                 // HM doubles, or:
    float* vz = reinterpret_cast<float*>(smem_raw);                     //   HM floats (z)
    float* vp = vz + HM;                                                //   HM floats (p)
    float* dzh = reinterpret_cast<float*>(vh64 + HM);                   // HM
    int* hidx = reinterpret_cast<int*>(dzh + HM);                       // HM
    float* val32s = reinterpret_cast<float*>(hidx + HM);                // nsl
    unsigned short* lcs = reinterpret_cast<unsigned short*>(val32s + D.slot_max);
    for (int k = threadIdx.x; k < nh; k += NT) hidx[k] = D.halo_idx[h0 + k];
    for (int k = threadIdx.x; k < nsl; k += NT) {
        lcs[k] = D.lcol[S0 + k];
        val32s[k] = D.val32[S0 + k];
    }
    const TagComm comm = tag_comm(D, g, epoch);
    PollHold hold;
    int phase = 0;
    // three sums and a maximum; the vectors go by plain stores, made visible
    // with the record
    auto allreduce = [&](const double (&v)[4], double (&o)[4]) {
        tag_allreduce_publish<NT, true, true>(comm, phase, v);
        const bool ok = tag_allreduce_wait<NT, true, true>(comm, phase, o, true, hold, [] {});
        ++phase;
        return ok;
    };
    const int N = D.N;
    float* rb[2] = {D.r32, D.r32 + N};
    float* wb[2] = {D.w32, D.w32 + N};
    float* sb[2] = {D.s32, D.s32 + N};
    float* pb = D.p32;
    float* dz = D.dz32;

    float r[RMAX], p[RMAX], sv[RMAX], w[RMAX], dd[RMAX];
    bool fr[RMAX];
    int row[RMAX], lbase[RMAX], wr[RMAX];
    int wmax = 0;
#pragma unroll
    for (int k = 0; k < RMAX; ++k) {
        const int sl = s_beg + warp + (NT / 32) * k;
        row[k] = (sl < s_end) ? sl * 32 + lane : -1;
        lbase[k] = 0;
        wr[k] = 0;
        if (sl < s_end) {
            lbase[k] = (int)(D.slice_off[sl] - S0) + lane;
            wr[k] = D.slice_w[sl];
            wmax = wr[k] > wmax ? wr[k] : wmax;
        }
        r[k] = p[k] = sv[k] = w[k] = 0.0f;
        dd[k] = 0.0f;   // reciprocal of the Jacobi diagonal; 0 off the free rows
        fr[k] = false;
    }
    // FP64 off-diagonal sums from the streamed FP64 coefficients and vh64
    auto offdiag64 = [&](double* off) {
#pragma unroll
        for (int k = 0; k < RMAX; ++k) off[k] = 0.0;
        for (int k0 = 0; k0 < wmax; k0 += 4) {
            double v[RMAX][4];
#pragma unroll
            for (int k = 0; k < RMAX; ++k)
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    v[k][u] = (k0 + u < wr[k]) ? __ldcg(D.val + S0 + lbase[k] + 32 * (k0 + u)) : 0.0;
#pragma unroll
            for (int k = 0; k < RMAX; ++k)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const double g = (k0 + u < wr[k]) ? vh64[lcs[lbase[k] + 32 * (k0 + u)]] : 0.0;
                    off[k] = fma(v[k][u], g, off[k]);
                }
        }
    };
    // FP32 off-diagonal sums from the resident coefficients and a float halo
    auto offdiag32 = [&](const float* vx, float* off) {
#pragma unroll
        for (int k = 0; k < RMAX; ++k) off[k] = 0.0f;
        for (int kk = 0; kk < wmax; ++kk) {
#pragma unroll
            for (int k = 0; k < RMAX; ++k)
                if (kk < wr[k]) {
                    const int sl = lbase[k] + 32 * kk;
                    off[k] = fmaf(val32s[sl], vx[lcs[sl]], off[k]);
                }
        }
    };
    auto stage64 = [&](const double* x) {
        __syncthreads();
        for (int k0 = threadIdx.x; k0 < nh; k0 += 4 * NT) {
            double a[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = k0 + u * NT;
                a[u] = __ldcg(x + (k < nh ? hidx[k] : 0));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (k0 + u * NT < nh) vh64[k0 + u * NT] = a[u];
        }
        __syncthreads();
    };
    // true residual of the own rows into r[], rb[buf]; partials: non-finite
    // entries, (r,r), max|r|
    auto true_residual = [&](int buf, double (&acc)[4]) {
        stage64(D.pres);
        double off[RMAX];
        offdiag64(off);
#pragma unroll
        for (int k = 0; k < RMAX; ++k) {
            const int i = row[k];
            if (i < 0) continue;
            const double y = fma(D.pdiag[i], D.pres[i], off[k]);
            double ri = (D.nflag[i] & 1) ? D.rhs1[i] - y : 0.0;
            if (!fr[k]) ri = 0.0;
            if (fr[k]) {
                if (!isfinite(ri)) acc[1] += 1.0;
                acc[2] = fma(ri, ri, acc[2]);
                acc[3] = max_bits(acc[3], fabs(ri));
            }
            r[k] = (float)ri;
            rb[buf][i] = r[k];
            pb[i] = p[k];
        }
    };
    // w = A z and s = A p from the staged halos (p taken as zero when
    // zero_p, which restarts the direction); partials of r.z, z.w, z.s, p.w
    // and p.s, from which the step length of the next direction
    // (z + beta p).A(z + beta p) follows directly
    auto refresh_ws = [&](int buf, bool zero_p, double (&acc)[5]) {
        __syncthreads();
        for (int k0 = threadIdx.x; k0 < nh; k0 += 4 * NT) {
            float a[4], c[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = k0 + u * NT;
                const int j = k < nh ? hidx[k] : 0;
                a[u] = __ldcg(rb[buf] + j);
                c[u] = zero_p ? 0.0f : __ldcg(pb + j);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = k0 + u * NT;
                if (k < nh) { vz[k] = a[u] * dzh[k]; vp[k] = c[u]; }
            }
        }
        __syncthreads();
        float offz[RMAX], offp[RMAX];
        offdiag32(vz, offz);
        offdiag32(vp, offp);
#pragma unroll
        for (int k = 0; k < RMAX; ++k) {
            const int i = row[k];
            if (i < 0) continue;
            if (zero_p) p[k] = 0.0f;
            const float pd = (float)D.pdiag[i];
            const float zi = r[k] * dd[k];
            w[k] = fr[k] ? fmaf(pd, zi, offz[k]) : 0.0f;
            sv[k] = fr[k] ? fmaf(pd, p[k], offp[k]) : 0.0f;
            wb[buf][i] = w[k];
            sb[buf][i] = sv[k];
            if (fr[k]) {
                const double zd = zi, pv = p[k];
                acc[0] = fma((double)r[k], zd, acc[0]);
                acc[1] = fma(zd, (double)w[k], acc[1]);
                acc[2] = fma(zd, (double)sv[k], acc[2]);
                acc[3] = fma(pv, (double)w[k], acc[3]);
                acc[4] = fma(pv, (double)sv[k], acc[4]);
            }
        }
    };

    // ---- phase 0a: FP64 r0 = b - A x0, its norm, dz
    double acc[4] = {0.0, 0.0, 0.0, 0.0}, t[4];   // [0]: invalid diagonals
#pragma unroll
    for (int k = 0; k < RMAX; ++k) {
        const int i = row[k];
        if (i < 0) continue;
        const uint8_t f = D.nflag[i];
        fr[k] = (f & 1) && !(f & 4);
        const double pd = D.pdiag[i];
        if (fr[k]) {
            if (g.precond && !(isfinite(pd) && pd > 1.0e-30)) acc[0] += 1.0;
            dd[k] = g.precond ? (float)(1.0 / pd) : 1.0f;
        }
        dz[i] = dd[k];
        sb[0][i] = 0.0f;
    }
    true_residual(0, acc);
    if (!allreduce(acc, t)) return;
    const double init = sqrt(t[2]);
    if (init <= 1.0e-300) { cg_finish(D, g, 0, 1, init, init, 0.0, t[3]); return; }
    if (cg_converged(g.conv_test, 1.0, t[3], g.rel_tol, g.abs_tol)) { cg_finish(D, g, 0, 1, init, init, 1.0, t[3]); return; }
    if (t[1] > 0.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, 0, R_PCG_RESID); return; }
    if (t[0] > 0.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 1, ST_PCG, 0, R_PCG_DIAG); return; }
    double rr_last = t[2];

    // ---- phase 0b: z0, w0 = A z0 (p = 0, s = 0)
    __syncthreads();
    for (int k = threadIdx.x; k < nh; k += NT) dzh[k] = __ldcg(dz + hidx[k]);
    // the five sums of a refresh, in two all-reduces
    auto allreduce5 = [&](const double (&v)[5], double (&o)[5]) {
        const double v0[4] = {v[0], v[1], v[2], 0.0}, v1[4] = {v[3], v[4], 0.0, 0.0};
        double o0[4], o1[4];
        if (!allreduce(v0, o0) || !allreduce(v1, o1)) return false;
        o[0] = o0[0]; o[1] = o0[1]; o[2] = o0[2]; o[3] = o1[0]; o[4] = o1[1];
        return true;
    };
    double a8[5] = {0.0, 0.0, 0.0, 0.0, 0.0}, t8[5];
    refresh_ws(0, true, a8);
    if (!allreduce5(a8, t8)) return;
    double gam = t8[0];
    if (gam <= 1.0e-300 || !isfinite(gam)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, 0, R_PCG_RZ0); return; }
    double den = t8[1];
    double beta = 0.0, fin = init, rel = 1.0, mx = 0.0, alpha = 0.0;
    int it = 0, conv = 0, outer = 0, last_fix = 0;
    for (it = 1; it <= g.max_iter; ++it) {
        if (fabs(den) <= 1.0e-300 || !isfinite(den)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_PAP); return; }
        alpha = gam / den;
        const float a32 = (float)alpha, b32 = (float)beta;
        const int po = (it - 1) & 1, pn = it & 1;
        __syncthreads();
        {
            const float* so = sb[po];
            const float* wo = wb[po];
            const float* ro = rb[po];
            for (int k0 = threadIdx.x; k0 < nh; k0 += 4 * NT) {
                float a[4], c[4], e[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int k = k0 + u * NT;
                    const int j = k < nh ? hidx[k] : 0;
                    a[u] = __ldcg(so + j);
                    c[u] = __ldcg(wo + j);
                    e[u] = __ldcg(ro + j);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int k = k0 + u * NT;
                    if (k < nh) {
                        const float sj = fmaf(b32, a[u], c[u]);
                        const float rj = fmaf(-a32, sj, e[u]);
                        vz[k] = rj * dzh[k];
                    }
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < RMAX; ++k) {
            const int i = row[k];
            if (i < 0) continue;
            const float zo = r[k] * dd[k];
            p[k] = fr[k] ? fmaf(b32, p[k], zo) : 0.0f;
            sv[k] = fmaf(b32, sv[k], w[k]);
            if (fr[k]) D.pres[i] = fma(alpha, (double)p[k], D.pres[i]);
            r[k] = fmaf(-a32, sv[k], r[k]);
            rb[pn][i] = r[k];
            sb[pn][i] = sv[k];
        }
        float off[RMAX];
        offdiag32(vz, off);
        double a6[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < RMAX; ++k) {
            const int i = row[k];
            if (i < 0) continue;
            const float zi = r[k] * dd[k];
            w[k] = fr[k] ? fmaf((float)D.pdiag[i], zi, off[k]) : 0.0f;
            wb[pn][i] = w[k];
            if (fr[k]) {
                a6[0] = fma((double)r[k], (double)zi, a6[0]);
                a6[1] = fma((double)zi, (double)w[k], a6[1]);
                a6[2] = fma((double)r[k], (double)r[k], a6[2]);
                a6[3] = max_bits(a6[3], fabs((double)r[k]));
            }
        }
        if (!allreduce(a6, t)) return;
        if (!isfinite(t[3])) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, it, R_PCG_RESID); return; }
        fin = sqrt(t[2]);
        mx = t[3];
        rel = fin / init;
        const bool candidate = cg_converged(g.conv_test, rel, mx, g.rel_tol, g.abs_tol);
        if (candidate || t[2] <= D.inner_tol * D.inner_tol * rr_last || it - last_fix >= RU_STALL) {
            // residual replacement from the FP64 coefficients and pressure
            double u1[4] = {0.0, 0.0, 0.0, 0.0};
            true_residual(pn, u1);
            if (!allreduce(u1, t)) return;
            ++outer;
            last_fix = it;
            if (t[1] > 0.0) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 4, ST_PCG, it, R_PCG_RESID); return; }
            fin = sqrt(t[2]);
            mx = t[3];
            rel = fin / init;
            // no progress of the true residual since the last correction:
            // the FP32 recurrences have lost the Krylov relations, restart
            const bool restart = t[2] >= rr_last;
            rr_last = t[2];
            if (cg_converged(g.conv_test, rel, mx, g.rel_tol, g.abs_tol)) { conv = 1; break; }
            double u2[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
            refresh_ws(pn, restart, u2);
            if (!allreduce5(u2, t8)) return;
            const double gn = t8[0];
            if (gn <= 1.0e-300 || !isfinite(gn)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_RZ); return; }
            // next direction z + beta p with its curvature computed, not recurred
            beta = restart ? 0.0 : gn / gam;
            den = t8[1] + beta * (t8[2] + t8[3]) + beta * beta * t8[4];
            gam = gn;
            continue;
        }
        const double gn = t[0];
        if (gn <= 1.0e-300 || !isfinite(gn)) { if (b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 3, ST_PCG, it, R_PCG_RZ); return; }
        beta = gn / gam;
        den = t[1] - beta * gn / alpha;
        gam = gn;
    }
    if (it > g.max_iter) it = g.max_iter;
    cg_finish(D, g, it, conv, init, fin, rel, mx);
    if (b == 0 && threadIdx.x == 0) seg_out(D, g)->outer = outer;
    if (!conv && b == 0 && threadIdx.x == 0) set_status(seg_status(D, g), 2, ST_PCG, it, R_PCG_MAXIT);
}

template <int RMAX, bool BATCH, int NT>
__global__ void __launch_bounds__(NT, NT >= 512 ? 1 : 2) k_pcg32m(PcgDev D)
{
    unsigned long long epoch;
    if (!tag_begin<BATCH>(D, epoch)) return;
    pcg32m_body<RMAX, BATCH, NT>(D, epoch);
    tag_end<BATCH>(D, epoch);
}

// ------------------------------------------------- two-level set-up kernels
// Aggregated operator P^T A P of the free rows: one CTA per nonzero (I, J)
// block; thread t sums entries t, t+T, ... (coefficient slots, or the
// diagonal of row -e-1), then warps and the CTA reduce in a fixed order.
// The diagonal is read by row position, or through row_node when that is
// given (the node-ordered diagonal: the same values on free rows).
__global__ void __launch_bounds__(256) k_coarse_blocks(const int* pair_ptr, const int2* pair_ij, const int* ent,
                                                       const double* val, const double* pdiag, const int* row_node,
                                                       int G, double* ac)
{
    __shared__ double sm[8];
    const int q = blockIdx.x;
    double s = 0.0;
    for (int k = pair_ptr[q] + threadIdx.x; k < pair_ptr[q + 1]; k += 256) {
        const int e = ent[k];
        s += e >= 0 ? val[e] : pdiag[row_node ? row_node[-e - 1] : -e - 1];
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += sm[w];
        ac[(size_t)pair_ij[q].x * G + pair_ij[q].y] = t;
    }
}

// In-place Gauss-Jordan inverse of the SPD coarse operator in shared memory
// (one CTA; warps take rows, lanes columns).  An aggregate without free rows
// has an empty row and column; it gets a unit diagonal and stays decoupled.
__global__ void __launch_bounds__(512) k_coarse_invert(int G, double* ac)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* a = reinterpret_cast<double*>(smem_raw);
    double* rowk = a + (size_t)G * G;
    double* colk = rowk + G;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int t = threadIdx.x; t < G * G; t += blockDim.x) a[t] = ac[t];
    __syncthreads();
    for (int t = threadIdx.x; t < G; t += blockDim.x)
        if (a[(size_t)t * G + t] == 0.0) a[(size_t)t * G + t] = 1.0;
    for (int k = 0; k < G; ++k) {
        __syncthreads();
        const double pinv = 1.0 / a[(size_t)k * G + k];
        for (int t = threadIdx.x; t < G; t += blockDim.x) {
            rowk[t] = a[(size_t)k * G + t] * pinv;   // new row k (its pivot entry fixed below)
            colk[t] = a[(size_t)t * G + k];
        }
        __syncthreads();
        for (int i = warp; i < G; i += nw) {
            double* ai = a + (size_t)i * G;
            if (i == k) {
                for (int j = lane; j < G; j += 32) ai[j] = (j == k) ? pinv : rowk[j];
            } else {
                const double ci = colk[i];
                for (int j = lane; j < G; j += 32) ai[j] = (j == k) ? -ci * pinv : fma(-ci, rowk[j], ai[j]);
            }
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < G * G; t += blockDim.x) ac[t] = a[t];
}

// The same Gauss-Jordan inverse with the matrix held in registers: thread
// (ty = warp, tx = lane) of 16 x 32 owns rows ty + 16a (a < 10) and columns
// tx + 32b (b < 5), so G <= 160.  Step k reads the old pivot row and column
// from shared memory; the owners of row and column k+1 publish their new
// values into the other half of a double buffer, so one barrier per pivot
// suffices.  Every entry goes through the operations of k_coarse_invert in
// the same order, so both give the same bits.
constexpr int CINV_RA = 10, CINV_CB = 5, CINV_MAX = 160;
__global__ void __launch_bounds__(512, 1) k_coarse_invert_reg(int G, double* ac)
{
    __shared__ double srow[2][CINV_MAX], scol[2][CINV_MAX];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    double v[CINV_RA][CINV_CB];
#pragma unroll
    for (int a = 0; a < CINV_RA; ++a)
#pragma unroll
        for (int b = 0; b < CINV_CB; ++b) {
            const int i = ty + 16 * a, j = tx + 32 * b;
            double x = (i < G && j < G) ? ac[(size_t)i * G + j] : 0.0;
            if (i == j && i < G && x == 0.0) x = 1.0;
            v[a][b] = x;
        }
    for (int t = threadIdx.x; t < 2 * CINV_MAX; t += blockDim.x) {
        (&srow[0][0])[t] = 0.0;
        (&scol[0][0])[t] = 0.0;
    }
    __syncthreads();
    if (ty == 0)
#pragma unroll
        for (int b = 0; b < CINV_CB; ++b) srow[0][tx + 32 * b] = v[0][b];
    if (tx == 0)
#pragma unroll
        for (int a = 0; a < CINV_RA; ++a) scol[0][ty + 16 * a] = v[a][0];
    for (int k = 0; k < G; ++k) {
        __syncthreads();
        const int cur = k & 1, nxt = cur ^ 1;
        const double pinv = 1.0 / srow[cur][k];
        double rk[CINV_CB];
#pragma unroll
        for (int b = 0; b < CINV_CB; ++b) rk[b] = srow[cur][tx + 32 * b] * pinv;
        // elimination, with column k and row k selected in place
#pragma unroll
        for (int a = 0; a < CINV_RA; ++a) {
            const int i = ty + 16 * a;
            const double ci = scol[cur][i];
            const double cneg = -ci * pinv;
#pragma unroll
            for (int b = 0; b < CINV_CB; ++b) {
                const int j = tx + 32 * b;
                const double t = fma(-ci, rk[b], v[a][b]);
                v[a][b] = (i == k) ? ((j == k) ? pinv : rk[b]) : ((j == k) ? cneg : t);
            }
        }
        const int k1 = k + 1;
        if (k1 < G) {
            if ((k1 & 15) == ty)
#pragma unroll
                for (int a = 0; a < CINV_RA; ++a)
                    if (ty + 16 * a == k1)
#pragma unroll
                        for (int b = 0; b < CINV_CB; ++b) srow[nxt][tx + 32 * b] = v[a][b];
            if ((k1 & 31) == tx)
#pragma unroll
                for (int b = 0; b < CINV_CB; ++b)
                    if (tx + 32 * b == k1)
#pragma unroll
                        for (int a = 0; a < CINV_RA; ++a) scol[nxt][ty + 16 * a] = v[a][b];
        }
    }
#pragma unroll
    for (int a = 0; a < CINV_RA; ++a)
#pragma unroll
        for (int b = 0; b < CINV_CB; ++b) {
            const int i = ty + 16 * a, j = tx + 32 * b;
            if (i < G && j < G) ac[(size_t)i * G + j] = v[a][b];
        }
}

// Self-test of the solvers' bounded waits: CTA `missing` leaves its part of one
// exchange out, so that the others' waits can only end by their limit (a
// second); with missing < 0 the exchange is complete and out[CTA] gets its sum.
// 0: the counter all-reduce; 1: the tagged all-reduce; 2: one row's tagged
// record, whose failed wait goes through the all-reduce after it as in
// k_pcg64c; 3: the cluster's mbarrier, every CTA staying to the end.
enum { WAIT_COUNTER, WAIT_TAGGED, WAIT_ROW, WAIT_CLUSTER, WAIT_FORMS };
template <int FORM>
__global__ void __launch_bounds__(512, 1) k_wait_selftest(PcgDev D, int missing, double* out)
{
    constexpr int NT = 512;
    const SegView g = seg_view<false>(D);
    const int b = g.b, G = g.G;
    bool ok = false;
    if constexpr (FORM == WAIT_COUNTER) {
        if (b == missing) return;
        double v[1] = {1.0}, o[1];
        ok = grid_allreduce_v<1, 1, NT>(v, D, g, 0, o);
        if (ok && threadIdx.x == 0) out[b] = o[0];
    } else {
        unsigned long long epoch;
        if (!tag_begin<false>(D, epoch)) return;
        const TagComm comm = tag_comm(D, g, epoch);
        const double v[4] = {1.0, 0.0, 0.0, 0.0};
        double t[4] = {0.0, 0.0, 0.0, 0.0};
        PollHold hold;
        if constexpr (FORM == WAIT_TAGGED) {
            if (b != missing) {
                tag_allreduce_publish<NT, false, false>(comm, 0, v);
                ok = tag_allreduce_wait<NT, false, false>(comm, 0, t, true, hold, [] {});
            }
        } else if constexpr (FORM == WAIT_ROW) {
            if (b != missing && threadIdx.x == 0) st_tag(D.xw + b, 0.0, comm.tag(0));
            double x = 0.0;
            unsigned long long xt = 0;
            SpinLimit lim;
            const bool got = threadIdx.x != 0 || tag_wait(D.xw + (b + 1) % G, comm.tag(0), x, xt, lim, comm.status);
            tag_allreduce_publish<NT, false, false>(comm, 0, v);
            ok = tag_allreduce_wait<NT, false, false>(comm, 0, t, got, hold, [] {});
            // the CTA whose record never came is not there for the next one
            if (ok) {
                tag_allreduce_publish<NT, false, false>(comm, 1, v);
                ok = tag_allreduce_wait<NT, false, false>(comm, 1, t, true, hold, [] {});
            }
        } else {
            __shared__ ClusterShared cs;
            const uint32_t bar = smem_addr(&cs.bar[0]);
            if (threadIdx.x == 0) mbar_init(bar);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            cluster_sync();
            if (threadIdx.x == NT - 1) mbar_expect(bar, 32u * G);
            cta_reduce4<NT, false>(v, [&](int q, int j, double x) {
                const uint32_t at = smem_addr(&cs.part[0][b][q]);
                for (int c = j; c < G && b != missing; c += 8) st_async_f64(cluster_addr(at, c), x, cluster_addr(bar, c));
            });
            ok = __syncthreads_and(mbar_wait(bar, 0, comm.status));
            if (ok)
                for (int c = 0; c < G; ++c) t[0] += cs.part[0][c][0];
            cluster_sync();
        }
        if (ok && threadIdx.x == 0) out[b] = t[0];
        tag_end<false>(D, epoch);
    }
}

}  // namespace

cbs3d_status selftest_waits(int device, int form, int* incomplete, int* complete, int* sums_ok)
{
    if (form < 0 || form >= WAIT_FORMS || !incomplete || !complete || !sums_ok) return CBS3D_INVALID_INPUT;
    CUDA_OK(cudaSetDevice(device));
    constexpr int G = 4;
    const void* fns[WAIT_FORMS] = {reinterpret_cast<const void*>(k_wait_selftest<WAIT_COUNTER>),
                                   reinterpret_cast<const void*>(k_wait_selftest<WAIT_TAGGED>),
                                   reinterpret_cast<const void*>(k_wait_selftest<WAIT_ROW>),
                                   reinterpret_cast<const void*>(k_wait_selftest<WAIT_CLUSTER>)};
    PcgDev D{};
    D.N = D.nslices = G;
    const unsigned long long one = 1;
    D.rec = dalloc<TagVal>(G * 2 * REC_STRIDE);
    D.xw = dalloc<TagVal>(2 * G);
    D.epoch = dalloc<unsigned long long>(1);
    D.bar = dalloc<unsigned>(4);
    D.part = dalloc<double>(G * 16);
    D.status = dalloc<DevStatus>(1);
    double* out = dalloc<double>(G);
    CUDA_OK(cudaMemset(D.rec, 0, G * 2 * REC_STRIDE * sizeof(TagVal)));
    CUDA_OK(cudaMemset(D.xw, 0, 2 * G * sizeof(TagVal)));
    CUDA_OK(cudaMemcpy(D.epoch, &one, sizeof one, cudaMemcpyHostToDevice));
    // the incomplete exchange, then the complete one on the same records
    double sums[G] = {};
    for (int missing : {1, -1}) {
        CUDA_OK(cudaMemset(D.bar, 0, 4 * sizeof(unsigned)));
        CUDA_OK(cudaMemset(D.status, 0, sizeof(DevStatus)));
        CUDA_OK(cudaMemset(out, 0, G * sizeof(double)));
        void* args[] = {&D, &missing, &out};
        if (form == WAIT_CLUSTER) {
            cudaLaunchConfig_t cfg{};
            cudaLaunchAttribute at{};
            at.id = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim.x = G;
            at.val.clusterDim.y = at.val.clusterDim.z = 1;
            cfg.gridDim = dim3(G);
            cfg.blockDim = dim3(512);
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            CUDA_OK(cudaLaunchKernelExC(&cfg, fns[form], args));
        } else {
            CUDA_OK(cudaLaunchCooperativeKernel(fns[form], dim3(G), dim3(512), args, 0, nullptr));
        }
        CUDA_OK(cudaDeviceSynchronize());
        DevStatus h{};
        CUDA_OK(cudaMemcpy(&h, D.status, sizeof h, cudaMemcpyDeviceToHost));
        (missing < 0 ? *complete : *incomplete) = h.code;
        CUDA_OK(cudaMemcpy(sums, out, sizeof sums, cudaMemcpyDeviceToHost));
        const bool none = missing >= 0;   // no CTA may have gone on
        bool right = true;
        for (double x : sums) right = right && x == (none ? 0.0 : 512.0 * G);
        *sums_ok = (none || *sums_ok) && right;
    }
    void* ptrs[] = {D.rec, D.xw, D.epoch, D.bar, D.part, D.status, out};
    for (void* q : ptrs) cudaFree(q);
    return CBS3D_OK;
}

cbs3d_status selftest_wait_timeout(int device, int* observed)
{
    int complete = 0, sums_ok = 0, code = 0;
    const cbs3d_status rc = selftest_waits(device, WAIT_COUNTER, &code, &complete, &sums_ok);
    if (observed) *observed = code;
    return rc;
}

namespace {
// Back-to-back grid all-reduces of the single-reduction kernel's kind (three
// sums per CTA, 512-thread CTAs, one per SM), each depending on the last.
__global__ void __launch_bounds__(512, 1) k_allreduce_probe(PcgDev D, int iters, double* out)
{
    unsigned long long epoch;
    if (!tag_begin<false>(D, epoch)) return;
    const TagComm comm = tag_comm(D, seg_view<false>(D), epoch);
    PollHold hold;
    double t[4] = {0.0, 0.0, 0.0, 0.0};
    for (int i = 0; i < iters; ++i) {
        const double v[4] = {1.0 + t[0] * 1.0e-300, (double)blockIdx.x, (double)threadIdx.x, 0.0};
        tag_allreduce_publish<512, false, false>(comm, i, v);
        if (!tag_allreduce_wait<512, false, false>(comm, i, t, true, hold, [] {})) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) out[0] = t[0];
    tag_end<false>(D, epoch);
}
}  // namespace

cbs3d_status allreduce_probe(int device, int iters, double* us)
{
    if (iters < 1 || !us) return CBS3D_INVALID_INPUT;
    CUDA_OK(cudaSetDevice(device));
    int sms = 0;
    CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    sms = std::min(sms, tag_grid_max(512));
    int per = 0;
    CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_allreduce_probe, 512, 0));
    if (per < 1) return CBS3D_CUDA_ERROR;
    PcgDev D{};
    D.nslices = sms;
    const size_t nrec = static_cast<size_t>(sms) * 2 * REC_STRIDE;
    const unsigned long long one = 1;
    D.rec = dalloc<TagVal>(nrec);
    D.epoch = dalloc<unsigned long long>(1);
    CUDA_OK(cudaMemset(D.rec, 0, nrec * sizeof(TagVal)));
    CUDA_OK(cudaMemcpy(D.epoch, &one, sizeof one, cudaMemcpyHostToDevice));
    D.status = dalloc<DevStatus>(1);
    double* out = dalloc<double>(1);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cbs3d_status rc = CBS3D_OK;
    float ms = 0.0f;
    CUDA_OK(cudaEventCreate(&e0));
    CUDA_OK(cudaEventCreate(&e1));
    for (int rep = 0; rep < 2 && rc == CBS3D_OK; ++rep) {   // the first launch warms up
        CUDA_OK(cudaMemset(D.status, 0, sizeof(DevStatus)));
        void* args[] = {&D, &iters, &out};
        CUDA_OK(cudaEventRecord(e0));
        CUDA_OK(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_allreduce_probe), dim3(sms), dim3(512),
                                            args, 0, nullptr));
        CUDA_OK(cudaEventRecord(e1));
        CUDA_OK(cudaEventSynchronize(e1));
        CUDA_OK(cudaEventElapsedTime(&ms, e0, e1));
        DevStatus h{};
        CUDA_OK(cudaMemcpy(&h, D.status, sizeof h, cudaMemcpyDeviceToHost));
        if (h.code != 0) rc = static_cast<cbs3d_status>(h.code);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(D.rec);
    cudaFree(D.epoch);
    cudaFree(D.status);
    cudaFree(out);
    if (rc == CBS3D_OK) *us = 1.0e3 * ms / iters;
    return rc;
}

cbs3d_status coarse_inverse(int device, int g, const double* a, double* ainv, int variant)
{
    if (!a || !ainv || g < 1 || (variant != 0 && variant != 1) || g > (variant == 0 ? CINV_MAX : 164))
        return CBS3D_INVALID_INPUT;
    CUDA_OK(cudaSetDevice(device));
    const size_t bytes = static_cast<size_t>(g) * g * sizeof(double);
    double* d = dalloc<double>(static_cast<size_t>(g) * g);
    cudaError_t e = cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        if (variant == 0) {
            k_coarse_invert_reg<<<1, 512>>>(g, d);
        } else {
            const size_t ismem = (static_cast<size_t>(g) * g + 2 * static_cast<size_t>(g)) * 8;
            e = raise_smem_limit(reinterpret_cast<const void*>(k_coarse_invert), ismem);
            if (e == cudaSuccess) k_coarse_invert<<<1, 512, ismem>>>(g, d);
        }
        if (e == cudaSuccess) e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpy(ainv, d, bytes, cudaMemcpyDeviceToHost);
    }
    cudaFree(d);
    CUDA_OK(e);
    return CBS3D_OK;
}

// ============================================================ PcgEngine
namespace {

// Placement of one CTA's halo in shared memory.  A warp's neighbour gather
// reads 32 doubles of the halo per slot (one per row of the slice); a double
// at halo position h sits in the bank pair h mod 16, and two lanes of a half
// warp whose values share a bank pair without sharing the value cost an
// extra shared-memory wavefront.  The order of the halo changes no value and
// no sum, so within every aligned block of 32 positions the block's entries
// (32 consecutive columns) are placed greedily: entries that occur in the
// most half-warp gathers first, each at the free position of the block
// whose bank pair has the fewest entries already placed in those gathers
// (weighted quadratically).  A block keeps its 32 entries, so the staging
// loads of each warp touch the same L2 sectors as in column order (a global
// bank placement spread them over 2.5x the sectors and made the 64^3
// iteration 17% slower).  64^3 jittered cavity, 148 CTAs: half-warp
// wavefronts of the gathers 666,745 -> 485,378 per iteration (ideal
// 391,104).  lc: the slots' halo indices (column order) of slices
// sb..se-1, offset by a0; returns pos, the position of each entry.
void bank_spread_halo(int nh, const unsigned short* lc, const long long* slice_off, const int* slice_w, int sb,
                      int se, long long a0, std::vector<int>& pos)
{
    std::vector<std::vector<int>> in_grp(static_cast<size_t>(nh));
    int ng = 0;
    for (int s = sb; s < se; ++s)
        for (int u = 0; u < slice_w[s]; ++u)
            for (int hw = 0; hw < 2; ++hw, ++ng)
                for (int l = 16 * hw; l < 16 * hw + 16; ++l) {
                    auto& v = in_grp[lc[slice_off[s] - a0 + 32 * u + l]];
                    if (v.empty() || v.back() != ng) v.push_back(ng);
                }
    std::vector<unsigned char> cnt(static_cast<size_t>(ng) * 16, 0);
    pos.assign(static_cast<size_t>(nh), 0);
    for (int b0 = 0; b0 < nh; b0 += 32) {
        const int b1 = std::min(nh, b0 + 32);
        int order[32];
        bool used[32] = {};
        for (int e = b0; e < b1; ++e) order[e - b0] = e;
        std::stable_sort(order, order + (b1 - b0), [&](int x, int y) {
            return in_grp[static_cast<size_t>(x)].size() > in_grp[static_cast<size_t>(y)].size();
        });
        for (int i = 0; i < b1 - b0; ++i) {
            const int e = order[i];
            const auto& gs = in_grp[static_cast<size_t>(e)];
            int best = -1;
            long long bc = 0;
            for (int j = 0; j < b1 - b0; ++j) {
                if (used[j]) continue;
                const int bank = (b0 + j) & 15;
                long long c = 0;
                for (int q : gs) {
                    const long long k = cnt[static_cast<size_t>(q) * 16 + bank];
                    c += 4 * k * k + k;
                }
                if (best < 0 || c < bc) { bc = c; best = j; }
            }
            used[best] = true;
            pos[static_cast<size_t>(e)] = b0 + best;
            const int bank = (b0 + best) & 15;
            for (int q : gs) {
                unsigned char& k = cnt[static_cast<size_t>(q) * 16 + bank];
                if (k < 255) ++k;
            }
        }
    }
}

// Shared-memory wavefronts of the neighbour gathers of slices sb..se-1 with
// the halo entries at `pos`: per slot and half warp, the largest number of
// distinct entries sharing a bank pair (at least one).
long long gather_wavefronts(const unsigned short* lc, const long long* slice_off, const int* slice_w, int sb, int se,
                            long long a0, const std::vector<int>& pos)
{
    long long w = 0;
    for (int s = sb; s < se; ++s)
        for (int u = 0; u < slice_w[s]; ++u)
            for (int hw = 0; hw < 2; ++hw) {
                int seen[16], nseen = 0, cnt[16] = {};
                for (int l = 16 * hw; l < 16 * hw + 16; ++l) {
                    const int p = pos[lc[slice_off[s] - a0 + 32 * u + l]];
                    bool dup = false;
                    for (int q = 0; q < nseen; ++q) dup = dup || seen[q] == p;
                    if (dup) continue;
                    seen[nseen++] = p;
                    ++cnt[p & 15];
                }
                int m = 1;
                for (int b = 0; b < 16; ++b) m = std::max(m, cnt[b]);
                w += m;
            }
    return w;
}

// Remote halo entries and own rows' places of the single-reduction kernel,
// built CTA by CTA from its halo's columns in order of their place.
struct RemoteLists {
    std::vector<int> ptr{0}, own;
    std::vector<int2> rem;
    int most = 0;
    explicit RemoteLists(size_t rows) : own(rows, 0xffff) {}
    // rows [r0, r1) belong to the CTA; cols[place] = row position
    void add_cta(int r0, int r1, const std::vector<int>& cols)
    {
        const size_t first = rem.size();
        for (size_t e = 0; e < cols.size(); ++e) {
            const int c = cols[e], place = static_cast<int>(e);
            int& o = own[static_cast<size_t>(c)];
            if (c >= r0 && c < r1) {
                o = (o & ~0xffff) | place;
            } else {
                o |= 1 << 16;
                rem.push_back(make_int2(c, place));
            }
        }
        // by row: a warp's requests touch neighbouring records
        std::sort(rem.begin() + static_cast<std::ptrdiff_t>(first), rem.end(), [](const int2& a, const int2& b) { return a.x < b.x; });
        ptr.push_back(static_cast<int>(rem.size()));
        most = std::max(most, static_cast<int>(rem.size() - first));
    }
};

// What each CTA of a cluster pushes to the others: (own row, consumer << 16 |
// entry), from the remote lists of CTAs whose rows start at row0[c].
void push_lists(const RemoteLists& r, const std::vector<int>& row0, std::vector<int>& ptr, std::vector<int2>& push, int& most)
{
    const int G = static_cast<int>(row0.size()) - 1;
    std::vector<std::vector<int2>> of(static_cast<size_t>(G));
    for (int c = 0; c < G; ++c)
        for (int e = r.ptr[static_cast<size_t>(c)]; e < r.ptr[static_cast<size_t>(c) + 1]; ++e) {
            const int row = r.rem[static_cast<size_t>(e)].x;
            const int o = static_cast<int>(std::upper_bound(row0.begin(), row0.end(), row) - row0.begin()) - 1;
            of[static_cast<size_t>(o)].push_back(make_int2(row - row0[static_cast<size_t>(o)], c << 16 | (e - r.ptr[static_cast<size_t>(c)])));
        }
    ptr.assign(1, 0);
    push.clear();
    most = 0;
    for (auto& v : of) {
        push.insert(push.end(), v.begin(), v.end());
        ptr.push_back(static_cast<int>(push.size()));
        most = std::max(most, static_cast<int>(v.size()));
    }
}

// k_pcg64c's dynamic shared memory: the halo's z, the remote entries (r, s,
// inverse diagonal, row, place), then the local columns at lcs_off
size_t cgcg_lcs_off(int hmax, int rem_max)
{
    return (static_cast<size_t>(hmax) * 8 + static_cast<size_t>(rem_max) * 30 + 15) & ~static_cast<size_t>(15);
}
// bytes of local columns of a CTA's slices [sb, se): every warp's rows padded
// to its widest slice, rounded up to `ch` slots
size_t cgcg_lcs_bytes(const int* slice_w, int sb, int se, int nwarps, int ch)
{
    size_t n = 0;
    for (int w = 0; w < nwarps && sb + w < se; ++w) {
        int m = 0, rows = 0;
        for (int q = sb + w; q < se; q += nwarps, ++rows) m = std::max(m, slice_w[q]);
        n += static_cast<size_t>(rows) * ((m + ch - 1) / ch * ch) * 64;
    }
    return n;
}
// the largest halo whose byte offsets fit 16 bits
constexpr int CGCG_HALO_MAX = 8190;
// k_pcg64c's form for a halo of hmax entries (with the spare place), rem_max
// of them remote, and lcsb bytes of columns: the remote entries' state in
// shared memory where it fits `limit` bytes, else in global memory, r and s
// staying where they alone fit.  64^3 without coordinates: 226,880 bytes in
// the first form, 167,920 in the second.
struct CgcgLayout {
    bool rg;
    size_t lcs, rs, bytes;
    CgcgLayout(int hmax, int rem_max, size_t lcsb, size_t limit, bool global_only = false)
        : rg(global_only || hmax - 1 > CGCG_HALO_MAX || cgcg_lcs_off(hmax, rem_max) + lcsb > limit),
          lcs(rg ? (8 * static_cast<size_t>(hmax) + 15) & ~static_cast<size_t>(15) : cgcg_lcs_off(hmax, rem_max)), rs(0),
          bytes(lcs + lcsb)
    {
        const size_t off = (bytes + 15) & ~static_cast<size_t>(15), with = off + 16 * static_cast<size_t>(rem_max);
        if (rg && rem_max > 0 && with <= limit) {
            rs = off;
            bytes = with;
        }
    }
};
constexpr size_t CGCG_SMEM_MAX = 220 * 1024;
// The second form is taken with r and s in shared memory and up to four rows
// per thread: 64^3 without coordinates 10.25 us per iteration against 11.6 on
// the global-vector kernel, a 900x16x16 channel 10.4 against 12.2; at five
// rows (70^3) 22.6 against 14.1, with r and s in global memory (a 1200x16x16
// channel) 20.7 against 14.5.
constexpr int RG_ROWS_MAX = 4;

// The remote entries and their state's initial content.
std::vector<RemoteState> remote_states(const std::vector<int2>& rem)
{
    std::vector<RemoteState> o;
    for (const int2& e : rem) o.push_back(RemoteState{0.0, e.x, e.y});
    return o;
}

// The rows split over g CTAs of nwarps warps: each CTA's halo (the distinct
// columns of its slots) in the order of its places in shared memory, its
// slots' columns as places, its remote entries, and the largest of each.
struct Partition {
    std::vector<int> hptr, hidx;
    std::vector<unsigned short> lcol;
    int hmax = 0;            // halo entries
    long long smax = 0;      // slots
    RemoteLists remote;
    size_t lcsb = 0;         // bytes of k_pcg64c's padded local columns
    bool fits = true;        // every place fits 16 bits
    explicit Partition(size_t rows) : remote(rows) {}
};
Partition partition_rows(const PressurePattern& P, const std::vector<int>& colp, int g, int nwarps)
{
    Partition o(static_cast<size_t>(P.nslices) * 32);
    o.hptr.assign(static_cast<size_t>(g) + 1, 0);
    o.lcol.assign(static_cast<size_t>(P.nslots), 0);
    std::vector<int> cols, hpos, hcols;
    for (int bb = 0; bb < g; ++bb) {
        const int sb = static_cast<int>(static_cast<long long>(bb) * P.nslices / g);
        const int se = static_cast<int>(static_cast<long long>(bb + 1) * P.nslices / g);
        const long long a0 = P.slice_off[static_cast<size_t>(sb)], a1 = P.slice_off[static_cast<size_t>(se)];
        cols.assign(colp.begin() + a0, colp.begin() + a1);
        std::sort(cols.begin(), cols.end());
        cols.erase(std::unique(cols.begin(), cols.end()), cols.end());
        if (cols.size() > 65535) { o.fits = false; return o; }
        for (long long t = a0; t < a1; ++t)
            o.lcol[static_cast<size_t>(t)] = static_cast<unsigned short>(
                std::lower_bound(cols.begin(), cols.end(), colp[static_cast<size_t>(t)]) - cols.begin());
        // the halo's order in shared memory: bank-spread
        const int nh = static_cast<int>(cols.size());
        bank_spread_halo(nh, o.lcol.data() + a0, P.slice_off.data(), P.slice_w.data(), sb, se, a0, hpos);
        for (long long t = a0; t < a1; ++t)
            o.lcol[static_cast<size_t>(t)] = static_cast<unsigned short>(hpos[o.lcol[static_cast<size_t>(t)]]);
        hcols.resize(cols.size());
        for (int e = 0; e < nh; ++e) hcols[static_cast<size_t>(hpos[static_cast<size_t>(e)])] = cols[static_cast<size_t>(e)];
        o.hidx.insert(o.hidx.end(), hcols.begin(), hcols.end());
        o.hptr[static_cast<size_t>(bb) + 1] = static_cast<int>(o.hidx.size());
        o.hmax = std::max(o.hmax, nh);
        o.smax = std::max(o.smax, a1 - a0);
        o.remote.add_cta(sb * 32, se * 32, hcols);
        o.lcsb = std::max(o.lcsb, cgcg_lcs_bytes(P.slice_w.data(), sb, se, nwarps, CGCG_ROUND));
    }
    return o;
}

// Halos of the global-vector kernels: each CTA's slices in the fewest parts (at
// most 8) of which each part's halo (16 bytes an entry) fits shared memory, the
// single-reduction kernel's table of the CTA's slices behind it included.
struct GlobalHalo {
    int parts = 0;           // 0: none fits
    int hmax = 0;
    size_t table = 0, table_bytes = 0;   // offset and size of the slice table
    std::vector<int> hptr, hidx;
    std::vector<unsigned short> lcol;
};
// 227 KB less the kernels' static shared memory (2,064 bytes)
constexpr size_t GLOBAL_SMEM_MAX = 229888;
GlobalHalo global_halo_in_parts(const PressurePattern& P, const std::vector<int>& colp, int g, bool with_table)
{
    GlobalHalo o;
    o.lcol.assign(static_cast<size_t>(P.nslots), 0);
    o.table_bytes = with_table ? static_cast<size_t>((P.nslices + g - 1) / g) * sizeof(int2) : 0;
    std::vector<int> cols;
    for (int kp = 1; kp <= 8 && o.parts == 0; ++kp) {
        o.hptr.assign(static_cast<size_t>(g) * kp + 1, 0);
        o.hidx.clear();
        o.hmax = 0;
        bool fits = true;
        for (int bb = 0; bb < g && fits; ++bb) {
            const int sb = static_cast<int>(static_cast<long long>(bb) * P.nslices / g);
            const int se = static_cast<int>(static_cast<long long>(bb + 1) * P.nslices / g);
            for (int q = 0; q < kp && fits; ++q) {
                const int pb = sb + static_cast<int>(static_cast<long long>(q) * (se - sb) / kp);
                const int pe = sb + static_cast<int>(static_cast<long long>(q + 1) * (se - sb) / kp);
                const long long a0 = P.slice_off[static_cast<size_t>(pb)], a1 = P.slice_off[static_cast<size_t>(pe)];
                cols.assign(colp.begin() + a0, colp.begin() + a1);
                std::sort(cols.begin(), cols.end());
                cols.erase(std::unique(cols.begin(), cols.end()), cols.end());
                const size_t bytes = cols.size() * 16 + 16;
                if (cols.size() > 65535 || bytes > 220 * 1024 || bytes + o.table_bytes > GLOBAL_SMEM_MAX) { fits = false; break; }
                for (long long t = a0; t < a1; ++t)
                    o.lcol[static_cast<size_t>(t)] = static_cast<unsigned short>(
                        std::lower_bound(cols.begin(), cols.end(), colp[static_cast<size_t>(t)]) - cols.begin());
                o.hidx.insert(o.hidx.end(), cols.begin(), cols.end());
                o.hptr[static_cast<size_t>(bb) * kp + q + 1] = static_cast<int>(o.hidx.size());
                o.hmax = std::max(o.hmax, static_cast<int>(cols.size()));
            }
        }
        if (fits) o.parts = kp;
    }
    o.table = static_cast<size_t>(o.hmax) * 16 + 16;
    return o;
}

// Columns as row positions: the solver works in row-position order.
std::vector<int> columns_by_position(const PressurePattern& P, int N)
{
    std::vector<int> pos_of(static_cast<size_t>(N), 0);
    for (size_t p = 0; p < P.row_node.size(); ++p)
        if (P.row_node[p] >= 0) pos_of[static_cast<size_t>(P.row_node[p])] = static_cast<int>(p);
    std::vector<int> colp(static_cast<size_t>(P.nslots));
    for (size_t t = 0; t < colp.size(); ++t) colp[t] = pos_of[static_cast<size_t>(P.col[t])];
    return colp;
}

// Each CTA's neighbours for the two-level kernel (itself and the owners of
// its halo entries), and every halo entry's owner as its place in that list.
struct CoarseNeighbours {
    std::vector<int> ptr{0}, ids;
    std::vector<unsigned char> hown;
    int most = 0;
    bool fits = true;        // every place fits 8 bits
};
CoarseNeighbours coarse_neighbours(int nslices, const std::vector<int>& hptr, const std::vector<int>& hidx)
{
    CoarseNeighbours o;
    const int G = static_cast<int>(hptr.size()) - 1;
    std::vector<int> cta_of_slice(static_cast<size_t>(nslices), 0);
    for (int b = 0; b < G; ++b) {
        const int sb = static_cast<int>(static_cast<long long>(b) * nslices / G);
        const int se = static_cast<int>(static_cast<long long>(b + 1) * nslices / G);
        for (int q = sb; q < se; ++q) cta_of_slice[static_cast<size_t>(q)] = b;
    }
    o.hown.assign(hidx.size(), 0);
    for (int b = 0; b < G; ++b) {
        std::vector<int> l(1, b);
        for (int k = hptr[static_cast<size_t>(b)]; k < hptr[static_cast<size_t>(b) + 1]; ++k)
            l.push_back(cta_of_slice[static_cast<size_t>(hidx[static_cast<size_t>(k)] / 32)]);
        std::sort(l.begin(), l.end());
        l.erase(std::unique(l.begin(), l.end()), l.end());
        if (l.size() > 255) { o.fits = false; return o; }
        for (int k = hptr[static_cast<size_t>(b)]; k < hptr[static_cast<size_t>(b) + 1]; ++k) {
            const int w = cta_of_slice[static_cast<size_t>(hidx[static_cast<size_t>(k)] / 32)];
            o.hown[static_cast<size_t>(k)] = static_cast<unsigned char>(std::lower_bound(l.begin(), l.end(), w) - l.begin());
        }
        o.ids.insert(o.ids.end(), l.begin(), l.end());
        o.ptr.push_back(static_cast<int>(o.ids.size()));
        o.most = std::max(o.most, static_cast<int>(l.size()));
    }
    return o;
}

// Instantiations of the single-reduction kernels by rows per thread, batch
// mode and CTA size.
// ... of the batch's 256-thread CTAs
template <bool RG>
const void* fn_cgcg_batch256(int rmax)
{
    return rmax == 1 ? reinterpret_cast<const void*>(k_pcg64c<1, true, 256, 0, 0, false, RG>)
         : rmax == 2 ? reinterpret_cast<const void*>(k_pcg64c<2, true, 256, 0, 0, false, RG>)
         : rmax == 4 ? reinterpret_cast<const void*>(k_pcg64c<4, true, 256, 0, 0, false, RG>)
                     : reinterpret_cast<const void*>(k_pcg64c<8, true, 256, 0, 0, false, RG>);
}
template <bool BATCH, int NT>
const void* fn_mixed(int rmax)
{
    return rmax == 1 ? reinterpret_cast<const void*>(k_pcg32m<1, BATCH, NT>)
         : rmax == 2 ? reinterpret_cast<const void*>(k_pcg32m<2, BATCH, NT>)
         : rmax == 4 ? reinterpret_cast<const void*>(k_pcg32m<4, BATCH, NT>)
                     : reinterpret_cast<const void*>(k_pcg32m<8, BATCH, NT>);
}
const void* fn_twolevel(int rmax)
{
    return rmax == 1 ? reinterpret_cast<const void*>(k_pcg64d<1>)
         : rmax == 2 ? reinterpret_cast<const void*>(k_pcg64d<2>)
         : rmax == 4 ? reinterpret_cast<const void*>(k_pcg64d<4>)
                     : reinterpret_cast<const void*>(k_pcg64d<8>);
}
// The single-case kernel by rows per thread: kt > 0 with that many rows'
// coefficients in tensor memory (every row up to four per thread, else the
// first four), ks = 1 with the first row's in shared memory ahead of them,
// kt = 0 with all of them streamed from L2 (one row per thread keeps them in
// registers).
const void* fn_cgcg_single(int rmax, int ks, int kt)
{
    if (ks && kt)
        return rmax == 2 ? reinterpret_cast<const void*>(k_pcg64c<2, false, 512, 1, 1>)
                         : reinterpret_cast<const void*>(k_pcg64c<4, false, 512, 1, 3>);
    if (kt)
        return rmax == 2 ? reinterpret_cast<const void*>(k_pcg64c<2, false, 512, 0, 2>)
             : rmax == 3 ? reinterpret_cast<const void*>(k_pcg64c<3, false, 512, 0, 3>)
             : rmax == 4 ? reinterpret_cast<const void*>(k_pcg64c<4, false, 512, 0, 4>)
             : rmax == 5 ? reinterpret_cast<const void*>(k_pcg64c<5, false, 512, 0, 4>)
                         : reinterpret_cast<const void*>(k_pcg64c<6, false, 512, 0, 4>);
    return rmax == 1 ? reinterpret_cast<const void*>(k_pcg64c<1, false, 512>)
         : rmax == 2 ? reinterpret_cast<const void*>(k_pcg64c<2, false, 512>)
         : rmax == 3 ? reinterpret_cast<const void*>(k_pcg64c<3, false, 512>)
         : rmax == 4 ? reinterpret_cast<const void*>(k_pcg64c<4, false, 512>)
         : rmax == 5 ? reinterpret_cast<const void*>(k_pcg64c<5, false, 512>)
                     : reinterpret_cast<const void*>(k_pcg64c<6, false, 512>);
}

// ... with the remote entries' state in global memory, up to four rows
template <bool BATCH>
const void* fn_cgcg_rg(int rmax)
{
    return rmax == 1 ? reinterpret_cast<const void*>(k_pcg64c<1, BATCH, 512, 0, 0, false, true>)
         : rmax == 2 ? reinterpret_cast<const void*>(k_pcg64c<2, BATCH, 512, 0, 2, false, true>)
         : rmax == 3 ? reinterpret_cast<const void*>(k_pcg64c<3, BATCH, 512, 0, 3, false, true>)
                     : reinterpret_cast<const void*>(k_pcg64c<4, BATCH, 512, 0, 4, false, true>);
}

// ... of the batch, one 512-thread CTA per SM
const void* fn_cgcg_batch512(int rmax)
{
    return rmax == 1 ? reinterpret_cast<const void*>(k_pcg64c<1, true, 512>)
         : rmax == 2 ? reinterpret_cast<const void*>(k_pcg64c<2, true, 512, 0, 2>)
         : rmax == 3 ? reinterpret_cast<const void*>(k_pcg64c<3, true, 512, 0, 3>)
         : rmax == 4 ? reinterpret_cast<const void*>(k_pcg64c<4, true, 512, 0, 4>)
         : rmax == 5 ? reinterpret_cast<const void*>(k_pcg64c<5, true, 512, 0, 4>)
         : rmax == 6 ? reinterpret_cast<const void*>(k_pcg64c<6, true, 512, 0, 4>)
                     : reinterpret_cast<const void*>(k_pcg64c<8, true, 512, 0, 4>);
}
// ... with rows wider than tensor memory holds (up to four)
const void* fn_cgcg_batch512_wide(int rmax)
{
    return rmax == 2 ? reinterpret_cast<const void*>(k_pcg64c<2, true, 512>)
         : rmax == 3 ? reinterpret_cast<const void*>(k_pcg64c<3, true, 512>)
                     : reinterpret_cast<const void*>(k_pcg64c<4, true, 512>);
}
// ... and the form that runs on one cluster
const void* fn_cgcg_cluster() { return reinterpret_cast<const void*>(k_pcg64c<1, false, 512, 0, 0, true>); }

// The mixed batch, and tilings whose 512-thread CTAs do not fit, run
// 256-thread CTAs, two per SM, with their coefficients streamed from L2.
constexpr int BATCH_THREADS = 256;

}  // namespace

void coarse_invert_launch(int g, double* a, cudaStream_t st)
{
    k_coarse_invert_reg<<<1, 512, 0, st>>>(g, a);
}

namespace {
// Whether the two-level kernel can run on a partition over G CTAs: its layout,
// and the coarse inverse's, in one CTA's shared memory.
bool two_level_fits(const CoarseNeighbours& nb, int G, int rows, int halo_max, int slot_max, int sms, size_t& smem,
                    size_t& ismem)
{
    if (G > 160 || !nb.fits) return false;
    smem = TwoLevelLayout(halo_max, slot_max, nb.most, G).bytes;
    ismem = (static_cast<size_t>(G) * G + 2 * static_cast<size_t>(G)) * 8;
    const void* fn = fn_twolevel(rows);
    int per = 0;
    const bool ok = smem <= 220 * 1024 && ismem <= 220 * 1024 && raise_smem_limit(fn, smem) == cudaSuccess &&
                    raise_smem_limit(reinterpret_cast<const void*>(k_coarse_invert), ismem) == cudaSuccess &&
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, 512, smem) == cudaSuccess && per * sms >= G;
    cudaGetLastError();
    return ok;
}
}  // namespace

cudaError_t pcg_raise_smem_limit(const void* fn, size_t smem) { return raise_smem_limit(fn, smem); }

cbs3d_status probe_partition(int nelem, int npoin, const int* intma, const int* mat_elem, const double* coord, int ctas,
                             cbs3d_pcg_partition* out)
{
    if (nelem < 1 || npoin < 1 || !intma || ctas < 1 || !out) return CBS3D_INVALID_INPUT;
    const std::vector<int> conn(intma, intma + 4 * static_cast<size_t>(nelem));
    for (int v : conn)
        if (v < 1 || v > npoin) return CBS3D_INVALID_INPUT;
    std::vector<int> mat(static_cast<size_t>(nelem), 0), n2e_ptr, n2e;
    if (mat_elem) mat.assign(mat_elem, mat_elem + nelem);
    build_incidence(conn, npoin, n2e_ptr, n2e);
    PressurePattern P;
    build_pressure_pattern(conn, mat, npoin, n2e_ptr, n2e, P, coord);
    const int g = std::min(ctas, P.nslices);
    const Partition part = partition_rows(P, columns_by_position(P, npoin), g, PCG_THREADS / 32);
    const GlobalHalo gh = global_halo_in_parts(P, columns_by_position(P, npoin), g, true);
    *out = cbs3d_pcg_partition{};
    out->ctas = g;
    out->single_form = -1;
    out->global_parts = gh.parts;
    out->global_bytes = static_cast<long long>(gh.table + gh.table_bytes);
    if (!part.fits) return CBS3D_OK;
    const CoarseNeighbours nb = coarse_neighbours(P.nslices, part.hptr, part.hidx);
    const int hmax = part.hmax + 1;   // the spare place
    const CgcgLayout lay(hmax, part.remote.most, part.lcsb, CGCG_SMEM_MAX);
    out->halo_max = hmax;
    out->slot_max = static_cast<int>(part.smax);
    out->remote_max = part.remote.most;
    out->neighbour_max = nb.most;
    out->single_form = lay.bytes > CGCG_SMEM_MAX ? -1 : !lay.rg ? 0 : lay.rs ? 1 : 2;
    out->two_level_bytes = static_cast<long long>(TwoLevelLayout(hmax, out->slot_max, nb.most, g).bytes);
    out->single_bytes = static_cast<long long>(lay.bytes);
    return CBS3D_OK;
}

int PcgEngine::launches_per_solve() const
{
    if (mgh) return 3 + mgh->launches_per_setup();
    return coarse ? 5 : 3;
}

void PcgEngine::build_coarse(const HostModel& m, const std::vector<int>& colp)
{
    const int G = nblocks;
    const PressurePattern& P = m.pat;
    std::vector<int> cta_of_slice(static_cast<size_t>(nslices), 0);
    for (int b = 0; b < G; ++b) {
        const int sb = static_cast<int>(static_cast<long long>(b) * nslices / G);
        const int se = static_cast<int>(static_cast<long long>(b + 1) * nslices / G);
        for (int q = sb; q < se; ++q) cta_of_slice[static_cast<size_t>(q)] = b;
    }
    std::vector<char> fixed(static_cast<size_t>(N), 0), freep(static_cast<size_t>(NP), 0);
    for (int v : m.bc_list) fixed[static_cast<size_t>(v - 1)] = 1;
    for (int pos = 0; pos < NP; ++pos) {
        const int node = P.row_node[static_cast<size_t>(pos)];
        freep[static_cast<size_t>(pos)] = node >= 0 && m.tf[static_cast<size_t>(node)] && !fixed[static_cast<size_t>(node)];
    }
    // entries of every nonzero block (I, J) of P^T A P, ascending
    std::vector<std::vector<int>> blocks(static_cast<size_t>(G) * G);
    for (int q = 0; q < nslices; ++q) {
        const int I = cta_of_slice[static_cast<size_t>(q)];
        for (int lane = 0; lane < 32; ++lane) {
            const int pos = q * 32 + lane;
            if (!freep[static_cast<size_t>(pos)]) continue;
            blocks[static_cast<size_t>(I) * G + I].push_back(-(pos + 1));
            for (int k = 0; k < P.slice_w[static_cast<size_t>(q)]; ++k) {
                const long long t = P.slice_off[static_cast<size_t>(q)] + lane + 32LL * k;
                const int c = colp[static_cast<size_t>(t)];
                if (!freep[static_cast<size_t>(c)]) continue;
                blocks[static_cast<size_t>(I) * G + cta_of_slice[static_cast<size_t>(c / 32)]].push_back(static_cast<int>(t));
            }
        }
    }
    std::vector<int> ptr(1, 0), ent;
    std::vector<int2> ij;
    for (int I = 0; I < G; ++I)
        for (int J = 0; J < G; ++J) {
            auto& v = blocks[static_cast<size_t>(I) * G + J];
            if (v.empty()) continue;
            std::sort(v.begin(), v.end());
            ent.insert(ent.end(), v.begin(), v.end());
            ptr.push_back(static_cast<int>(ent.size()));
            ij.push_back(make_int2(I, J));
        }
    const CoarseNeighbours nb = coarse_neighbours(nslices, h_hptr, h_hidx);
    npairs = static_cast<int>(ij.size());
    d_pair_ptr = dalloc<int>(ptr.size());
    d_pair_ij = dalloc<int2>(ij.size());
    d_pair_ent = dalloc<int>(ent.size());
    d_ac = dalloc<double>(static_cast<size_t>(G) * G);
    d_nbr_ptr = dalloc<int>(nb.ptr.size());
    d_nbr_ids = dalloc<int>(nb.ids.size());
    d_hown = dalloc<unsigned char>(nb.hown.size());
    CUDA_OK(cudaMemcpy(d_pair_ptr, ptr.data(), ptr.size() * sizeof(int), cudaMemcpyHostToDevice));
    CUDA_OK(cudaMemcpy(d_pair_ij, ij.data(), ij.size() * sizeof(int2), cudaMemcpyHostToDevice));
    CUDA_OK(cudaMemcpy(d_pair_ent, ent.data(), ent.size() * sizeof(int), cudaMemcpyHostToDevice));
    CUDA_OK(cudaMemcpy(d_nbr_ptr, nb.ptr.data(), nb.ptr.size() * sizeof(int), cudaMemcpyHostToDevice));
    CUDA_OK(cudaMemcpy(d_nbr_ids, nb.ids.data(), nb.ids.size() * sizeof(int), cudaMemcpyHostToDevice));
    if (!nb.hown.empty()) CUDA_OK(cudaMemcpy(d_hown, nb.hown.data(), nb.hown.size(), cudaMemcpyHostToDevice));
    cdev = CoarseDev{G, nb.most, d_nbr_ptr, d_nbr_ids, d_hown, d_ac};
    coarse = true;
}

void PcgEngine::init(const HostModel& m, const uint8_t* nflag, const double* pfix, DevStatus* status,
                     int device, int blocks_override, bool mixed_mode, int kernel_choice, bool two_level,
                     bool multigrid)
{
    N = m.N;
    E = m.E;
    mixed = mixed_mode;
    const PressurePattern& P = m.pat;
    nslices = P.nslices;
    nslots = P.nslots;
    ncontrib = static_cast<long long>(P.cent.size());
    nnz_offdiag = 0;
    for (size_t q = 0; q + 1 < P.cptr.size(); ++q) nnz_offdiag += (P.cptr[q + 1] > P.cptr[q]) ? 1 : 0;
    NP = nslices * 32;
    d_row_node = dalloc<int>(P.row_node.size());
    CUDA_OK(cudaMemcpy(d_row_node, P.row_node.data(), P.row_node.size() * sizeof(int), cudaMemcpyHostToDevice));
    const std::vector<int> colp = columns_by_position(P, N);
    d_slice_off = dalloc<long long>(P.slice_off.size());
    d_slice_w = dalloc<int>(P.slice_w.size());
    d_col = dalloc<int>(static_cast<size_t>(nslots));
    d_cptr = dalloc<long long>(P.cptr.size());
    d_cent = dalloc<int>(static_cast<size_t>(ncontrib));
    d_val = dalloc<double>(static_cast<size_t>(nslots));
    CUDA_OK(cudaMemcpy(d_slice_off, P.slice_off.data(), P.slice_off.size() * sizeof(long long), cudaMemcpyHostToDevice));
    CUDA_OK(cudaMemcpy(d_slice_w, P.slice_w.data(), P.slice_w.size() * sizeof(int), cudaMemcpyHostToDevice));
    if (nslots) CUDA_OK(cudaMemcpy(d_col, colp.data(), static_cast<size_t>(nslots) * sizeof(int), cudaMemcpyHostToDevice));
    CUDA_OK(cudaMemcpy(d_cptr, P.cptr.data(), P.cptr.size() * sizeof(long long), cudaMemcpyHostToDevice));
    if (ncontrib) CUDA_OK(cudaMemcpy(d_cent, P.cent.data(), static_cast<size_t>(ncontrib) * sizeof(int), cudaMemcpyHostToDevice));
    CUDA_OK(cudaMemset(d_val, 0, static_cast<size_t>(nslots ? nslots : 1) * sizeof(double)));
    const size_t n = static_cast<size_t>(NP);
    d_r = dalloc<double>(2 * n); d_z = dalloc<double>(n); d_pA = dalloc<double>(n);
    d_pB = dalloc<double>(n); d_q = dalloc<double>(2 * n);
    d_xp = dalloc<double>(n); d_bp = dalloc<double>(n); d_dp = dalloc<double>(n);
    d_fp = dalloc<uint8_t>(n);
    CUDA_OK(cudaMemset(d_pB, 0, n * sizeof(double)));
    if (mixed) {
        d_val32 = dalloc<float>(static_cast<size_t>(nslots));
        d_f32 = dalloc<float>(8 * n);
        CUDA_OK(cudaMemset(d_f32, 0, 8 * n * sizeof(float)));
    }
    d_nflag = nflag;
    d_pfix = pfix;
    d_status = status;

    int sms = 0;
    CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    // Register-resident kernel when every thread's rows fit its register
    // arrays; otherwise the kernel that keeps the vectors in global memory.
    auto grid_for = [&](const void* fn) {
        int per_sm = 0;
        CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, PCG_THREADS, 0));
        int g = sms * (per_sm < 2 ? per_sm : 2);
        if (blocks_override > 0 && blocks_override < g) g = blocks_override;
        if (g > nslices) g = nslices > 0 ? nslices : 1;
        return g;
    };
    // whether a cluster of `c` CTAs of a kernel can run with `bytes` of shared memory
    auto cluster_fits = [&](const void* fk, int c, size_t bytes) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = static_cast<unsigned>(c);
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.gridDim = dim3(static_cast<unsigned>(c));
        cfg.blockDim = dim3(PCG_THREADS);
        cfg.dynamicSmemBytes = bytes;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        const bool ok = bytes <= 227 * 1024 && raise_smem_limit(fk, bytes) == cudaSuccess &&
                        cudaFuncSetAttribute(fk, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&n, fk, &cfg) == cudaSuccess && n >= 1;
        cudaGetLastError();
        return ok;
    };
    auto upload_partition = [&](const Partition& part, int hmax) {
        d_halo_ptr = dalloc<int>(part.hptr.size());
        d_halo_idx = dalloc<int>(part.hidx.size());
        d_lcol = dalloc<unsigned short>(part.lcol.size());
        CUDA_OK(cudaMemcpy(d_halo_ptr, part.hptr.data(), part.hptr.size() * sizeof(int), cudaMemcpyHostToDevice));
        CUDA_OK(cudaMemcpy(d_halo_idx, part.hidx.data(), part.hidx.size() * sizeof(int), cudaMemcpyHostToDevice));
        if (!part.lcol.empty()) CUDA_OK(cudaMemcpy(d_lcol, part.lcol.data(), part.lcol.size() * sizeof(unsigned short), cudaMemcpyHostToDevice));
        dev_halo_max = hmax;
        dev_slot_max = static_cast<int>(part.smax);
        h_hptr = part.hptr;
        h_hidx = part.hidx;
    };
    bool coarse_planned = false;
    rmax = 0;
    variant = 1;
    nblocks = grid_for(reinterpret_cast<const void*>(k_pcg64<false>));
    if (kernel_choice == 0 || kernel_choice == 3 || kernel_choice == 4 || kernel_choice == 10 || kernel_choice == 11) {
        const void* hc3[4] = {reinterpret_cast<const void*>(k_pcg64h<1>), reinterpret_cast<const void*>(k_pcg64h<2>),
                              reinterpret_cast<const void*>(k_pcg64h<4>), reinterpret_cast<const void*>(k_pcg64h<8>)};
        const int want = kernel_choice == 3 ? 3 : 4;
        const int nt = PCG_THREADS, nwarps = nt / 32;
        // rows per thread: the mixed and the two-level kernel ("special") have
        // 1, 2, 4 and 8; the single-reduction kernel up to six (beyond, the
        // global-vector kernel is as fast: 76^3 22.0 us per iteration against
        // 25.4 with eight rows).  A mesh that the special kernel does not fit
        // is tiled as without the option (76^3 in mixed precision, a step: 25.2
        // ms with eight rows, 16.4 on the kernel that Jacobi takes there).
        struct Tiling { int rows; bool cluster, special; };
        std::vector<Tiling> tilings;
        if (want == 3 || mixed || two_level)
            for (int r : {1, 2, 4, 8}) tilings.push_back({r, false, want == 4});
        if (want == 4) {
            // one cluster where it holds the mesh at one row per thread (16^3
            // 2.00 us per iteration against 2.37 on the whole chip; at two
            // rows 3.0 against 2.4, as the chip then has one row per thread)
            if (kernel_choice == 0 && blocks_override <= 0 && nslices <= CLUSTER_MAX * nwarps) tilings.push_back({1, true, false});
            for (int r = 1; r <= 6; ++r) tilings.push_back({r, false, false});
        }
        bool special_fits = true;
        for (int c = 0; c < static_cast<int>(tilings.size()) && variant == 1; ++c) {
            const int rr = tilings[static_cast<size_t>(c)].rows;
            const bool cl = tilings[static_cast<size_t>(c)].cluster;
            const bool special = tilings[static_cast<size_t>(c)].special;
            if (special && !special_fits) continue;
            const void* fn = want == 3 ? hc3[c] : special ? fn_mixed<false, 512>(rr) : fn_cgcg_single(rr, 0, 0);
            int per_sm = 0;
            CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, nt, 0));
            int g = want == 4 ? std::min(sms, tag_grid_max(nt)) : sms * (per_sm < 2 ? per_sm : 2);
            if (cl) g = (nslices + nwarps * rr - 1) / (nwarps * rr);
            if (blocks_override > 0 && blocks_override < g) g = blocks_override;
            if (g > nslices) g = nslices > 0 ? nslices : 1;
            const int per_cta = (nslices + g - 1) / g;
            if ((per_cta + nwarps - 1) / nwarps > rr) continue;
            Partition part = partition_rows(P, colp, g, nwarps);
            int hmax = part.hmax;
            const long long smax = part.smax;
            const RemoteLists& remote = part.remote;
            if (!part.fits) {
                special_fits = false;
                continue;
            }
            if (want == 4) ++hmax;   // the spare place
            if (special) {
                const size_t ms = static_cast<size_t>(hmax) * 16 + static_cast<size_t>(smax) * 6 + 16;
                mixed_ok = mixed && ms <= 220 * 1024 && raise_smem_limit(fn, ms) == cudaSuccess &&
                           cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, nt, ms) == cudaSuccess && per_sm * sms >= g;
                cudaGetLastError();
                // the two-level kernel needs rows for every warp of the grid
                const bool two = !mixed_ok && two_level && nslices >= 16 * sms &&
                                 two_level_fits(coarse_neighbours(nslices, part.hptr, part.hidx), g, rr, hmax,
                                                static_cast<int>(smax), sms, coarse_smem, coarse_ismem);
                if (!mixed_ok && !two) {
                    special_fits = false;
                    continue;
                }
                mixed_smem = ms;
                coarse_planned = two;
                variant = 4;
                nthreads = nt;
                rmax = rr;
                nblocks = g;
                rem_total = static_cast<long long>(remote.rem.size());
                upload_partition(part, hmax);
                break;
            }
            const CgcgLayout lay(hmax, remote.most, part.lcsb, CGCG_SMEM_MAX);
            const bool rg = want == 4 && lay.rg;
            const size_t smem = want == 4 ? lay.bytes : static_cast<size_t>(hmax) * 12 + static_cast<size_t>(smax) * 2 + 16;
            if ((rg && (cl || !lay.rs || rr > RG_ROWS_MAX)) || smem > (want == 4 ? CGCG_SMEM_MAX : 200 * 1024)) {
                // more rows per thread on the same grid need as much
                if (want == 4 && !cl) break;
                continue;
            }
            if (rg) fn = fn_cgcg_rg<false>(rr);
            std::vector<int> pptr;
            std::vector<int2> push;
            int pmost = 0;
            cluster = 0;
            size_t cl_off = 0, cl_smem = 0;
            if (cl) {
                std::vector<int> row0;
                for (int bb = 0; bb <= g; ++bb) row0.push_back(32 * static_cast<int>(static_cast<long long>(bb) * nslices / g));
                push_lists(remote, row0, pptr, push, pmost);
                cl_off = (smem + 15) & ~static_cast<size_t>(15);
                cl_smem = cl_off + static_cast<size_t>(remote.most) * 16 + static_cast<size_t>(rr) * nt * 8 + static_cast<size_t>(pmost) * 6;
                if (cluster_fits(fn_cgcg_cluster(), g, cl_smem + static_cast<size_t>(rr) * nt * 8 + 16)) cluster = g;
                else continue;
            }
            CUDA_OK(raise_smem_limit(fn, smem));
            CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, nt, smem));
            if (per_sm * sms < g) continue;
            variant = want;
            nthreads = nt;
            rmax = rr;
            nblocks = g;
            halo_smem = smem;
            cgcg_smem = smem;
            cgcg_rg = rg;
            cgcg_rs_off = rg ? static_cast<int>(lay.rs) : 0;
            // Tensor memory: 128 columns = 64 doubles per thread, the slots
            // of a row padded to the widest slice of the mesh.  Up to four
            // rows all live there, of more the first four; choice 11 (two or
            // four rows) keeps the first in shared memory instead, where it
            // fits beside the halo.  The grid must be resident with one CTA
            // per SM: each CTA takes all 512 columns, so a second one on the
            // SM would wait for the first to finish.
            cgcg_ks = cgcg_kt = 0;
            cgcg_coef_off = cgcg_tm_w = 0;
            if (cluster) cgcg_smem = cl_smem;
            auto resident = [&](int ks, int kt, size_t bytes) {
                if (cluster) return cluster_fits(fn_cgcg_cluster(), g, bytes);
                const void* fk = rg ? fn : fn_cgcg_single(rr, ks, kt);
                int per2 = 0;
                const bool ok = bytes <= 227 * 1024 && raise_smem_limit(fk, bytes) == cudaSuccess &&
                                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per2, fk, nt, bytes) == cudaSuccess &&
                                per2 * sms >= g;
                cudaGetLastError();
                return ok;
            };
            if (want == 4 && kernel_choice != 10) {
                int wmx = 0;
                for (int q = 0; q < nslices; ++q) wmx = std::max(wmx, P.slice_w[static_cast<size_t>(q)]);
                const int chw = CGCG_ROUND, tw = (wmx + chw - 1) / chw * chw;
                if (kernel_choice == 11 && !rg && (rr == 2 || rr == 4) && tw > 0 && (rr - 1) * tw <= 64) {
                    long long cmax = 0;
                    for (int bb = 0; bb < g; ++bb) {
                        const int sb = static_cast<int>(static_cast<long long>(bb) * nslices / g);
                        const int se = static_cast<int>(static_cast<long long>(bb + 1) * nslices / g);
                        const int sc = std::min(sb + nwarps, se);
                        cmax = std::max(cmax, P.slice_off[static_cast<size_t>(sc)] - P.slice_off[static_cast<size_t>(sb)]);
                    }
                    const size_t off = (cgcg_smem + 15) & ~static_cast<size_t>(15);
                    if (resident(1, rr - 1, off + static_cast<size_t>(cmax) * 8)) {
                        cgcg_ks = 1;
                        cgcg_kt = rr - 1;
                        cgcg_smem = off + static_cast<size_t>(cmax) * 8;
                        cgcg_coef_off = static_cast<int>(off);
                    }
                }
                const int kt = rr == 1 ? 0 : std::min(rr, 4);
                if (rg) {
                    // the slots of a row that fit; any others stream from L2
                    if (kt > 0) cgcg_tm_w = std::min(tw, 64 / kt / chw * chw);
                } else {
                    if (!cgcg_ks && kt > 0 && tw > 0 && kt * tw <= 64 && resident(0, kt, cgcg_smem)) cgcg_kt = kt;
                    if (cgcg_kt) cgcg_tm_w = tw;
                }
            }
            // the rows' diagonal in shared memory (64^3: 12.05 -> 11.95 us
            // per iteration; in registers it was slower)
            cgcg_pds_off = 0;
            if (want == 4) {
                const size_t off = (cgcg_smem + 15) & ~static_cast<size_t>(15);
                const size_t with = off + static_cast<size_t>(rr) * nt * 8;
                if (resident(cgcg_ks, cgcg_kt, with)) {
                    cgcg_smem = with;
                    cgcg_pds_off = static_cast<int>(off);
                }
            }
            // ... and their pressure, where the kernel keeps it in memory
            cgcg_xs_off = 0;
            if (want == 4 && (rr == 3 || rr > 4)) {
                const size_t off = (cgcg_smem + 15) & ~static_cast<size_t>(15);
                const size_t with = off + static_cast<size_t>(rr) * nt * 8;
                if (resident(cgcg_ks, cgcg_kt, with)) {
                    cgcg_smem = with;
                    cgcg_xs_off = static_cast<int>(off);
                }
            }
            upload_partition(part, hmax);
            if (want == 4) {
                dev_rem_max = remote.most;
                rem_total = static_cast<long long>(remote.rem.size());
                cgcg_lcs = static_cast<int>(lay.lcs);
                d_rem_ptr = dalloc<int>(remote.ptr.size());
                d_rem = dalloc<int2>(remote.rem.size());
                d_own = dalloc<int>(remote.own.size());
                CUDA_OK(cudaMemcpy(d_rem_ptr, remote.ptr.data(), remote.ptr.size() * sizeof(int), cudaMemcpyHostToDevice));
                if (!remote.rem.empty()) CUDA_OK(cudaMemcpy(d_rem, remote.rem.data(), remote.rem.size() * sizeof(int2), cudaMemcpyHostToDevice));
                if (rg) {
                    const std::vector<RemoteState> st = remote_states(remote.rem);
                    d_rem_state = dalloc<RemoteState>(st.size());
                    CUDA_OK(cudaMemcpy(d_rem_state, st.data(), st.size() * sizeof(RemoteState), cudaMemcpyHostToDevice));
                }
                CUDA_OK(cudaMemcpy(d_own, remote.own.data(), remote.own.size() * sizeof(int), cudaMemcpyHostToDevice));
                if (cluster) {
                    cgcg_cl_off = static_cast<int>(cl_off);
                    dev_push_max = pmost;
                    d_push_ptr = dalloc<int>(pptr.size());
                    d_push = dalloc<int2>(push.size());
                    CUDA_OK(cudaMemcpy(d_push_ptr, pptr.data(), pptr.size() * sizeof(int), cudaMemcpyHostToDevice));
                    if (!push.empty()) CUDA_OK(cudaMemcpy(d_push, push.data(), push.size() * sizeof(int2), cudaMemcpyHostToDevice));
                }
            }
        }
    }
    if (variant == 1 && N > 0 && kernel_choice != 2) {
        // the global-vector kernel with its neighbour values staged in shared
        // memory: each CTA's slices in the fewest parts (at most 8) whose
        // halos fit
        // automatic and choice 5: the single-reduction kernel; choice 1:
        // the two-reduction one (bitwise the same arithmetic as choices 2, 3)
        global_cgcg = kernel_choice != 1;
        const int g = global_cgcg ? std::min(nblocks, tag_grid_max(PCG_THREADS)) : nblocks;
        const void* fh = global_cgcg ? reinterpret_cast<const void*>(k_pcg64g) : reinterpret_cast<const void*>(k_pcg64<true>);
        const GlobalHalo H = global_halo_in_parts(P, colp, g, global_cgcg);
        const size_t smem = H.table + H.table_bytes;
        // the slices' slots and widths behind the halo, and rows per warp in
        // tensor memory: rounds of eight slots, 2.5 columns per slot of 128
        cgcg_tm_w = g_tm_rows = cgcg_lcs = 0;
        if (global_cgcg) {
            cgcg_lcs = static_cast<int>(H.table);
            int wmx = 0;
            for (int q = 0; q < nslices; ++q) wmx = std::max(wmx, P.slice_w[static_cast<size_t>(q)]);
            const int tw = (wmx + 7) / 8 * 8;
            if (tw > 0 && 5 * tw <= 256 && g <= sms) {
                cgcg_tm_w = tw;
                g_tm_rows = 256 / (5 * tw);
            }
        }
        int per = 0;
        if (H.parts > 0 && raise_smem_limit(fh, smem) == cudaSuccess &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fh, PCG_THREADS, smem) == cudaSuccess && per * sms >= g) {
            d_halo_ptr = dalloc<int>(H.hptr.size());
            d_halo_idx = dalloc<int>(H.hidx.size());
            d_lcol = dalloc<unsigned short>(H.lcol.size());
            CUDA_OK(cudaMemcpy(d_halo_ptr, H.hptr.data(), H.hptr.size() * sizeof(int), cudaMemcpyHostToDevice));
            CUDA_OK(cudaMemcpy(d_halo_idx, H.hidx.data(), H.hidx.size() * sizeof(int), cudaMemcpyHostToDevice));
            CUDA_OK(cudaMemcpy(d_lcol, H.lcol.data(), H.lcol.size() * sizeof(unsigned short), cudaMemcpyHostToDevice));
            dev_halo_max = H.hmax;
            nblocks = g;
            global_halo_parts = H.parts;
            global_halo = true;
            global_halo_smem = smem;
            global_halo_total = static_cast<long long>(H.hidx.size());
            // the slots that tensor memory holds (every other row of a warp)
            g_tm_slots = 0;
            for (int bb = 0; bb < g * PCG_WARPS; ++bb) {
                const int b = bb / PCG_WARPS, warp = bb % PCG_WARPS;
                const int sb = static_cast<int>(static_cast<long long>(b) * nslices / g);
                const int se = static_cast<int>(static_cast<long long>(b + 1) * nslices / g);
                for (int q = 0, left = g_tm_rows; q < H.parts; ++q) {
                    const int p1 = sb + static_cast<int>(static_cast<long long>(q + 1) * (se - sb) / H.parts);
                    for (int sl = sb + static_cast<int>(static_cast<long long>(q) * (se - sb) / H.parts) + warp;
                         sl < p1 && left > 0; sl += 2 * PCG_WARPS, --left)
                        g_tm_slots += 32LL * P.slice_w[static_cast<size_t>(sl)];
                }
            }
        } else {
            cgcg_tm_w = g_tm_rows = cgcg_lcs = 0;
        }
        cudaGetLastError();
    }
    // register-resident rows with their neighbours gathered from L2: choice 2,
    // and where no halo fits (80^3: 71 us per iteration against 24 with one)
    if (variant == 1 && (kernel_choice == 2 || (kernel_choice != 1 && kernel_choice != 5 && !global_halo))) {
        const int rm[4] = {1, 2, 4, 8};
        const void* cands[4] = {reinterpret_cast<const void*>(k_pcg64r<1>), reinterpret_cast<const void*>(k_pcg64r<2>),
                                reinterpret_cast<const void*>(k_pcg64r<4>), reinterpret_cast<const void*>(k_pcg64r<8>)};
        for (int c = 0; c < 4; ++c) {
            const int g = grid_for(cands[c]);
            const int per_cta = (nslices + g - 1) / g;
            if ((per_cta + PCG_WARPS - 1) / PCG_WARPS <= rm[c]) { rmax = rm[c]; nblocks = g; variant = 2; break; }
        }
    }
    if (coarse_planned) build_coarse(m, colp);
    if (multigrid && !mixed && !coarse) {
        mgh = new MgHierarchy;
        bool ok = false;
        try {
            ok = mgh->build(m, colp, nflag, d_slice_off, d_slice_w, d_col, device, sms, blocks_override);
        } catch (...) {
            mgh->release();
            delete mgh;
            mgh = nullptr;
            throw;
        }
        if (!ok) {
            // the caller asked for multigrid: say why it runs Jacobi-PCG instead
            std::fprintf(stderr, "cbs3d: multigrid preconditioner unavailable for this mesh (%s); "
                                 "Jacobi-PCG is used\n", mgh->why.c_str());
            mgh->release();
            delete mgh;
            mgh = nullptr;
        }
    }
    d_part = dalloc<double>(static_cast<size_t>(nblocks) * 16);
    d_bar = dalloc<unsigned>(4);
    d_out = dalloc<CgOut>(1);
    CUDA_OK(cudaMemset(d_bar, 0, 4 * sizeof(unsigned)));
    if (variant == 4 || global_cgcg) {
        const size_t nx = variant == 4 ? 2 * n : 0, nrec = static_cast<size_t>(nblocks) * 2 * REC_STRIDE;
        d_rec = dalloc<TagVal>(nrec);
        d_xw = dalloc<TagVal>(nx);
        d_epoch = dalloc<unsigned long long>(1);
        const unsigned long long one = 1;   // tags are never 0, the records' first content
        CUDA_OK(cudaMemset(d_rec, 0, nrec * sizeof(TagVal)));
        if (nx) CUDA_OK(cudaMemset(d_xw, 0, nx * sizeof(TagVal)));
        CUDA_OK(cudaMemcpy(d_epoch, &one, sizeof one, cudaMemcpyHostToDevice));
    }

    dev = PcgDev{};
    dev.N = NP; dev.E = E; dev.nslices = nslices; dev.nblocks = nblocks;
    dev.slice_off = d_slice_off; dev.slice_w = d_slice_w; dev.col = d_col; dev.val = d_val;
    dev.val32 = d_val32; dev.cptr = d_cptr; dev.cent = d_cent;
    dev.nflag = d_nflag; dev.pfix = d_pfix;
    dev.r = d_r; dev.z = d_z; dev.pA = d_pA; dev.pB = d_pB; dev.q = d_q;
    if (mixed) {
        dev.r32 = d_f32; dev.w32 = d_f32 + 2 * n; dev.s32 = d_f32 + 4 * n;
        dev.p32 = d_f32 + 6 * n; dev.dz32 = d_f32 + 7 * n;
    }
    dev.slot_max = dev_slot_max;
    dev.part = d_part; dev.bar = d_bar; dev.status = d_status; dev.out = d_out;
    dev.halo_ptr = d_halo_ptr; dev.halo_idx = d_halo_idx; dev.lcol = d_lcol; dev.halo_max = dev_halo_max;
    dev.rec = d_rec; dev.xw = d_xw; dev.epoch = d_epoch;
    dev.push_ptr = d_push_ptr; dev.push = d_push; dev.push_max = dev_push_max; dev.cl_off = cgcg_cl_off;
    dev.rem_ptr = d_rem_ptr; dev.rem = d_rem; dev.own = d_own; dev.rem_max = dev_rem_max;
    dev.rem_state = d_rem_state; dev.rs_off = cgcg_rs_off;
    dev.lcs_off = cgcg_lcs;
    dev.coef_off = cgcg_coef_off;
    dev.pds_off = cgcg_pds_off;
    dev.xs_off = cgcg_xs_off;
    dev.tm_w = cgcg_tm_w;
    dev.tm_rows = g_tm_rows;
    dev.halo_parts = global_halo ? global_halo_parts : 0;
    dev.row_node = d_row_node;
}

void PcgEngine::release()
{
    if (mgh) {
        mgh->release();
        delete mgh;
        mgh = nullptr;
    }
    mg_ready = false;
    void* ptrs[] = {d_slice_off, d_slice_w, d_col, d_cptr, d_cent, d_val, d_val32, d_r, d_z, d_pA,
                    d_pB, d_q, d_f32, d_part, d_bar, d_out, d_halo_ptr, d_halo_idx, d_lcol, d_row_node,
                    d_rec, d_xw, d_epoch, d_rem_ptr, d_rem, d_own, d_push_ptr, d_push, d_rem_state,
                    d_xp, d_bp, d_dp, d_fp, d_pair_ptr, d_pair_ij, d_pair_ent, d_ac, d_nbr_ptr, d_nbr_ids, d_hown};
    for (void* p : ptrs) if (p) cudaFree(p);
    d_pair_ptr = nullptr; d_pair_ij = nullptr; d_pair_ent = nullptr; d_ac = nullptr;
    d_nbr_ptr = nullptr; d_nbr_ids = nullptr; d_hown = nullptr;
    coarse = false;
    d_rec = d_xw = nullptr; d_epoch = nullptr; d_rem_ptr = d_own = d_push_ptr = nullptr; d_rem = d_push = nullptr;
    d_rem_state = nullptr;
    d_slice_off = nullptr; d_slice_w = nullptr; d_col = nullptr; d_cptr = nullptr; d_cent = nullptr;
    d_val = nullptr; d_val32 = nullptr; d_r = d_z = d_pA = d_pB = d_q = nullptr; d_f32 = nullptr;
    d_part = nullptr; d_bar = nullptr; d_out = nullptr;
    d_halo_ptr = nullptr; d_halo_idx = nullptr; d_lcol = nullptr; d_row_node = nullptr;
    d_xp = d_bp = d_dp = nullptr; d_fp = nullptr;
}

void PcgEngine::coarse_setup(const double* pdiag, const int* row_node, cudaStream_t st)
{
    const int G = nblocks;
    CUDA_OK(cudaMemsetAsync(d_ac, 0, static_cast<size_t>(G) * G * sizeof(double), st));
    k_coarse_blocks<<<static_cast<unsigned>(npairs), 256, 0, st>>>(d_pair_ptr, d_pair_ij, d_pair_ent, d_val, pdiag,
                                                                  row_node, G, d_ac);
    if (G <= CINV_MAX)
        k_coarse_invert_reg<<<1, 512, 0, st>>>(G, d_ac);
    else
        k_coarse_invert<<<1, 512, coarse_ismem, st>>>(G, d_ac);
}

void PcgEngine::prepare_coarse(const double* d_pdiag_node, cudaStream_t st)
{
    if (mgh) {
        mgh->setup(d_val, d_pdiag_node, d_row_node, st);
        mg_ready = true;
        return;
    }
    if (!coarse) return;
    coarse_setup(d_pdiag_node, d_row_node, st);
    coarse_ready = true;
}

void PcgEngine::assemble_from_state(const DevState& S, cudaStream_t st)
{
    if (!nslots) return;
    const int T = 256;
    k_ell_from_state<<<static_cast<unsigned>((nslots + T - 1) / T), T, 0, st>>>(S, d_cptr, d_cent, d_val, d_val32, nslots);
}

void PcgEngine::assemble_from_gstif(const double* gstif, cudaStream_t st)
{
    if (!nslots) return;
    const int T = 256;
    k_ell_from_gstif<<<static_cast<unsigned>((nslots + T - 1) / T), T, 0, st>>>(gstif, d_cptr, d_cent, d_val, d_val32, nslots);
}

void PcgEngine::multiply(const double* pdiag, const double* x, double* y, cudaStream_t st)
{
    PcgDev D = dev;
    D.pdiag = const_cast<double*>(pdiag);
    k_ell_multiply<<<(nslices * 32 + 255) / 256, 256, 0, st>>>(D, x, y);
}

cbs3d_status PcgEngine::solve(double* pres, double* rhs1, double* pdiag, int precond, int conv_test,
                              int max_iter, double rel_tol, double abs_tol, cudaStream_t st, bool sync,
                              cudaEvent_t ev0, cudaEvent_t ev1)
{
    PcgDev D = dev;
    D.pres = pres; D.rhs1 = rhs1; D.pdiag = pdiag;
    D.precond = precond; D.conv_test = conv_test; D.max_iter = max_iter;
    D.rel_tol = rel_tol; D.abs_tol = abs_tol; D.inner_tol = inner_tol;
    k_impose_perm_in<<<(NP + 255) / 256, 256, 0, st>>>(D, d_xp, d_bp, d_dp, d_fp);
    D.pres = d_xp; D.rhs1 = d_bp; D.pdiag = d_dp; D.nflag = d_fp;
    // the counter of the kernels that do not exchange tagged records
    if (!(variant == 4 && !coarse) && !(global_halo && global_cgcg)) CUDA_OK(cudaMemsetAsync(d_bar, 0, 4 * sizeof(unsigned), st));
    CUDA_OK(cudaMemsetAsync(d_out, 0, sizeof(CgOut), st));
    void* args[] = {&D};
    const void* fn = !global_halo ? reinterpret_cast<const void*>(k_pcg64<false>)
                     : global_cgcg ? reinterpret_cast<const void*>(k_pcg64g)
                                   : reinterpret_cast<const void*>(k_pcg64<true>);
    size_t smem = global_halo ? global_halo_smem : 0;
    if (variant == 2) {
        if (rmax == 1) fn = reinterpret_cast<const void*>(k_pcg64r<1>);
        else if (rmax == 2) fn = reinterpret_cast<const void*>(k_pcg64r<2>);
        else if (rmax == 4) fn = reinterpret_cast<const void*>(k_pcg64r<4>);
        else fn = reinterpret_cast<const void*>(k_pcg64r<8>);
    } else if (variant == 3) {
        if (rmax == 1) fn = reinterpret_cast<const void*>(k_pcg64h<1>);
        else if (rmax == 2) fn = reinterpret_cast<const void*>(k_pcg64h<2>);
        else if (rmax == 4) fn = reinterpret_cast<const void*>(k_pcg64h<4>);
        else fn = reinterpret_cast<const void*>(k_pcg64h<8>);
        smem = halo_smem;
    } else if (variant == 4 && mixed_ok) {
        fn = fn_mixed<false, 512>(rmax);
        smem = mixed_smem;
    } else if (variant == 4) {
        fn = cluster ? fn_cgcg_cluster() : cgcg_rg ? fn_cgcg_rg<false>(rmax) : fn_cgcg_single(rmax, cgcg_ks, cgcg_kt);
        smem = cgcg_smem;
    }
    CoarseDev C = cdev;
    void* args2[] = {&D, &C};
    if (coarse) {
        // the aggregated operator of this solve and its inverse, unless
        // prepare_coarse made them already
        if (!coarse_ready) coarse_setup(d_dp, nullptr, st);
        coarse_ready = false;
        fn = fn_twolevel(rmax);
        smem = coarse_smem;
    }
    if (mgh && precond == 1) {
        // the multigrid set-up of this solve, unless prepare_coarse made it
        if (!mg_ready) mgh->setup(d_val, d_dp, nullptr, st);
        mg_ready = false;
        if (ev0) CUDA_OK(cudaEventRecord(ev0, st));
        mgh->launch(D, st);
        if (ev1) CUDA_OK(cudaEventRecord(ev1, st));
    } else {
        mg_ready = false;
        if (ev0) CUDA_OK(cudaEventRecord(ev0, st));
        if (cluster) {
            // one cluster: its CTAs run together by that alone
            cudaLaunchConfig_t cfg{};
            cudaLaunchAttribute at{};
            at.id = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim.x = static_cast<unsigned>(cluster);
            at.val.clusterDim.y = at.val.clusterDim.z = 1;
            cfg.gridDim = dim3(static_cast<unsigned>(cluster));
            cfg.blockDim = dim3(nthreads);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = st;
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            CUDA_OK(cudaLaunchKernelExC(&cfg, fn, args));
        } else {
            CUDA_OK(cudaLaunchCooperativeKernel(fn, dim3(nblocks), dim3(nthreads), coarse ? args2 : args, smem, st));
        }
        if (ev1) CUDA_OK(cudaEventRecord(ev1, st));
    }
    k_perm_out<<<(NP + 255) / 256, 256, 0, st>>>(D, d_xp, pres);
    if (sync) CUDA_OK(cudaStreamSynchronize(st));
    return CBS3D_OK;
}

cbs3d_status PcgEngine::read_result(cbs3d_cg_result& r, cudaStream_t st)
{
    CgOut o{};
    CUDA_OK(cudaMemcpyAsync(&o, d_out, sizeof o, cudaMemcpyDeviceToHost, st));
    CUDA_OK(cudaStreamSynchronize(st));
    std::memset(&r, 0, sizeof r);
    r.iterations = o.iterations;
    r.initial_l2 = o.initial_l2;
    r.final_l2 = o.final_l2;
    r.final_relative_l2 = o.rel;
    r.final_max_abs = o.max_abs;
    r.converged = o.converged;
    r.matvec_calls = o.iterations + 1;
    r.outer_sweeps = o.outer;
    return o.converged ? CBS3D_OK : CBS3D_NOT_CONVERGED;
}

size_t PcgEngine::bytes_per_iter() const
{
    if (mgh) {
        // level 0: three products (pre-smoothing residual, post-smoothing,
        // A p) over the coefficients; per node the pressure read and written,
        // z and q written and read back, the smoothed residual written and
        // read by the restriction; coarse levels: two products each
        size_t b = static_cast<size_t>(nnz_offdiag) * 24 + static_cast<size_t>(N) * 64;
        for (int l = 1; l < mgh->Lc; ++l)
            b += static_cast<size_t>(mgh->n[static_cast<size_t>(l)]) * (16 * mgh->W[static_cast<size_t>(l)] + 48);
        return b;
    }
    if (variant == 4 && mixed_ok) {
        // coefficients resident in shared memory; per node: r, w, s of the
        // previous iteration read once for staging (12), r, s, w written (12),
        // pressure read and written (16), pdiag read (8)
        return static_cast<size_t>(N) * 48;
    }
    if (variant == 4) {
        // coefficient per pair entry and the diagonal per node (both on chip
        // for the solve); per remote halo entry the record of its w written
        // and read (32)
        return static_cast<size_t>(nnz_offdiag) * 8 + static_cast<size_t>(N) * 8 + static_cast<size_t>(rem_total) * 32;
    }
    if (variant == 3) {
        // coefficient per pair entry; per node: halo staging of z and the
        // previous direction (each node is in about one CTA's halo per owner
        // plus the overlap, counted once here), z read back, new direction and
        // z written, pressure read and written
        return static_cast<size_t>(nnz_offdiag) * 8 + static_cast<size_t>(N) * 56;
    }
    if (rmax > 0) {
        // coefficient + column per pair entry; per node the z and previous
        // direction gathered once, z read back, new direction and z written,
        // pressure read and written
        return static_cast<size_t>(nnz_offdiag) * 12 + static_cast<size_t>(N) * 56;
    }
    // Phase A: coefficient + column per pair entry; z and previous p of the
    // row (16 B), pdiag (8), new p written (8), q written (8), node flag (1).
    // Phase B: q, r, pres, pdiag read (32), r, pres, z written (24).  With the
    // shared-memory halo the columns are 16-bit and every halo entry's z and
    // previous p are read once per iteration.
    if (global_halo && global_cgcg) {
        // single reduction: coefficient + 16-bit column per pair entry, but
        // for the rows in tensor memory; per node r, s, w of the previous
        // iteration, p, pressure, inverse diagonal and diagonal read (56),
        // node flag (1), p, pressure and the new r, s, w written (40); per
        // halo entry r, s, w (24) and, with several parts per CTA, the inverse
        // diagonal (8).  What L2 serves of that is counted too.
        const double streamed = nslots > 0 ? 1.0 - static_cast<double>(g_tm_slots) / static_cast<double>(nslots) : 0.0;
        return static_cast<size_t>(static_cast<double>(nnz_offdiag) * 10.0 * streamed) + static_cast<size_t>(N) * 97 +
               static_cast<size_t>(global_halo_total) * (global_halo_parts > 1 ? 32 : 24);
    }
    if (global_halo)
        return static_cast<size_t>(nnz_offdiag) * 10 + static_cast<size_t>(N) * 97 +
               static_cast<size_t>(global_halo_total) * 16;
    return static_cast<size_t>(nnz_offdiag) * 12 + static_cast<size_t>(N) * 97;
}

// ================================================================ batch
void PcgBatch::init(const std::vector<PcgBatchMember>& members, int dev_id, bool mixed_mode, double inner_tol)
{
    mem = members;
    device = dev_id;
    mixed = mixed_mode;
    const size_t K = mem.size();
    CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    gmax = 2 * sms;   // the most CTAs of a wave (two of BATCH_THREADS per SM)
    slice0.assign(K, 0); nsl.assign(K, 0); N_k.assign(K, 0);
    slot0.assign(K, 0); nslot.assign(K, 0);
    nslices = 0; nslots = 0;
    for (size_t k = 0; k < K; ++k) {
        const PressurePattern& P = mem[k].m->pat;
        slice0[k] = nslices; nsl[k] = P.nslices; N_k[k] = mem[k].m->N;
        slot0[k] = nslots; nslot[k] = P.nslots;
        nslices += P.nslices;
        nslots += P.nslots;
    }
    NP = nslices * 32;
    // concatenated pattern: global slot offsets, widths, columns as global
    // row positions, and each position's instance-local node
    h_slice_off.assign(static_cast<size_t>(nslices) + 1, 0);
    std::vector<int> sw(static_cast<size_t>(nslices), 0), rn(static_cast<size_t>(NP), -1);
    h_col.assign(static_cast<size_t>(nslots), 0);
    for (size_t k = 0; k < K; ++k) {
        const PressurePattern& P = mem[k].m->pat;
        const int p0 = slice0[k] * 32;
        std::vector<int> pos_of(static_cast<size_t>(N_k[k]), 0);
        for (size_t p = 0; p < P.row_node.size(); ++p) {
            rn[static_cast<size_t>(p0) + p] = P.row_node[p];
            if (P.row_node[p] >= 0) pos_of[static_cast<size_t>(P.row_node[p])] = p0 + static_cast<int>(p);
        }
        for (int s = 0; s < P.nslices; ++s) {
            h_slice_off[static_cast<size_t>(slice0[k] + s)] = slot0[k] + P.slice_off[static_cast<size_t>(s)];
            sw[static_cast<size_t>(slice0[k] + s)] = P.slice_w[static_cast<size_t>(s)];
        }
        for (long long t = 0; t < P.nslots; ++t)
            h_col[static_cast<size_t>(slot0[k] + t)] = pos_of[static_cast<size_t>(P.col[static_cast<size_t>(t)])];
        long long* cp = dalloc<long long>(P.cptr.size());
        int* ce = dalloc<int>(P.cent.size());
        CUDA_OK(cudaMemcpy(cp, P.cptr.data(), P.cptr.size() * sizeof(long long), cudaMemcpyHostToDevice));
        if (!P.cent.empty()) CUDA_OK(cudaMemcpy(ce, P.cent.data(), P.cent.size() * sizeof(int), cudaMemcpyHostToDevice));
        d_cptr.push_back(cp);
        d_cent.push_back(ce);
    }
    h_slice_off[static_cast<size_t>(nslices)] = nslots;
    h_slice_w = sw;
    d_slice_off = dalloc<long long>(h_slice_off.size());
    d_slice_w = dalloc<int>(sw.size());
    d_col = dalloc<int>(h_col.size());
    d_row_node = dalloc<int>(rn.size());
    CUDA_OK(cudaMemcpy(d_slice_off, h_slice_off.data(), h_slice_off.size() * sizeof(long long), cudaMemcpyHostToDevice));
    CUDA_OK(cudaMemcpy(d_slice_w, sw.data(), sw.size() * sizeof(int), cudaMemcpyHostToDevice));
    if (!h_col.empty()) CUDA_OK(cudaMemcpy(d_col, h_col.data(), h_col.size() * sizeof(int), cudaMemcpyHostToDevice));
    CUDA_OK(cudaMemcpy(d_row_node, rn.data(), rn.size() * sizeof(int), cudaMemcpyHostToDevice));
    d_lcol = dalloc<unsigned short>(static_cast<size_t>(nslots));
    d_val = dalloc<double>(static_cast<size_t>(nslots));
    CUDA_OK(cudaMemset(d_val, 0, static_cast<size_t>(nslots ? nslots : 1) * sizeof(double)));
    const size_t n = static_cast<size_t>(NP);
    d_r = dalloc<double>(2 * n); d_q = dalloc<double>(2 * n);
    d_z = dalloc<double>(n); d_pA = dalloc<double>(n); d_pB = dalloc<double>(n);
    d_xp = dalloc<double>(n); d_bp = dalloc<double>(n); d_dp = dalloc<double>(n);
    d_fp = dalloc<uint8_t>(n);
    CUDA_OK(cudaMemset(d_pB, 0, n * sizeof(double)));
    if (mixed) {
        d_val32 = dalloc<float>(static_cast<size_t>(nslots));
        d_f32 = dalloc<float>(8 * n);
        CUDA_OK(cudaMemset(d_f32, 0, 8 * n * sizeof(float)));
    }
    d_own = dalloc<int>(n);
    d_rec = dalloc<TagVal>(K * static_cast<size_t>(gmax) * 2 * REC_STRIDE);
    d_xw = dalloc<TagVal>(2 * n);
    d_epoch = dalloc<unsigned long long>(K);
    {
        const std::vector<unsigned long long> one(K, 1);   // tags are never 0, the records' first content
        CUDA_OK(cudaMemset(d_rec, 0, K * static_cast<size_t>(gmax) * 2 * REC_STRIDE * sizeof(TagVal)));
        CUDA_OK(cudaMemset(d_xw, 0, 2 * n * sizeof(TagVal)));
        CUDA_OK(cudaMemcpy(d_epoch, one.data(), K * sizeof(unsigned long long), cudaMemcpyHostToDevice));
    }
    d_out = dalloc<CgOut>(K);
    CUDA_OK(cudaMemset(d_out, 0, K * sizeof(CgOut)));

    base = PcgDev{};
    base.N = NP; base.nslices = nslices; base.inner_tol = inner_tol;
    base.slice_off = d_slice_off; base.slice_w = d_slice_w; base.col = d_col; base.val = d_val;
    base.val32 = d_val32; base.row_node = d_row_node;
    base.pres = d_xp; base.rhs1 = d_bp; base.pdiag = d_dp; base.nflag = d_fp;
    base.r = d_r; base.z = d_z; base.pA = d_pA; base.pB = d_pB; base.q = d_q;
    if (mixed) {
        base.r32 = d_f32; base.w32 = d_f32 + 2 * n; base.s32 = d_f32 + 4 * n;
        base.p32 = d_f32 + 6 * n; base.dz32 = d_f32 + 7 * n;
    }
    base.lcol = d_lcol;
    base.xw = d_xw; base.own = d_own;
}

void PcgBatch::free_waves()
{
    for (Wave& w : waves) {
        void* ptrs[] = {w.d_cta_inst, w.d_inst, w.d_hptr, w.d_hidx, w.d_rptr, w.d_rem, w.d_rem_state, w.d_rem_rs};
        for (void* p : ptrs) if (p) cudaFree(p);
    }
    waves.clear();
}

bool PcgBatch::plan(const PcgBatchPlan& p, std::string* why)
{
    // FP64: one 512-thread CTA per SM with the coefficients in tensor memory
    // (one row per thread: in registers), else two 256-thread CTAs per SM.  12
    // cavities of 10..32 hexes per side, two steps: 10.2 -> 5.7 ms.
    // Mixed: the FP32 kernel (two 256-thread CTAs per SM) where every wave's
    // coefficients fit its shared memory; a plan of which some wave would run
    // in FP64 anyway runs there as a whole (48 cavities of 10..40, a step:
    // 22.1 ms in FP32 and FP64 waves of 256 threads, 12.2 in FP64 waves of 512).
    const bool fp32 = mixed && !p.fp64;
    return (fp32 && plan_threads(p, BATCH_THREADS, true, why)) || plan_threads(p, 512, false, why) ||
           plan_threads(p, BATCH_THREADS, false, why);
}

bool PcgBatch::plan_threads(const PcgBatchPlan& p, int nt, bool all_fp32, std::string* why)
{
    const int gmax = std::min(nt == 512 ? sms : 2 * sms, tag_grid_max(nt)), nwarps = nt / 32;
    if (p.rmax != 1 && p.rmax != 2 && p.rmax != 4 && p.rmax != 8) {
        if (why) *why = "rows per thread must be 1, 2, 4 or 8";
        return false;
    }
    const int K = static_cast<int>(mem.size());
    const int cap = nwarps * p.rmax;   // slices one CTA holds in registers
    std::vector<int> minc(static_cast<size_t>(K));
    for (int k = 0; k < K; ++k) {
        minc[static_cast<size_t>(k)] = std::max(1, (nsl[static_cast<size_t>(k)] + cap - 1) / cap);
        if (minc[static_cast<size_t>(k)] > gmax) {
            if (why) *why = "instance " + std::to_string(k) + " needs more CTAs than one launch holds at this tiling";
            return false;
        }
    }
    // first-fit decreasing by slices into waves of at most gmax CTAs
    std::vector<int> order(static_cast<size_t>(K));
    for (int k = 0; k < K; ++k) order[static_cast<size_t>(k)] = k;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return nsl[static_cast<size_t>(a)] > nsl[static_cast<size_t>(b)]; });
    std::vector<std::vector<int>> packs;
    std::vector<int> used;
    for (int k : order) {
        size_t w = 0;
        while (w < packs.size() && used[w] + minc[static_cast<size_t>(k)] > gmax) ++w;
        if (w == packs.size()) { packs.emplace_back(); used.push_back(0); }
        packs[w].push_back(k);
        used[w] += minc[static_cast<size_t>(k)];
    }
    const void* c32[4] = {fn_mixed<true, BATCH_THREADS>(1), fn_mixed<true, BATCH_THREADS>(2), fn_mixed<true, BATCH_THREADS>(4),
                          fn_mixed<true, BATCH_THREADS>(8)};
    const int ci = p.rmax == 1 ? 0 : p.rmax == 2 ? 1 : p.rmax == 4 ? 2 : 3;

    struct HostWave {
        int G = 0, hmax = 0;
        long long smax = 0;
        std::vector<int> cta_inst, hptr, hidx, rptr;
        std::vector<int2> rem;
        int rmost = 0;
        size_t lcsb = 0;
        int rows = 1;            // rows per thread of the wave's kernel
        std::vector<PcgInst> inst;
    };
    std::vector<HostWave> hw(packs.size());
    std::vector<int> own(static_cast<size_t>(NP), 0xffff);
    std::vector<unsigned short> lcol(static_cast<size_t>(nslots), 0);
    for (size_t w = 0; w < packs.size(); ++w) {
        HostWave& H = hw[w];
        const std::vector<int>& mk = packs[w];
        std::vector<int> G(mk.size());
        int tot = 0;
        for (size_t j = 0; j < mk.size(); ++j) { G[j] = minc[static_cast<size_t>(mk[j])]; tot += G[j]; }
        if (p.spread) {
            // spare CTAs, one at a time, to the instance with the most slices per CTA
            while (tot < gmax) {
                int best = -1;
                double bw = 0.0;
                for (size_t j = 0; j < mk.size(); ++j) {
                    if (G[j] >= nsl[static_cast<size_t>(mk[j])]) continue;
                    const double wpc = static_cast<double>(nsl[static_cast<size_t>(mk[j])]) / G[j];
                    if (wpc > bw) { bw = wpc; best = static_cast<int>(j); }
                }
                if (best < 0) break;
                ++G[static_cast<size_t>(best)];
                ++tot;
            }
        }
        H.G = tot;
        if (nt == 512) {
            // the fewest rows per thread that hold every CTA's slices
            int most = 1;
            for (size_t j = 0; j < mk.size(); ++j) most = std::max(most, (nsl[static_cast<size_t>(mk[j])] + G[j] - 1) / G[j]);
            H.rows = (most + nwarps - 1) / nwarps;
            if (H.rows > 6) H.rows = 8;
        } else {
            H.rows = p.rmax;
        }
        H.hptr.push_back(0);
        RemoteLists remote(0);
        remote.own.swap(own);   // the rows of all waves, each in one of them
        int cta = 0;
        for (size_t j = 0; j < mk.size(); ++j) {
            const int k = mk[j];
            const PressurePattern& P = mem[static_cast<size_t>(k)].m->pat;
            PcgInst I{};
            I.cta0 = cta; I.ncta = G[j];
            I.s0 = slice0[static_cast<size_t>(k)]; I.s1 = I.s0 + nsl[static_cast<size_t>(k)];
            I.precond = mem[static_cast<size_t>(k)].m->p.cg_preconditioner;
            I.conv_test = mem[static_cast<size_t>(k)].m->p.cg_conv_test;
            I.max_iter = mem[static_cast<size_t>(k)].m->p.cg_max_iter;
            I.rel_tol = mem[static_cast<size_t>(k)].m->p.relToler;
            I.abs_tol = mem[static_cast<size_t>(k)].m->p.absToler;
            I.rec = d_rec + static_cast<size_t>(k) * static_cast<size_t>(this->gmax) * 2 * REC_STRIDE;
            I.epoch = d_epoch + k;
            I.status = mem[static_cast<size_t>(k)].d_status;
            I.out = d_out + k;
            H.inst.push_back(I);
            (void)P;
            std::vector<int> cols;
            for (int b = 0; b < G[j]; ++b) {
                H.cta_inst.push_back(static_cast<int>(j));
                const int sb = I.s0 + static_cast<int>(static_cast<long long>(b) * (I.s1 - I.s0) / G[j]);
                const int se = I.s0 + static_cast<int>(static_cast<long long>(b + 1) * (I.s1 - I.s0) / G[j]);
                const long long a0 = h_slice_off[static_cast<size_t>(sb)], a1 = h_slice_off[static_cast<size_t>(se)];
                cols.assign(h_col.begin() + a0, h_col.begin() + a1);
                std::sort(cols.begin(), cols.end());
                cols.erase(std::unique(cols.begin(), cols.end()), cols.end());
                if (cols.size() > 65535) {
                    if (why) *why = "a CTA halo exceeds 65535 columns";
                    return false;
                }
                for (long long t = a0; t < a1; ++t)
                    lcol[static_cast<size_t>(t)] = static_cast<unsigned short>(
                        std::lower_bound(cols.begin(), cols.end(), h_col[static_cast<size_t>(t)]) - cols.begin());
                H.hidx.insert(H.hidx.end(), cols.begin(), cols.end());
                H.hptr.push_back(static_cast<int>(H.hidx.size()));
                H.hmax = std::max(H.hmax, static_cast<int>(cols.size()));
                H.smax = std::max(H.smax, a1 - a0);
                remote.add_cta(sb * 32, se * 32, cols);
                H.lcsb = std::max(H.lcsb, cgcg_lcs_bytes(h_slice_w.data(), sb, se, nwarps, CGCG_ROUND));
            }
            cta += G[j];
        }
        own.swap(remote.own);
        H.rptr = std::move(remote.ptr);
        H.rem = std::move(remote.rem);
        H.rmost = remote.most;
    }
    // kernels and shared memory of every wave, before anything is replaced
    std::vector<Wave> nw(hw.size());
    for (size_t w = 0; w < hw.size(); ++w) {
        const HostWave& H = hw[w];
        Wave& W = nw[w];
        W.G = H.G; W.rmax = H.rows; W.threads = nt;
        const size_t s32 = static_cast<size_t>(H.hmax) * 16 + static_cast<size_t>(H.smax) * 6 + 16;
        auto fits = [&](const void* fn, size_t smem) {
            if (smem > 220 * 1024) return false;
            if (raise_smem_limit(fn, smem) != cudaSuccess) {
                cudaGetLastError();
                return false;
            }
            int per = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, nt, smem) != cudaSuccess) {
                cudaGetLastError();
                return false;
            }
            return per * sms >= H.G;
        };
        if (nt == 512) {
            // the slots of a row in tensor memory padded to the wave's widest
            int wmx = 0;
            for (const PcgInst& I : H.inst)
                for (int q = I.s0; q < I.s1; ++q) wmx = std::max(wmx, h_slice_w[static_cast<size_t>(q)]);
            const int ch = CGCG_ROUND, tw = (wmx + ch - 1) / ch * ch, kt = std::min(H.rows, 4);
            const CgcgLayout lay(H.hmax + 1, H.rmost, H.lcsb, CGCG_SMEM_MAX);
            // rows too wide for tensor memory stream their coefficients from
            // L2 (centred boxes of 28 and 32, rows of 26 neighbours: 8.1 ms a
            // step against 9.4 on 256-thread CTAs).  A wave on at most half
            // the SMs is faster on twice as many CTAs of 256 threads then
            // (centred boxes of 6 to 20 on the fewest CTAs: 4.2 against 5.8)
            const bool wide = !lay.rg && H.rows > 1 && kt * tw > 64;
            W.rg = lay.rg;
            W.fn = lay.rg ? fn_cgcg_rg<true>(H.rows) : wide ? fn_cgcg_batch512_wide(H.rows) : fn_cgcg_batch512(H.rows);
            W.smem = lay.bytes;
            W.lcs_off = static_cast<int>(lay.lcs);
            W.rs_off = static_cast<int>(lay.rs);
            if ((lay.rg && (!lay.rs || H.rows > RG_ROWS_MAX)) || (wide && (2 * H.G <= sms || H.rows > 4)) || !fits(W.fn, W.smem)) {
                if (why) *why = "a wave does not fit co-resident at this tiling";
                return false;
            }
            W.tm_w = std::min(tw, 64 / kt / ch * ch);
            // the rows' diagonal, and their pressure where the kernel keeps it
            // in memory, behind that
            for (int what = 0; what < 2; ++what) {
                if (what == 1 && !(H.rows == 3 || H.rows > 4)) continue;
                const size_t off = (W.smem + 15) & ~static_cast<size_t>(15), with = off + static_cast<size_t>(H.rows) * nt * 8;
                if (!fits(W.fn, with)) continue;
                (what ? W.xs_off : W.pds_off) = static_cast<int>(off);
                W.smem = with;
            }
        }
        else if (mixed && !p.fp64 && fits(c32[ci], s32)) { W.mixed = true; W.fn = c32[ci]; W.smem = s32; }
        else if (!all_fp32) {
            // as much of the remote entries' state in shared memory as lets
            // the wave's CTAs be resident together
            W.mixed = false;
            W.smem = CGCG_SMEM_MAX + 1;
            for (int form = 0; form < 3 && !fits(W.fn, W.smem); ++form) {
                const CgcgLayout lay(H.hmax + 1, H.rmost, H.lcsb, form < 2 ? CGCG_SMEM_MAX : 0, form > 0);
                W.rg = lay.rg;
                W.fn = lay.rg ? fn_cgcg_batch256<true>(p.rmax) : fn_cgcg_batch256<false>(p.rmax);
                W.smem = lay.bytes;
                W.lcs_off = static_cast<int>(lay.lcs);
                W.rs_off = static_cast<int>(lay.rs);
            }
            if (!fits(W.fn, W.smem)) {
                if (why) *why = "a wave does not fit co-resident at this tiling";
                return false;
            }
        }
        else {
            if (why) *why = "a wave does not fit co-resident at this tiling";
            return false;
        }
    }
    free_waves();
    mixed_any = false;
    CUDA_OK(cudaMemcpy(d_lcol, lcol.data(), lcol.size() * sizeof(unsigned short), cudaMemcpyHostToDevice));
    CUDA_OK(cudaMemcpy(d_own, own.data(), own.size() * sizeof(int), cudaMemcpyHostToDevice));
    for (size_t w = 0; w < hw.size(); ++w) {
        const HostWave& H = hw[w];
        Wave& W = nw[w];
        W.d_cta_inst = dalloc<int>(H.cta_inst.size());
        W.d_inst = dalloc<PcgInst>(H.inst.size());
        W.d_hptr = dalloc<int>(H.hptr.size());
        W.d_hidx = dalloc<int>(H.hidx.size());
        CUDA_OK(cudaMemcpy(W.d_cta_inst, H.cta_inst.data(), H.cta_inst.size() * sizeof(int), cudaMemcpyHostToDevice));
        CUDA_OK(cudaMemcpy(W.d_inst, H.inst.data(), H.inst.size() * sizeof(PcgInst), cudaMemcpyHostToDevice));
        CUDA_OK(cudaMemcpy(W.d_hptr, H.hptr.data(), H.hptr.size() * sizeof(int), cudaMemcpyHostToDevice));
        if (!H.hidx.empty()) CUDA_OK(cudaMemcpy(W.d_hidx, H.hidx.data(), H.hidx.size() * sizeof(int), cudaMemcpyHostToDevice));
        W.d_rptr = dalloc<int>(H.rptr.size());
        W.d_rem = dalloc<int2>(H.rem.size());
        CUDA_OK(cudaMemcpy(W.d_rptr, H.rptr.data(), H.rptr.size() * sizeof(int), cudaMemcpyHostToDevice));
        if (!H.rem.empty()) CUDA_OK(cudaMemcpy(W.d_rem, H.rem.data(), H.rem.size() * sizeof(int2), cudaMemcpyHostToDevice));
        W.dev = base;
        W.dev.nblocks = W.G;
        W.dev.cta_inst = W.d_cta_inst;
        W.dev.inst = W.d_inst;
        W.dev.halo_ptr = W.d_hptr;
        W.dev.halo_idx = W.d_hidx;
        W.dev.halo_max = H.hmax;
        W.dev.rem_ptr = W.d_rptr;
        W.dev.rem = W.d_rem;
        W.dev.rem_max = H.rmost;
        W.dev.tm_w = W.tm_w; W.dev.pds_off = W.pds_off; W.dev.xs_off = W.xs_off;
        if (!W.mixed) {
            W.dev.halo_max = H.hmax + 1;   // the spare place
            W.dev.lcs_off = W.lcs_off;
            W.dev.rs_off = W.rs_off;
        }
        if (W.rg) {
            const std::vector<RemoteState> st = remote_states(H.rem);
            W.d_rem_state = dalloc<RemoteState>(st.size());
            W.d_rem_rs = dalloc<double>(W.rs_off ? 0 : 2 * st.size());
            if (!st.empty()) CUDA_OK(cudaMemcpy(W.d_rem_state, st.data(), st.size() * sizeof(RemoteState), cudaMemcpyHostToDevice));
            W.dev.rem_state = W.d_rem_state;
            W.dev.rem_rs = W.d_rem_rs;
        }
        W.dev.slot_max = static_cast<int>(H.smax);
        mixed_any = mixed_any || W.mixed;
    }
    waves = std::move(nw);
    current = p;
    return true;
}

void PcgBatch::release()
{
    free_waves();
    for (long long* p : d_cptr) cudaFree(p);
    for (int* p : d_cent) cudaFree(p);
    d_cptr.clear();
    d_cent.clear();
    void* ptrs[] = {d_slice_off, d_slice_w, d_col, d_row_node, d_lcol, d_val, d_val32, d_r, d_z, d_pA, d_pB, d_q,
                    d_xp, d_bp, d_dp, d_fp, d_f32, d_out, d_own, d_rec, d_xw, d_epoch};
    for (void* p : ptrs) if (p) cudaFree(p);
    d_own = nullptr; d_rec = d_xw = nullptr; d_epoch = nullptr;
    d_slice_off = nullptr; d_slice_w = d_col = d_row_node = nullptr; d_lcol = nullptr; d_val = nullptr;
    d_val32 = nullptr; d_r = d_z = d_pA = d_pB = d_q = nullptr; d_xp = d_bp = d_dp = nullptr; d_fp = nullptr;
    d_f32 = nullptr; d_out = nullptr;
}

void PcgBatch::prepare(int k, const DevState& S, cudaStream_t st)
{
    const size_t kk = static_cast<size_t>(k);
    const int T = 256;
    if (nslot[kk])
        k_ell_from_state<<<static_cast<unsigned>((nslot[kk] + T - 1) / T), T, 0, st>>>(
            S, d_cptr[kk], d_cent[kk], d_val + slot0[kk], d_val32 ? d_val32 + slot0[kk] : nullptr, nslot[kk]);
    PcgDev D = base;
    D.nflag = mem[kk].d_nflag;
    D.pfix = mem[kk].d_pfix;
    D.pres = S.pres; D.rhs1 = S.rhs1; D.pdiag = S.pdiag;
    const int p0 = slice0[kk] * 32, np = nsl[kk] * 32;
    D.N = np;
    D.row_node = d_row_node + p0;
    k_impose_perm_in<<<(np + T - 1) / T, T, 0, st>>>(D, d_xp + p0, d_bp + p0, d_dp + p0, d_fp + p0);
}

void PcgBatch::solve(cudaStream_t st)
{
    CUDA_OK(cudaMemsetAsync(d_out, 0, mem.size() * sizeof(CgOut), st));
    for (Wave& W : waves) {
        void* args[] = {&W.dev};
        CUDA_OK(cudaLaunchCooperativeKernel(W.fn, dim3(static_cast<unsigned>(W.G)), dim3(static_cast<unsigned>(W.threads)), args, W.smem, st));
    }
}

void PcgBatch::finish(int k, double* pres, cudaStream_t st)
{
    const size_t kk = static_cast<size_t>(k);
    const int T = 256;
    const int p0 = slice0[kk] * 32, np = nsl[kk] * 32;
    PcgDev D = base;
    D.N = np;
    D.row_node = d_row_node + p0;
    k_perm_out<<<(np + T - 1) / T, T, 0, st>>>(D, d_xp + p0, pres);
}

}  // namespace cbs3d

extern "C" cbs3d_status cbs3d_probe_halo_placement(int nh, int nslices, const long long* slice_off, const int* slice_w,
                                                   const unsigned short* lc, int* pos, long long* wavefronts)
{
    try {
        if (nh < 1 || nh > 65535 || nslices < 1 || !slice_off || !slice_w || !lc || !pos || !wavefronts)
            return CBS3D_INVALID_INPUT;
        if (slice_off[0] != 0) return CBS3D_INVALID_INPUT;
        for (int q = 0; q < nslices; ++q)
            if (slice_w[q] < 0 || slice_off[q + 1] - slice_off[q] != 32LL * slice_w[q]) return CBS3D_INVALID_INPUT;
        for (long long t = 0; t < slice_off[nslices]; ++t)
            if (lc[t] >= nh) return CBS3D_INVALID_INPUT;
        std::vector<int> id(static_cast<size_t>(nh)), pv;
        for (int e = 0; e < nh; ++e) id[static_cast<size_t>(e)] = e;
        wavefronts[0] = cbs3d::gather_wavefronts(lc, slice_off, slice_w, 0, nslices, 0, id);
        cbs3d::bank_spread_halo(nh, lc, slice_off, slice_w, 0, nslices, 0, pv);
        wavefronts[1] = cbs3d::gather_wavefronts(lc, slice_off, slice_w, 0, nslices, 0, pv);
        for (int e = 0; e < nh; ++e) pos[e] = pv[static_cast<size_t>(e)];
        return CBS3D_OK;
    } catch (...) {
        return CBS3D_INTERNAL;
    }
}
