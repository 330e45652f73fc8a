// Resident state of the fused step, shared by the FP64 (step.cu) and the mixed-precision (mixed.cu)
// translation units.
#pragma once
#include <vector>

#include "fluid.cuh"
#include "sources.cuh"

namespace mhd
{
// Kernel classes of the step, timed with CUDA events on the handle's stream when profiling is on.  "cfl" keeps its place in
// the list that callers read, but the CFL step is part of the prepare pass and no launch has that class.
enum StepKernel { KP_PREPARE = 0, KP_CFL, KP_GRAD, KP_FLUX, KP_UPDATE, KP_FACE_CAND, KP_EDGE_EMF, KP_CT, KP_GYRATE, KP_COUNT };
static const char *const kStepKernelNames[KP_COUNT] = {"prepare", "cfl",            "limited_gradients", "face_flux", "update",
                                                        "face_candidate", "edge_emf", "ct",                "gyrate"};

using Profiler = EventProfiler<KP_COUNT>;

// Single-precision tables of the mixed path, derived once from the FP64 mesh (tetrahedral meshes):
// structure of arrays over cells / faces / edges so that every warp load is coalesced.
struct MixedTables
{
    DBuf<float> K;              // stencil: dl_j = sum_k K_jk (w_k - w_c), K_jk = dx_j^T I wd_k, [16][nc]
    DBuf<float> recon;          // cell field from face fluxes: B_c = sum_j recon[j] Phi_{f_j}, [12][nc]
    DBuf<float4> fn;            // per face: canonical unit normal, |A|
    DBuf<int4> fe;              // per (triangular) face: its 3 edges, negative-sign bits 0-2 and active bit 3
    DBuf<float4> eth;           // per edge: unit tangent, length
    DBuf<int8_t> emode;         // per edge: 0 UCT, 1 zero (wall edge, not owned, no fluid cell, no face), 2 inflow
    // per e2f entry, in the orthonormal basis (e1, e2) of the plane normal to the edge that edge_basis builds
    // from the single-precision tangent: the in-face unit direction m away from the edge and the face's unit
    // normal n, (m.e1, m.e2, n.e1, n.e2); and (sigma = t.(m x n), w_ef)
    DBuf<float4> emn;
    DBuf<float2> esw;
    DBuf<float> vol_inv;        // per cell: 1 / V
};
} // namespace mhd

struct MhdState
{
    std::atomic<int> refs{1};
    mhd::Hold<MhdMesh> hold; // first: released last
    MhdMesh *mesh = nullptr;
    MhdStepParams prm{};
    mhd::FluidParams fp{};
    int nsp = 0, group = 0;
    bool mixed = false;
    mhd::DBuf<double> fv; // FP64 state on a mesh of one cell kind, if memory allows: face values (launch_face_values); others keep grad
    mhd::DBuf<double> U0, U1, W, grad, F, phi0, phi1, phi_add, badd, bind, btot, up, Ef, E, mass, stage;
    mhd::SrcParams src;     // two-ion J x B force and gyration (off unless params.lorentz)
    mhd::DBuf<double> J;    // cell current of the induced field (3 per cell) when the J x B force is on
    mhd::DBuf<double> dpe;  // grad p_e (3 per cell) when the ambipolar terms are on
    mhd::DBuf<double> pn;   // nodal p_e of the ambipolar EMF
    mhd::DBuf<int8_t> pok;  // the node has fluid cells
    mhd::DBuf<double> photo, vst; // source fields of the chemistry terms (empty: absent)
    mhd::DBuf<double> ne_eff, E_impl; // semi-implicit step: n_e,eff per cell, the implicit EMF per edge
    mhd::DBuf<int8_t> dir_inflow;     // semi-implicit step: the Dirichlet (inflow) edges of the solve
    mhd::DBuf<float4> g32;  // mixed precision: face terms A_f x b_f of the cell current (per face)
    mhd::DBuf<float4> d32;  // mixed precision: face terms (p_R - p_L) A_f / 2 of grad p_e (per face)
    mhd::DBuf<int32_t> wall_slot; // the caller's Dirichlet wall states: slot per face (-1: ghost_state)
    mhd::DBuf<double> wall_prim;  // [species][slot][5]
    mhd::DBuf<double> mres; // explicit resistive EMF: m_e = eta_e / star1_e per edge (empty: off)
    int8_t *floor_flags = nullptr; // when set, the update records the floors it applied ([s*nc + c])
    uint32_t *sw_edge = nullptr;   // switch log of the edge EMF (null: off), with fp.sw_lim, sw_flux, sw_floor
    uint32_t *sw_face = nullptr;   // switch log of the face EMF candidates' a_f (null: off)
    mhd::DBuf<double> efgeo;       // FP64 state: the UCT's per-(edge, slot) face geometry (build_edge_face_geo), or empty
    mhd::DBuf<double> pa;          // with efgeo: the stage's phi_ind / |A| per face, left by the face-candidate pass
    mhd::DBuf<double> scal; // [0] dt
    mhd::DBuf<unsigned long long> dt_bits;
    mhd::DBuf<int> flag;
    mhd::DBuf<unsigned> cfl_count; // finished blocks of the CFL pass
    // mixed precision: FP32 bulk arrays (the state U and the face fluxes Phi stay FP64)
    mhd::MixedTables mt;
    mhd::DBuf<float> W32, grad32, F32, E32;
    mhd::DBuf<float4> Ef32; // per face: EMF candidate E_f (3) and Phi_ind / |A|
    mhd::DBuf<float4> up32, bt32, bi32, badd32;
    double *pinned = nullptr;
    int64_t launches = 0; // kernels launched by the step since creation
    mhd::Profiler prof;
    ~MhdState()
    {
        if (pinned) cudaFreeHost(pinned);
    }
};

namespace mhd
{
// Where the CFL step's minimum over the cells goes: the running minimum (bits of a positive double) and the invalid flag
// of this step, the count of finished blocks (all three re-armed by the last block), the step size on the device, and the
// step size and the flag in the pinned host buffer, so that the host reads them after a synchronisation without a copy.
struct CflOut
{
    unsigned long long *bits;
    int *flag;
    unsigned *count;
    double *dt, *host;
    double dt_max;
};
inline CflOut cfl_out(const MhdState *st, double dt_max)
{
    return CflOut{st->dt_bits.p, st->flag.p, st->cfl_count.p, st->scal.p, st->pinned, dt_max};
}
#ifdef __CUDACC__
// gdt = min(gdt, dt_max); invalid unless finite and positive (Solver.cpp:233-236)
__device__ __forceinline__ void cfl_finish(const CflOut &o, double g, int invalid)
{
    g = (o.dt_max < g) ? o.dt_max : g;
    if (!isfinite(g) || g <= 0) invalid |= 1;
    *o.dt = g;
    o.host[0] = g;
    reinterpret_cast<int *>(o.host + 1)[0] = invalid;
}
// Block minimum of v (min is exact, so the order of the reduction does not matter), one atomic per block; the grid's last
// block finishes the step size.  bad: a thread met a step that is zero, negative or NaN (the reference's "invalid time
// step").  Every thread of the block calls it.
__device__ __forceinline__ void cfl_reduce(const CflOut &o, double v, bool bad)
{
    constexpr double inf = 1.0 / 0.0;
    __shared__ double sh[32];
    __shared__ bool last;
    for (int k = 16; k > 0; k >>= 1)
    {
        const double u = __shfl_xor_sync(0xffffffffu, v, k);
        v = (u < v) ? u : v;
    }
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    const int any = __syncthreads_or(bad);
    if (threadIdx.x == 0)
    {
        for (unsigned w = 1; w < (blockDim.x >> 5); ++w) v = (sh[w] < v) ? sh[w] : v;
        if (any) atomicOr(o.flag, 1);
        if (v < inf) atomicMin(o.bits, static_cast<unsigned long long>(__double_as_longlong(v)));
        __threadfence();
        last = atomicAdd(o.count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || threadIdx.x != 0) return;
    __threadfence();
    const unsigned long long b = atomicExch(o.bits, static_cast<unsigned long long>(__double_as_longlong(inf)));
    cfl_finish(o, __longlong_as_double(static_cast<long long>(b)), atomicExch(o.flag, 0));
    *o.count = 0;
}
#endif

// A stage's two chains after the prepare pass: the fluid's (face values, fluxes, update) on the mesh's stream and the EMF's
// (cell current, face candidates, edge EMF, CT) on the mesh's side stream.  They share their inputs and meet twice: the
// update reads what the EMF chain's first passes leave, and the stage ends when both have.  A pass of a small mesh is a few
// waves of blocks whose last one leaves most SMs idle, and its launch costs as much as its work: there the other chain's
// blocks fill the gaps.  A pass that saturates DRAM gains nothing and loses nothing.  Per step, one stream -> two:
// mixed 24k cells 46 -> 41 us, 221k 251 -> 205 us, 14.2M 10.94 -> 10.96 ms; FP64 24k 81 -> 75 us, 1.8M 3.25 -> 3.22 ms.
// So every size takes two streams, except while the passes are timed one by one by the profiler.
struct StageFork
{
    MhdMesh *m;
    cudaStream_t main, emf;
    bool on;
    StageFork(MhdState *s, bool fork) : m(s->mesh), main(s->mesh->stream), emf(s->mesh->stream), on(fork && !s->prof.on)
    {
        if (!on) return;
        emf = m->side;
        MHD_CUDA(cudaEventRecord(m->ev_prep, main));
        MHD_CUDA(cudaStreamWaitEvent(emf, m->ev_prep, 0));
    }
    void faces_done() // what the update reads has been enqueued on emf
    {
        if (on) MHD_CUDA(cudaEventRecord(m->ev_face, emf));
    }
    void before_update()
    {
        if (on) MHD_CUDA(cudaStreamWaitEvent(main, m->ev_face, 0));
    }
    void join()
    {
        if (!on) return;
        MHD_CUDA(cudaEventRecord(m->ev_ct, emf));
        MHD_CUDA(cudaStreamWaitEvent(main, m->ev_ct, 0));
        on = false;
    }
    ~StageFork() // an exception between: the side stream still rejoins
    {
        if (on && cudaEventRecord(m->ev_ct, emf) == cudaSuccess) cudaStreamWaitEvent(main, m->ev_ct, 0);
    }
};
void mixed_setup(MhdState *st);
// one FP64 stage (Us, phis) -> (Uo, phio) at the step size in st->scal[0]; stage2 averages with Uo, phio in place
void fp64_stage(MhdState *st, const double *Us, const double *phis, double *Uo, double *phio, bool stage2);
// gyrate_close: stage 2 applies the closing half-step gyration in its update (two-ion sources on)
void mixed_stage(MhdState *st, const double *Us, const double *phis, double *Uo, double *phio, bool stage2, bool cfl, double dt_max,
                 bool prepared = false, bool gyrate_close = false);
// the opening half-step gyration of U0, renewing its primitives and u+ (stage 1 then runs prepared)
void mixed_gyrate_open(MhdState *st);
void mixed_badd(MhdState *st);
// primitives, cell fields (and with cfl the device CFL step) of (Us, phis) in mixed precision
// turned: the opening gyration follows and writes the primitives and u+ of the owned fluid cells
void mixed_prepare(MhdState *st, const double *Us, const double *phis, bool cfl, double dt_max, bool turned);
// the CFL step of a mesh without cells: dt_max
void cfl_empty(MhdState *st, double dt_max);
} // namespace mhd
