// nvcc-flags: -fmad=false
// Fluid right-hand side on the device: primitives, limited least-squares gradients, Rusanov
// face fluxes, and the deterministic (atomic-free) gather of face fluxes into cells.
// FP64, reference-exact: every expression keeps the reference's operation order and this file
// is compiled without multiply-add contraction, so results round exactly as the host code does.
#include "kernels.cuh"

namespace mhd
{
// mhd::to_prim over n cells
__global__ void k_to_prim(SField<const double> U, SField<double> W, int32_t n, int nsp, double gamma, double rho_floor, double p_floor)
{
    const int32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    for (int s = 0; s < nsp; ++s)
    {
        const Prim5 w = to_prim(U(s, c, 0), U(s, c, 1), U(s, c, 2), U(s, c, 3), U(s, c, 4), gamma, rho_floor, p_floor);
        W(s, c, 0) = w.rho; W(s, c, 1) = w.u; W(s, c, 2) = w.v; W(s, c, 3) = w.w; W(s, c, 4) = w.p;
    }
}

// One component of mhd::ghost_state (Common/fluid/Reconstruction.cpp:9-24); (cu, cv, cw) the velocity
// of the inside state, wc its component q.
__device__ __forceinline__ double ghost_component(int kind, bool absorb, int q, double wc, double cu, double cv, double cw, V3 n,
                                                  const Prim5 &fs)
{
    if (kind == 1)
    {
        if (absorb) return (q == 0 || q == 4) ? 1e-12 : 0.0;
        if (q == 0 || q == 4) return wc;
        const double un = cu * n.x + cv * n.y + cw * n.z;
        const double nq = q == 1 ? n.x : (q == 2 ? n.y : n.z);
        return wc - 2 * un * nq;
    }
    if (kind == 2) return q == 0 ? fs.rho : q == 1 ? fs.u : q == 2 ? fs.v : q == 3 ? fs.w : fs.p;
    return wc;
}

// The Barth-Jespersen psi (with the relative limiter's rel >= 0 on top, 0: off): min over the faces of (hi - w)/dl
// (dl > 0) and (lo - w)/dl (dl < 0).  A correctly rounded quotient is monotone, so the minimum sits at the largest dl
// (dpos) and the most negative one (dneg), and of those two the smaller one can be told from the products: p1 < p2
// means n1/dpos < n2/dneg exactly, so only that quotient is formed (both where the products tie).  Quotients of at
// least 1 leave psi = 1, and a zero numerator (the cell is its neighbourhood's extreme, about one cell and variable
// in three) gives 0 without entering the divider's slow path.  The result is the reference's, bit for bit.
__device__ __forceinline__ double limiter_psi(double wc, double lo, double hi, double dpos, double dneg, double rel)
{
    double psi = 1.0;
    const double n1 = hi - wc, n2 = lo - wc;
    const bool c1 = dpos > 1e-300 && n1 < dpos, c2 = dneg < -1e-300 && n2 > dneg;
    if (c1 || c2)
    {
        bool first = c1;
        if (c1 && c2)
        {
            const double p1 = n1 * -dneg, p2 = -n2 * dpos;
            first = p1 < p2;
            if (p1 == p2 && n2 != 0) psi = dmin(psi, n1 / dpos);
        }
        const double num = first ? n1 : n2, den = first ? dpos : dneg;
        psi = num == 0 ? 0.0 : dmin(psi, num / den);
    }
    if (rel > 0)
    {
        const double a = dmax(dpos, -dneg);
        if (a > 1e-300) psi = dmin(psi, rel * wc / a);
    }
    return psi;
}

// mhd::Stencil::limited_gradients (Common/fluid/Reconstruction.cpp:80-142): least-squares gradient
// from the precomputed w*d and the symmetric inverse, Barth-Jespersen psi over all faces of the cell,
// optional relative limiter on rho and p, clamp to [0, 1]; zero for cells without a valid stencil.
// One thread per (cell, primitive variable): blockDim = (32, 5), warp q of a block handles variable
// q of 32 consecutive cells.  Each variable's fit and limiter are independent of the others (wall
// ghosts only read the velocity), so the per-thread state is small, occupancy high, and the five
// warps share the cell's geometry through L1.  The reference's arithmetic order is kept per variable.
__global__ void __launch_bounds__(160) k_limited_gradients_v(MeshView m, FluidParams p, SField<const double> W, SField<double> G)
{
    const int32_t c = blockIdx.x * 32 + threadIdx.x;
    const int q = threadIdx.y;
    if (c >= m.nc) return;
    if (c >= m.no_cells || !m.st_valid[c])
    {
        for (int s = 0; s < p.nsp; ++s)
            for (int a = 0; a < 3; ++a) G(s, c, 3 * q + a) = 0.0;
        return;
    }
    const int32_t k0 = m.c2f_ptr[c], k1 = m.c2f_ptr[c + 1];
    const V3 xc = ld3(m.cell_center, c);
    const double *Ip = m.st_inv + 6 * (int64_t)c;
    const double I00 = Ip[0], I01 = Ip[1], I02 = Ip[2], I11 = Ip[3], I12 = Ip[4], I22 = Ip[5];
    for (int s = 0; s < p.nsp; ++s)
    {
        const double wc = W(s, c, q);
        double lo = wc, hi = wc, r0 = 0, r1 = 0, r2 = 0;
        for (int32_t k = k0; k < k1; ++k)
        {
            const int32_t nb = m.st_nb[k];
            if (nb == INT32_MIN) continue;
            double wn;
            if (nb >= 0) wn = W(s, nb, q);
            else
            {
                const int32_t f = -(nb + 1);
                const int kind = m.face_kind[f];
                const V3 n = (double(m.c2f_sgn[k]) / m.face_area_mag[f]) * ld3(m.face_area, f);
                const bool vel = kind == 1 && !p.absorb[s] && q >= 1 && q <= 3;
                const double *wg = wall_ghost(p, kind, f, s);
                wn = wg ? wg[q]
                        : ghost_component(kind, p.absorb[s] != 0, q, wc, vel ? W(s, c, 1) : 0.0, vel ? W(s, c, 2) : 0.0,
                                          vel ? W(s, c, 3) : 0.0, n, p.fs[s]);
            }
            const double dq = wn - wc;
            r0 += m.st_wd[3 * (int64_t)k] * dq;
            r1 += m.st_wd[3 * (int64_t)k + 1] * dq;
            r2 += m.st_wd[3 * (int64_t)k + 2] * dq;
            lo = dmin(lo, wn);
            hi = dmax(hi, wn);
        }
        const double g0 = I00 * r0 + I01 * r1 + I02 * r2;
        const double g1 = I01 * r0 + I11 * r1 + I12 * r2;
        const double g2 = I02 * r0 + I12 * r1 + I22 * r2;
        double psi = 1.0;
        if (p.limit)
        {
            double dpos = 0, dneg = 0;
            for (int32_t k = k0; k < k1; ++k)
            {
                const V3 dx = ld3(m.face_center, m.c2f_idx[k]) - xc;
                const double dl = g0 * dx.x + g1 * dx.y + g2 * dx.z;
                if (dl > dpos) dpos = dl;
                if (dl < dneg) dneg = dl;
            }
            psi = limiter_psi(wc, lo, hi, dpos, dneg, p.rel_limit > 0 && (q == 0 || q == 4) ? p.rel_limit : 0.0);
        }
        const double ps = dmax(0.0, dmin(1.0, psi));
        G(s, c, 3 * q) = ps * g0;
        G(s, c, 3 * q + 1) = ps * g1;
        G(s, c, 3 * q + 2) = ps * g2;
    }
}

// The same limited gradients on a mesh whose cells all have NF faces (4: tetrahedra, 6: hexahedra).  blockDim = (32, 5):
// warp q of a block handles variable q of 32 consecutive cells for NS species.  The cells' stencil rows (6 NF + 6 doubles
// per cell, structure of arrays) are copied to shared memory asynchronously, once for the ten (variable, species) pairs,
// while the neighbour ids and then the neighbour values are gathered: two memory latencies in series instead of three,
// and a thread's registers hold one variable's chain.  Per variable the arithmetic and its order are those of the
// reference (slots and faces in c2f order).
// GRAD: the limited gradients G.  FACE: the limited values at the cell's NF faces (the face_state of FluxRHS.cpp:16-27
// with its positivity fallback, which the density and pressure warps tell the others through shared memory),
// FV[(s*5 + q)*NF*nc + NF*c + j]: the flux pass gathers 5 values per side from them instead of 5 + 15 and two centres,
// and a cell forms each of its face states once.
// SI: the stride of W's cells (1: species-major state, 5: the reference's layout).
// Bound by the FP64 pipe and shared-memory reads (56% of the issue slots, 66% of the L1 throughput): 1.77M tetrahedra, two
// species: 355 us a launch, 470 as one thread per (cell, species) with the stencil in 128 registers; without the staging
// 483; 5 or 7 blocks per SM 381 and 372.  295k hexahedra: 115 us, 226 with one CSR loop per variable.
template <int NF, int NS, int SI, bool LOG, bool GRAD, bool FACE>
__global__ void __launch_bounds__(160, NF == 4 ? 6 : 5) k_limited_slots(MeshView m, FluidParams p, SField<const double> W,
                                                                              SField<double> G, double *__restrict__ FV)
{
    pdl_begin();
    constexpr int ROWS = 6 * NF + 6; // w d (3 per slot), dx (3 per slot), inverse (6)
    __shared__ double geo[ROWS][32];
    __shared__ uint32_t pos[2][NS][NF]; // per face slot the cells whose density (0) / pressure (1) there is positive
    const int lane = threadIdx.x, q = threadIdx.y;
    const int32_t c = blockIdx.x * 32 + lane;
    const int64_t n = m.nc;
    const bool in = c < m.nc, live = in && c < m.no_cells && m.st_valid[c];
    if (in)
#pragma unroll
        for (int r = 0; r < ROWS; r += 5)
            if (r + q < ROWS) cp_async8(&geo[r + q][lane], m.t_wd + (r + q) * n + c);
    cp_async_commit();
    double v[NS][NF], fv[NS][NF], wc[NS];
    if (live)
    {
        int32_t nb[NF];
        bool bnd = false;
#pragma unroll
        for (int j = 0; j < NF; ++j)
        {
            nb[j] = m.t_nb[j * n + c];
            bnd |= nb[j] < 0;
        }
#pragma unroll
        for (int s = 0; s < NS; ++s)
        {
            const double *w = W.p + s * W.ss + q * W.sm;
            wc[s] = w[SI * (int64_t)c];
#pragma unroll
            for (int j = 0; j < NF; ++j) v[s][j] = nb[j] >= 0 ? w[SI * (int64_t)nb[j]] : wc[s]; // skipped: enters no sum, no bound
        }
        if (bnd)
#pragma unroll
            for (int j = 0; j < NF; ++j)
            {
                if (nb[j] >= 0 || nb[j] == INT32_MIN) continue;
                const int32_t f = -(nb[j] + 1);
                const int kind = m.face_kind[f];
                const double sg = m.t_sg[j * n + c];
                const D4 fn = ld_d4(m.fna + 4 * (int64_t)f);
#pragma unroll
                for (int s = 0; s < NS; ++s)
                {
                    const bool vel = kind == 1 && !p.absorb[s] && q >= 1 && q <= 3;
                    const double *wg = wall_ghost(p, kind, f, s);
                    v[s][j] = wg ? wg[q]
                                 : ghost_component(kind, p.absorb[s] != 0, q, wc[s], vel ? W(s, c, 1) : 0.0, vel ? W(s, c, 2) : 0.0,
                                                   vel ? W(s, c, 3) : 0.0, mk(sg * fn.x, sg * fn.y, sg * fn.z), p.fs[s]);
                }
            }
    }
    cp_async_wait<0>();
    __syncthreads();
    if (live)
    {
        double r[NS][3], lo[NS], hi[NS];
        int jlo[NS], jhi[NS]; // switch log: the slots of the extremes
#pragma unroll
        for (int s = 0; s < NS; ++s)
        {
            r[s][0] = r[s][1] = r[s][2] = 0;
            lo[s] = hi[s] = wc[s];
            jlo[s] = jhi[s] = 7;
        }
#pragma unroll
        for (int j = 0; j < NF; ++j)
        {
            const double w0 = geo[3 * j][lane], w1 = geo[3 * j + 1][lane], w2 = geo[3 * j + 2][lane];
#pragma unroll
            for (int s = 0; s < NS; ++s)
            {
                const double dq = v[s][j] - wc[s];
                r[s][0] += w0 * dq;
                r[s][1] += w1 * dq;
                r[s][2] += w2 * dq;
                if (LOG && v[s][j] < lo[s]) jlo[s] = j;
                if (LOG && hi[s] < v[s][j]) jhi[s] = j;
                lo[s] = dmin(lo[s], v[s][j]);
                hi[s] = dmax(hi[s], v[s][j]);
            }
        }
        const double(*I)[32] = geo + 6 * NF;
        const double I00 = I[0][lane], I01 = I[1][lane], I02 = I[2][lane], I11 = I[3][lane], I12 = I[4][lane], I22 = I[5][lane];
        const double(*dx)[32] = geo + 3 * NF;
        double g[NS][3], dpos[NS], dneg[NS];
        int jpos[NS], jneg[NS];
#pragma unroll
        for (int s = 0; s < NS; ++s)
        {
            g[s][0] = I00 * r[s][0] + I01 * r[s][1] + I02 * r[s][2];
            g[s][1] = I01 * r[s][0] + I11 * r[s][1] + I12 * r[s][2];
            g[s][2] = I02 * r[s][0] + I12 * r[s][1] + I22 * r[s][2];
            dpos[s] = dneg[s] = 0;
            jpos[s] = jneg[s] = 7;
        }
#pragma unroll
        for (int j = 0; j < NF; ++j)
        {
            const double x = dx[3 * j][lane], y = dx[3 * j + 1][lane], z = dx[3 * j + 2][lane];
#pragma unroll
            for (int s = 0; s < NS; ++s)
            {
                const double dl = g[s][0] * x + g[s][1] * y + g[s][2] * z;
                if (LOG && dl > dpos[s]) jpos[s] = j;
                if (LOG && dl < dneg[s]) jneg[s] = j;
                if (dl > dpos[s]) dpos[s] = dl;
                if (dl < dneg[s]) dneg[s] = dl;
            }
        }
#pragma unroll
        for (int s = 0; s < NS; ++s)
        {
            double psi = 1.0;
            if (p.limit)
            {
                const bool rel_on = p.rel_limit > 0 && (q == 0 || q == 4);
                psi = limiter_psi(wc[s], lo[s], hi[s], dpos[s], dneg[s], rel_on ? p.rel_limit : 0.0);
                if (LOG)
                    sw_log(p.sw_lim, (s * 5 + q) * n + c,
                           limiter_code(psi, wc[s], lo[s], hi[s], dpos[s], dneg[s], jlo[s], jhi[s], jpos[s], jneg[s], p.rel_limit, rel_on));
            }
            const double ps = dmax(0.0, dmin(1.0, psi));
#pragma unroll
            for (int a = 0; a < 3; ++a) g[s][a] = ps * g[s][a];
            if (GRAD)
                for (int a = 0; a < 3; ++a) G(s, c, 3 * q + a) = g[s][a];
        }
        if (FACE)
#pragma unroll
            for (int j = 0; j < NF; ++j)
            {
                const double x = dx[3 * j][lane], y = dx[3 * j + 1][lane], z = dx[3 * j + 2][lane];
#pragma unroll
                for (int s = 0; s < NS; ++s) fv[s][j] = wc[s] + g[s][0] * x + g[s][1] * y + g[s][2] * z;
            }
    }
    else if (in)
    {
        // zero gradient: every face value is the cell value
#pragma unroll
        for (int s = 0; s < NS; ++s)
        {
            if (GRAD)
                for (int a = 0; a < 3; ++a) G(s, c, 3 * q + a) = 0.0;
            wc[s] = FACE ? W(s, c, q) : 0.0;
#pragma unroll
            for (int j = 0; j < NF; ++j) fv[s][j] = wc[s];
        }
    }
    if constexpr (FACE)
    {
        // density and pressure decide: a face where either is not positive takes the cell state
        if (q == 0 || q == 4)
#pragma unroll
            for (int s = 0; s < NS; ++s)
#pragma unroll
                for (int j = 0; j < NF; ++j)
                {
                    const uint32_t b = __ballot_sync(0xffffffffu, in && fv[s][j] > 0);
                    if (lane == 0) pos[q >> 2][s][j] = b;
                }
        __syncthreads();
        if (!in) return;
#pragma unroll
        for (int s = 0; s < NS; ++s)
        {
#pragma unroll
            for (int j = 0; j < NF; ++j)
                if (!((pos[0][s][j] & pos[1][s][j]) >> lane & 1u)) fv[s][j] = wc[s];
            double *o = FV + ((s * 5 + q) * n + c) * NF;
            if constexpr (NF == 4) st_d4(o, fv[s][0], fv[s][1], fv[s][2], fv[s][3]);
            else
#pragma unroll
                for (int j = 0; j < NF; j += 2) *reinterpret_cast<double2 *>(o + j) = make_double2(fv[s][j], fv[s][j + 1]);
        }
    }
}

// the instances of one launch: species in pairs (the last one alone for an odd count)
template <int NF, bool LOG, bool GRAD, bool FACE>
void launch_slots(const MeshView &m, FluidParams p, SField<const double> W, SField<double> G, double *FV, cudaStream_t s)
{
    const dim3 block(32, 5);
    const int grid = grid_for(m.nc, 32), nsp = p.nsp;
    for (int s0 = 0; s0 < nsp; s0 += 2)
    {
        const bool pair = nsp - s0 > 1;
        if (W.si == 1)
            launch_pdl(pair ? k_limited_slots<NF, 2, 1, LOG, GRAD, FACE> : k_limited_slots<NF, 1, 1, LOG, GRAD, FACE>, grid, block, 0, s, m, p,
                       W, G, FV);
        else if constexpr (!FACE && !LOG) // the reference's layout: one species a call
            launch_pdl(k_limited_slots<NF, 1, 5, false, GRAD, false>, grid, block, 0, s, m, p, W, G, FV);
        // the next pair's species become 0 and 1
        W.p += 2 * W.ss;
        if (GRAD) G.p += 2 * G.ss;
        if (FACE) FV += 10 * (int64_t)NF * m.nc;
        if (p.wall_prim) p.wall_prim += 10 * p.wall_n;
        if (p.sw_lim) p.sw_lim += 10 * (int64_t)m.nc;
        for (int k = 0; k + 2 < kMaxSpecies; ++k)
        {
            p.fs[k] = p.fs[k + 2];
            p.absorb[k] = p.absorb[k + 2];
        }
    }
}

// Face loop of mhd::fluid_flux_rhs (Common/fluid/FluxRHS.cpp:36-69): Rusanov flux of the
// reconstructed face states times |A|, per face and species (SoA: F[(s*5 + m)*nf + f]).
// Faces that the reference skips (Skip kind, no owned fluid cell) get zero.
template <bool LOG>
__global__ void __launch_bounds__(128) k_face_flux(MeshView m, FluidParams p, SField<const double> W, SField<const double> G,
                                                   double *__restrict__ F)
{
    // one species per grid row (blockIdx.y)
    const int32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = blockIdx.y;
    if (f >= m.nf || s >= p.nsp) return;
    const int64_t nf = m.nf;
    const int kind = m.face_kind[f];
    const int32_t p0 = m.f2c_ptr[f], cnt = m.f2c_ptr[f + 1] - p0;
    bool any_owned = false;
    for (int q = 0; q < cnt; ++q)
    {
        const int32_t cc = m.f2c_idx[p0 + q];
        any_owned |= cc < m.no_cells && m.material[cc] == 0;
    }
    if (kind == 4 || !any_owned)
    {
        for (int q = 0; q < 5; ++q) F[(s * 5 + q) * nf + f] = 0.0;
        return;
    }
    const double A = m.face_area_mag[f];
    const V3 n = (1.0 / A) * ld3(m.face_area, f);
    const V3 xf = ld3(m.face_center, f);
    const bool interior = cnt == 2 && kind == 0;
    int32_t cL = -1, cR = -1, c = -1;
    int sgn = 0;
    if (interior)
    {
        cL = m.face_L[f];
        cR = m.face_R[f];
    }
    else
    {
        c = m.f2c_idx[p0];
        sgn = m.f2c_sgn[p0];
        if (cnt == 2 && m.material[c] != 0)
        {
            c = m.f2c_idx[p0 + 1];
            sgn = m.f2c_sgn[p0 + 1];
        }
    }
    {
        Prim5 L, R;
        double g[15];
        uint32_t code = 0; // switch log: the face states' positivity fallbacks (bits 2, 3), Rusanov's choices
        auto state_of = [&](int32_t cc, uint32_t bit) {
            const Prim5 w{W(s, cc, 0), W(s, cc, 1), W(s, cc, 2), W(s, cc, 3), W(s, cc, 4)};
            for (int q = 0; q < 15; ++q) g[q] = G(s, cc, q);
            if (LOG && face_state_fallback(w, g, xf - ld3(m.cell_center, cc))) code |= bit;
            return face_state(w, g, xf - ld3(m.cell_center, cc));
        };
        if (interior)
        {
            L = state_of(cL, 4u);
            R = state_of(cR, 8u);
        }
        else
        {
            const Prim5 in = state_of(c, 4u);
            const double *wg = wall_ghost(p, kind, f, s);
            const Prim5 gh = wg ? Prim5{wg[0], wg[1], wg[2], wg[3], wg[4]} : ghost_state(kind, p.absorb[s] != 0, in, double(sgn) * n, p.fs[s]);
            if (sgn > 0) { L = in; R = gh; }
            else { R = in; L = gh; }
        }
        double Fl[5];
        rusanov(L, R, n, p.gamma, Fl);
        if (LOG)
            sw_log(p.sw_flux, s * nf + f,
                   code | rusanov_code(L, R, n, p.gamma, !interior && kind == 1 && !p.absorb[s] && !wall_ghost(p, kind, f, s)));
        for (int q = 0; q < 5; ++q) F[(s * 5 + q) * nf + f] = Fl[q] * A;
    }
}

// The same face flux from the face values that k_limited_slots<..., FACE> left: one 16-byte and one 32-byte record
// per face, then 5 values per side.  Species in neighbouring blocks, which read the same records.  64% of the DRAM peak
// on 1.77M tetrahedra, two species: 208 us a launch (78 registers: 214) against 482 from the gradients.
__global__ void __launch_bounds__(128, 7) k_face_flux_fv(MeshView m, FluidParams p, int64_t nnz, const double *__restrict__ FV,
                                                      double *__restrict__ F)
{
    pdl_begin();
    const int s = blockIdx.x % p.nsp;
    const int32_t f = (blockIdx.x / p.nsp) * blockDim.x + threadIdx.x;
    if (f >= m.nf) return;
    const int64_t nf = m.nf;
    double *Fo = F + s * 5 * nf + f;
    const int4 r = m.frec[f];
    const int type = r.z & 15;
    if (type == FF_NONE)
    {
        for (int q = 0; q < 5; ++q) Fo[q * nf] = 0.0;
        return;
    }
    const D4 n4 = ld_d4(m.fna + 4 * (int64_t)f);
    const V3 n = mk(n4.x, n4.y, n4.z);
    const double *fv = FV + s * 5 * nnz;
    auto state = [&](int32_t k) { return Prim5{fv[k], fv[nnz + k], fv[2 * nnz + k], fv[3 * nnz + k], fv[4 * nnz + k]}; };
    Prim5 L = state(r.x), R;
    if (type == FF_INTERIOR) R = state(r.y);
    else
    {
        const int kind = r.z >> 4;
        const double sg = type == FF_INSIDE_L ? 1.0 : -1.0;
        const double *wg = wall_ghost(p, kind, f, s);
        R = wg ? Prim5{wg[0], wg[1], wg[2], wg[3], wg[4]} : ghost_state(kind, p.absorb[s] != 0, L, sg * n, p.fs[s]);
        if (type == FF_INSIDE_R)
        {
            const Prim5 t = L;
            L = R;
            R = t;
        }
    }
    double Fl[5];
    rusanov(L, R, n, p.gamma, Fl);
    for (int q = 0; q < 5; ++q) Fo[q * nf] = Fl[q] * n4.w;
}

// Scatter of Common/fluid/FluxRHS.cpp:70-72 as a gather: rhs_c = sum_f -s_cf F_f / V_c over the
// faces of each owned fluid cell, zero elsewhere.  The faces are visited in ascending id, the
// order in which the reference's face loop scatters into the cell, so the sum rounds the same.
__global__ void k_gather_rhs(MeshView m, int nsp, const double *__restrict__ F, SField<double> rhs)
{
    const int32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= m.nc) return;
    const int64_t nf = m.nf;
    if (c >= m.no_cells || m.material[c] != 0)
    {
        for (int s = 0; s < nsp; ++s)
            for (int q = 0; q < 5; ++q) rhs(s, c, q) = 0.0;
        return;
    }
    const double V = m.cell_volume[c];
    const int32_t k0 = m.c2f_ptr[c], k1 = m.c2f_ptr[c + 1];
    for (int s = 0; s < nsp; ++s)
    {
        double r[5] = {0, 0, 0, 0, 0};
        for (int32_t k = k0; k < k1; ++k)
        {
            const int32_t f = m.cfa_idx[k];
            const bool out = m.cfa_sgn[k] > 0;
            for (int q = 0; q < 5; ++q)
            {
                const double v = F[(s * 5 + q) * nf + f] / V;
                r[q] = out ? r[q] - v : r[q] + v;
            }
        }
        for (int q = 0; q < 5; ++q) rhs(s, c, q) = r[q];
    }
}

void launch_limited_gradients(const MeshView &m, const FluidParams &p, SField<const double> W, SField<double> G, cudaStream_t s)
{
    if (!m.nc) return;
    // the switch log is the differentiated run's, which needs tetrahedra
    if (m.faces_per_cell == 4)
        (p.sw_lim && p.limit ? launch_slots<4, true, true, false> : launch_slots<4, false, true, false>)(m, p, W, G, nullptr, s);
    else if (m.faces_per_cell == 6) launch_slots<6, false, true, false>(m, p, W, G, nullptr, s);
    else k_limited_gradients_v<<<grid_for(m.nc, 32), dim3(32, 5), 0, s>>>(m, p, W, G);
    MHD_LAUNCH_CHECK();
}

// the face values of the first-order scheme: every face the cell's value
template <int NF>
__global__ void __launch_bounds__(128) k_cell_face_values(int32_t nc, int nrow, const double *__restrict__ W, double *__restrict__ FV)
{
    pdl_begin();
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; // (species, variable) row and cell
    if (i >= (int64_t)nrow * nc) return;
    const double w = W[i];
    for (int j = 0; j < NF; ++j) FV[i * NF + j] = w;
}

void launch_face_values(const MeshView &m, const FluidParams &p, SField<const double> W, bool second_order, const SField<double> *G,
                        double *FV, cudaStream_t s)
{
    if (!m.nc) return;
    if (!second_order)
    {
        const int64_t rows = 5 * p.nsp;
        launch_pdl(m.faces_per_cell == 4 ? k_cell_face_values<4> : k_cell_face_values<6>, grid_for(rows * m.nc, 128), 128, 0, s, m.nc,
                   static_cast<int>(rows), W.p, FV);
    }
    else if (m.faces_per_cell == 6) launch_slots<6, false, false, true>(m, p, W, SField<double>{}, FV, s);
    else if (G) launch_slots<4, true, true, true>(m, p, W, *G, FV, s);
    else launch_slots<4, false, false, true>(m, p, W, SField<double>{}, FV, s);
    MHD_LAUNCH_CHECK();
}

void launch_face_flux_fv(const MeshView &m, const FluidParams &p, const double *FV, double *F, cudaStream_t s)
{
    if (!m.nf) return;
    launch_pdl(k_face_flux_fv, grid_for(m.nf, 128) * p.nsp, 128, 0, s, m, p, (int64_t)m.faces_per_cell * m.nc, FV, F);
    MHD_LAUNCH_CHECK();
}

void launch_face_flux(const MeshView &m, const FluidParams &p, SField<const double> W, SField<const double> G, double *F, cudaStream_t s)
{
    if (!m.nf) return;
    (p.sw_flux ? k_face_flux<true> : k_face_flux<false>)<<<dim3(grid_for(m.nf, 128), p.nsp), 128, 0, s>>>(m, p, W, G, F);
    MHD_LAUNCH_CHECK();
}

__global__ void k_wall_slots(MeshView m, const int32_t *__restrict__ faces, int32_t n, int32_t *__restrict__ slot, int *__restrict__ err)
{
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t f = faces[i];
    if (f < 0 || f >= m.nf || m.face_kind[f] != 1)
    {
        atomicOr(err, 1);
        return;
    }
    if (atomicCAS(slot + f, -1, i) != -1) atomicOr(err, 2);
}

void build_wall_slots(const MeshView &m, const int32_t *faces, int32_t n, int32_t *slot, cudaStream_t s)
{
    if (m.nf) MHD_CUDA(cudaMemsetAsync(slot, 0xff, (size_t)m.nf * sizeof(int32_t), s));
    if (!n) return;
    DBuf<int> err;
    err.alloc(1);
    MHD_CUDA(cudaMemsetAsync(err.p, 0, sizeof(int), s));
    k_wall_slots<<<grid_for(n, 128), 128, 0, s>>>(m, faces, n, slot, err.p);
    MHD_LAUNCH_CHECK();
    int h = 0;
    MHD_CUDA(cudaMemcpyAsync(&h, err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    MHD_CUDA(cudaStreamSynchronize(s));
    MHD_REQUIRE(!(h & 1), "wall ghost faces must be faces of kind wall");
    MHD_REQUIRE(!(h & 2), "wall ghost faces must be distinct");
}

static FluidParams single_species(int32_t species, const MhdPrim *fs, double gamma, int limit, double rel_limit)
{
    FluidParams p{};
    p.nsp = 1;
    p.limit = limit;
    p.gamma = gamma;
    p.rel_limit = rel_limit;
    if (fs) p.fs[0] = Prim5{fs->rho, fs->u, fs->v, fs->w, fs->p};
    p.absorb[0] = species == 1; // reference ghost_state: species 1 is absorbed at walls
    return p;
}
} // namespace mhd

using namespace mhd;

extern "C" {

int mhd_gpu_to_prim(MhdMesh *mesh, const double *U, int32_t n, double gamma, double rho_floor, double p_floor, double *W)
{
    return guarded([&] {
        MHD_REQUIRE(mesh && n >= 0 && MHD_ARR(U, n) && MHD_ARR(W, n), "bad argument");
        if (!n) return;
        k_to_prim<<<grid_for(n, 256), 256, 0, mesh->stream>>>(SField<const double>{U, 0, 5, 1}, SField<double>{W, 0, 5, 1}, n, 1,
                                                              gamma, rho_floor, p_floor);
        MHD_LAUNCH_CHECK();
    });
}

int mhd_gpu_limited_gradients(MhdMesh *mesh, const double *W, int32_t species, const MhdPrim *fs, int32_t limit, double rel_limit,
                              double *grad)
{
    return guarded([&] {
        MHD_REQUIRE(mesh && fs && MHD_ARR(W, mesh->v.nc) && MHD_ARR(grad, mesh->v.nc), "bad argument");
        MHD_REQUIRE(species >= 0, "negative species");
        const MeshView &m = mesh->v;
        if (!m.nc) return;
        const FluidParams p = single_species(species, fs, 0.0, limit, rel_limit);
        launch_limited_gradients(m, p, SField<const double>{W, 0, 5, 1}, SField<double>{grad, 0, 15, 1}, mesh->stream);
    });
}

int mhd_gpu_limited_gradients_wall(MhdMesh *mesh, const double *W, int32_t species, const MhdPrim *fs, int32_t limit, double rel_limit,
                                   int32_t n_wall, const int32_t *wall_faces, const double *wall_prims, double *grad)
{
    return guarded([&] {
        MHD_REQUIRE(mesh && fs && MHD_ARR(W, mesh->v.nc) && MHD_ARR(grad, mesh->v.nc), "bad argument");
        MHD_REQUIRE(species >= 0, "negative species");
        MHD_REQUIRE(n_wall >= 0 && (!n_wall || (wall_faces && wall_prims)), "bad wall ghost table");
        const MeshView &m = mesh->v;
        if (!m.nc) return;
        FluidParams p = single_species(species, fs, 0.0, limit, rel_limit);
        DBuf<int32_t> slot;
        slot.alloc(m.nf ? (size_t)m.nf : 1);
        build_wall_slots(m, wall_faces, n_wall, slot.p, mesh->stream);
        p.wall_slot = slot.p;
        p.wall_prim = wall_prims;
        p.wall_n = n_wall;
        launch_limited_gradients(m, p, SField<const double>{W, 0, 5, 1}, SField<double>{grad, 0, 15, 1}, mesh->stream);
        MHD_CUDA(cudaStreamSynchronize(mesh->stream)); // the slot map is freed on return
    });
}

int mhd_gpu_flux_rhs_wall(MhdMesh *mesh, double gamma, int32_t species, const MhdPrim *fs, const double *W, const double *grad,
                          int32_t n_wall, const int32_t *wall_faces, const double *wall_prims, double *rhs)
{
    return guarded([&] {
        MHD_REQUIRE(mesh && fs && MHD_ARR(W, mesh->v.nc) && MHD_ARR(grad, mesh->v.nc) && MHD_ARR(rhs, mesh->v.nc), "bad argument");
        MHD_REQUIRE(gamma > 1.0, "gamma must exceed 1");
        MHD_REQUIRE(n_wall >= 0 && (!n_wall || (wall_faces && wall_prims)), "bad wall ghost table");
        const MeshView &m = mesh->v;
        if (!m.nc) return;
        FluidParams p = single_species(species, fs, gamma, 1, 0.0);
        DBuf<int32_t> slot;
        slot.alloc(m.nf ? (size_t)m.nf : 1);
        build_wall_slots(m, wall_faces, n_wall, slot.p, mesh->stream);
        p.wall_slot = slot.p;
        p.wall_prim = wall_prims;
        p.wall_n = n_wall;
        mesh->scratch_face.alloc(5 * static_cast<size_t>(m.nf));
        k_face_flux<false><<<grid_for(m.nf, 128), 128, 0, mesh->stream>>>(m, p, SField<const double>{W, 0, 5, 1},
                                                                   SField<const double>{grad, 0, 15, 1}, mesh->scratch_face.p);
        MHD_LAUNCH_CHECK();
        k_gather_rhs<<<grid_for(m.nc, 256), 256, 0, mesh->stream>>>(m, 1, mesh->scratch_face.p, SField<double>{rhs, 0, 5, 1});
        MHD_LAUNCH_CHECK();
        MHD_CUDA(cudaStreamSynchronize(mesh->stream));
    });
}

int mhd_gpu_flux_rhs(MhdMesh *mesh, double gamma, int32_t species, const MhdPrim *fs, const double *W, const double *grad, double *rhs)
{
    return guarded([&] {
        MHD_REQUIRE(mesh && fs && MHD_ARR(W, mesh->v.nc) && MHD_ARR(grad, mesh->v.nc) && MHD_ARR(rhs, mesh->v.nc), "bad argument");
        MHD_REQUIRE(gamma > 1.0, "gamma must exceed 1");
        const MeshView &m = mesh->v;
        if (!m.nc) return;
        const FluidParams p = single_species(species, fs, gamma, 1, 0.0);
        mesh->scratch_face.alloc(5 * static_cast<size_t>(m.nf));
        k_face_flux<false><<<grid_for(m.nf, 128), 128, 0, mesh->stream>>>(m, p, SField<const double>{W, 0, 5, 1},
                                                                   SField<const double>{grad, 0, 15, 1}, mesh->scratch_face.p);
        MHD_LAUNCH_CHECK();
        k_gather_rhs<<<grid_for(m.nc, 256), 256, 0, mesh->stream>>>(m, 1, mesh->scratch_face.p, SField<double>{rhs, 0, 5, 1});
        MHD_LAUNCH_CHECK();
    });
}

} // extern "C"
