// Device functions of the magnetic-field side shared by several translation units.
// FP64, reference-exact: include only from files compiled with -fmad=false.
#pragma once
#include "common.cuh"

namespace mhd
{
// A cell without a fit (a singular normal matrix) has a zero field, whatever its fluxes: the diagonal of an inverse is
// positive, so three zeros mark it.
__device__ __forceinline__ bool cell_fit_skipped(const MeshView &m, int32_t c)
{
    const int64_t n = m.nc;
    return m.cinv[c] == 0 && m.cinv[4 * n + c] == 0 && m.cinv[8 * n + c] == 0;
}

// uns::reconstruct_cell_vector (src/uns/geometry/Reconstruct.cpp:8-46): area-weighted least squares
// b . n_f = flux_f / A_f.  The normal matrix depends on the metric alone: its inverse comes from the mesh
// (MeshView::cinv), and the right-hand side sum (s n)(s flux) is formed as sum n flux (the sign squares away exactly).
__device__ __forceinline__ V3 cell_vector(const MeshView &m, const double *__restrict__ flux, int32_t c)
{
    double r0 = 0, r1 = 0, r2 = 0;
    auto add = [&](int32_t f) {
        const D4 n = ld_d4(m.fna + 4 * (int64_t)f);
        if (n.w <= 0) return;
        const double phi = flux[f];
        r0 += n.x * phi;
        r1 += n.y * phi;
        r2 += n.z * phi;
    };
    if (m.faces_per_cell == 4)
    {
        const int4 f = *reinterpret_cast<const int4 *>(m.c2f_idx + 4 * (int64_t)c);
        add(f.x); add(f.y); add(f.z); add(f.w);
    }
    else
        for (int32_t k = m.c2f_ptr[c]; k < m.c2f_ptr[c + 1]; ++k) add(m.c2f_idx[k]);
    const int64_t n = m.nc;
    const double *I = m.cinv + c;
    const V3 b = mk(I[0] * r0 + I[n] * r1 + I[2 * n] * r2, I[3 * n] * r0 + I[4 * n] * r1 + I[5 * n] * r2,
                    I[6 * n] * r0 + I[7 * n] * r1 + I[8 * n] * r2);
    return cell_fit_skipped(m, c) ? mk(0, 0, 0) : b;
}

// (d1^T star2 phi)_e: the resistive current flux of ImplicitInduction::apply_F (ImplicitInduction.cpp:133-137)
// at edge e, its faces in ascending order (e2f rows), each term sgn * (star2_f phi_f)
__device__ __forceinline__ double resistive_p0(const MeshView &m, const double *__restrict__ phi, int32_t e)
{
    double p0 = 0.0;
    for (int32_t k = m.e2f_ptr[e]; k < m.e2f_ptr[e + 1]; ++k)
    {
        const int32_t f = m.e2f_idx[k];
        p0 += m.e2f_sgn[k] * (m.star2[f] * phi[f]);
    }
    return p0;
}
} // namespace mhd
