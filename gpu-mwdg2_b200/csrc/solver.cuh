// Per-leaf solver kernels, grid-stride over the device-side leaf count: one thread per leaf, in
// the DG2 stage kernels two lanes per leaf (one axis each). Each kernel gathers the leaf and
// its neighbours straight from the hierarchy, replacing the reference's sequence
// load_soln_and_nghbr_coeffs -> add_ghost_cells -> friction_implicit ->
// copy_to_buf_assem_sol -> limit_slopes -> dg2_update (or fv1_update) -> get_dt_CFL
// and its five materialised neighbour copies.
#pragma once

#include "kernels.cuh"

namespace mw {

// A first-order cell (neighbours/load_soln_and_nghbr_coeffs.cu:3-104, h = eta - z). The loop over
// the one mode changes the compiler's order of the loads: written out, k_hwfv1<float> spills more
// (4096^2 catchment, two steps 1356 -> 1386 us).
template <typename T> struct Cell { T h[1], qx[1], qy[1], z[1]; };
template <typename T> __device__ __forceinline__ void load_cell(const Hier<T>& hr, int a, Cell<T>& c)
{
#pragma unroll
    for (int m = 0; m < 1; ++m)
    {
        c.z[m] = hr.s[3][m][a];
        c.h[m] = hr.s[0][m][a] - c.z[m];
        c.qx[m] = hr.s[1][m][a];
        c.qy[m] = hr.s[2][m][a];
    }
}

// Non-reflecting wave maker of the Monai valley benchmark (operators/non_reflective_wave.cuh:
// 15-94): the characteristic reaching the boundary cell is traced back over one step by
// Newton's method (at most 101 iterations); the outgoing invariant there and the incoming
// one set by the target level h_inlet (still water 0.13535 m) give the boundary depth and
// velocity. The arithmetic follows the reference term by term, so both builds agree.
template <typename T>
__device__ __forceinline__ void monai_inflow(T h_inlet, T dt, T dxl, T hp, T up, T hb, T ub, T g, T& h_out, T& u_out)
{
    const T tol = T(1e-6), xa = -dxl / T(2.0);
    T p0 = dxl / T(2.0), p1 = p0 - dxl / T(2.0), dp = T(0.0), f1 = T(0.0);
    T f0 = (p0 - xa) + dt * ((ub - (p0 - xa) / dxl * (ub - up)) - sqrt(g * (hb - (p0 - xa) / dxl * (hb - hp))));
    int cond = 0;
    for (int k = 0; k <= 100 && cond == 0; ++k)
    {
        const T df = T(1.0) + dt * ((up - ub) / dxl - T(0.5) * pow((g * (hb - (p0 - xa) / dxl * (hb - hp))), T(-0.5)) *
                                                         (g * (hp - hb) / dxl));
        if (fabs(df) <= T(0.0))
        {
            cond = 1;   // zero slope: keep the current point
            dp = p1 - p0;
            p1 = p0;
        }
        else
        {
            dp = f0 / df;
            p1 = p0 - dp;
        }
        f1 = (p1 - xa) + dt * ((ub - (p1 - xa) / dxl * (ub - up)) - sqrt(g * (hb - (p1 - xa) / dxl * (hb - hp))));
        const T relerr = fabs(dp) / (fabs(p1) + T(0.0));
        if (relerr < tol) cond = 2;
        if (fabs(f1) < tol) cond = 3;
        if (relerr <= tol && fabs(f1) < tol) cond = 4;
        p0 = p1;
        f0 = f1;
    }
    const T hr = hb - (hb - hp) * (p1 - xa) / dxl;
    const T ur = ub - (ub - up) * (p1 - xa) / dxl;
    const T cr = sqrt(g * hr);
    const T beta_minus = ur - T(2.0) * cr;
    const T beta_plus = T(2.0) * sqrt(g * (h_inlet + T(0.13535))) + h_inlet * sqrt(g / T(0.13535));
    h_out = T(1.0) / T(16.0) / g * (beta_plus - beta_minus) * (beta_plus - beta_minus);
    u_out = T(0.5) * (beta_plus + beta_minus);
}

// Ghost cells of a leaf at the domain border, raster cases
// (neighbours/add_ghost_cells.cu:18-500): directions N, E, S, W in order; a fine
// boundary cell of an HFIX/HVAR/QFIX/QVAR segment also resets the leaf's own depth.
// gh/gq*: mode-0 values of the ghost in direction d (slopes are zero, bed = own bed).
template <typename T>
__device__ __forceinline__ void ghost_pass(T& own_h0, T own_qx0, T own_qy0, T own_z0, const int32_t (&nid)[4], int level,
                                           int act, const Params<T>& P, const Bnd<T>& B, T dt, T (&gh)[4], T (&gqx)[4],
                                           T (&gqy)[4])
{
    const int code = act - lvl_idx(level);
    const int x = compact(code), y = compact(code >> 1);
    const bool finest = (level == P.L);
#pragma unroll
    for (int d = 0; d < 4; ++d)
    {
        if (nid[d] != -1) continue;
        gh[d] = own_h0;
        gqx[d] = (d == 1 || d == 3) ? T(0.0) : own_qx0;
        gqy[d] = (d == 0 || d == 2) ? T(0.0) : own_qy0;
        const int c = (d == 0 || d == 2) ? x : y;
        const bool bound = (c >= B.start[d] && c <= B.end[d]);
        const bool border = (d == 0) ? (y == P.ysz - 1) : (d == 1) ? (x == P.xsz - 1) : (d == 2) ? (y == 0) : (x == 0);
        if (!(finest && bound && border)) continue;
        const int t = B.type[d];
        if (t == FREE)
        {
            const T q = (d == 0 || d == 2) ? own_qy0 : own_qx0;
            gh[d] = pow((q * q) / P.g, T(1.0) / T(3.0));
            gqx[d] = own_qx0;
            gqy[d] = own_qy0;
        }
        else if ((t == HFIX || t == HVAR) && d == 3 && B.west_special == 1)
        {
            // monai: the ghost carries the wave maker's state, the leaf keeps its own
            const T up = (own_h0 > P.tol_h) ? own_qx0 / own_h0 : T(0.0);
            T hb, ub;
            monai_inflow(B.inlet[d], dt, P.dx, own_h0, up, T(0.13535), T(0.0), P.g, hb, ub);
            gh[d] = hb - own_z0;
            gqx[d] = hb * ub;
        }
        else if ((t == HFIX || t == HVAR) && d == 3 && B.west_special == 2)
        {
            // oregon-seaside: wave-maker speed s(t), the ghost reflects the leaf's velocity about 2s
            gh[d] = own_h0;
            const T s = T(0.6) * exp(-T(0.25) * (B.time - T(14.75)) * (B.time - T(14.75)));
            const T v0 = (own_h0 > P.tol_h) ? own_qx0 / own_h0 : T(0.0);
            gqx[d] = ((T(2.0) * s - v0) * gh[d]);
        }
        else if (t == HFIX || t == HVAR)
        {
            own_h0 = B.inlet[d] - own_z0;
            gh[d] = own_h0;
        }
        else if (t == QFIX || t == QVAR)
        {
            own_h0 = B.inlet[d] * dt / P.dx;
            gh[d] = own_h0;
        }
    }
}

// operators/friction_implicit.cu:155-264 -- implicit friction on the mode-0 value and,
// for MWDG2, on the four Gauss-point values, whose differences rebuild the slopes.
// One out-of-line copy of the implicit Manning update of a point value (apply_friction):
// the stage kernel applies it at 9 to 13 points per lane of a moving leaf (3 of the leaf, 3 of
// each neighbour, 5 of one of another size) and would otherwise hold as many inlined copies
// of its pow and divisions, which stall warps on instruction fetch.
template <typename T> struct Q2 { T qx, qy; };
template <typename T> __device__ __noinline__ Q2<T> friction_point(T h, T qx, T qy, T tol_h, T tol_s, T n, T g, T dt)
{
    apply_friction(h, tol_h, tol_s, qx, qy, n, g, dt);
    return {qx, qy};
}

// Friction of a first-order cell.
template <typename T> __device__ __forceinline__ void friction_cell(Cell<T>& c, const Params<T>& P, T dt)
{
    apply_friction(c.h[0], P.tol_h, P.tol_s, c.qx[0], c.qy[0], P.manning, P.g, dt);
}

// ---------------------------------------------------------------- DG2: two lanes per leaf
//
// Lane 0 of a pair takes the leaf's y axis (faces N and S), lane 1 its x axis (E and W). A lane
// holds of the own cell mode 0 and the axis' slope mode (1y or 1x), which is all that the
// axis' face values, limiter and friction points read, and writes fields as (h, n, t): the
// depth, the discharge along the axis and the one across it, so both lanes run one code.

// A lane's arrays, chosen without indexing the parameter block by a runtime value.
template <typename T> struct Axis
{
    T *h0, *hm, *n0, *nm, *t0, *tm;   // modes 0 and m (the axis' slope) of h (or eta), n and t
};
template <typename T> __device__ __forceinline__ Axis<T> axis_of(const Hier<T>& h, bool x)
{
    return {h.s[0][0], x ? h.s[0][1] : h.s[0][2], x ? h.s[1][0] : h.s[2][0], x ? h.s[1][1] : h.s[2][2],
            x ? h.s[2][0] : h.s[1][0], x ? h.s[2][1] : h.s[1][2]};
}
template <typename T> __device__ __forceinline__ Axis<T> axis_of(const Leaves<T>& l, bool x)
{
    return {l.un[0], x ? l.un[1] : l.un[2], x ? l.un[3] : l.un[6], x ? l.un[4] : l.un[8],
            x ? l.un[6] : l.un[3], x ? l.un[7] : l.un[5]};
}

// Friction of a point value in a lane's (n, t) order.
template <typename T>
__device__ __forceinline__ void friction_axis(bool x, T h, T& n, T& t, const Params<T>& P, T dt)
{
    const Q2<T> r = friction_point(h, x ? n : t, x ? t : n, P.tol_h, P.tol_s, P.manning, P.g, dt);
    n = x ? r.qx : r.qy;
    t = x ? r.qy : r.qx;
}

// Friction of a cell's slope along one axis: the point values at its two face centres there
// (value -/+ slope), whose half difference is the new slope.
template <typename T>
__device__ __forceinline__ void friction_slope(bool x, T h0, T n0, T t0, T hm, T& nm, T& tm, const Params<T>& P, T dt)
{
    T ln = n0 - nm, lt = t0 - tm, un = n0 + nm, ut = t0 + tm;
    friction_axis(x, h0 - hm, ln, lt, P, dt);
    friction_axis(x, h0 + hm, un, ut, P, dt);
    nm = T(0.5) * (un - ln);
    tm = T(0.5) * (ut - lt);
}

// What the limiter and the flux of a face need from its neighbour: the values at the face
// (suffix f) and mode 0.
template <typename T> struct NbFace
{
    T h0, n0, t0, z0, hf, nf, tf, zf, etaf;
};

// The neighbour `nid` (level nlvl; -1: the ghost cell with depth gh and discharges gn, gt over
// the own bed z0, slopes zero) across the high (N, E) or low (S, W) face of a leaf centred
// at (xc, yc): its coefficients, rubbed when `fric`, at the shared face
// (operators/get_leg_basis.cuh:12-40 with get_{x,y}_face_{coord,unit}.cuh).
template <typename T>
__device__ __forceinline__ NbFace<T> neighbour(const Hier<T>& hr, const Axis<T>& A, bool x, bool high, int nid, int nlvl, T gh,
                                               T gn, T gt, T z0, T xc, T yc, T dxl, bool fric, const Params<T>& P, T dt)
{
    // c*[0]: mode 0, c*[1]: the slope along the axis, c*[2]: across it
    T h[3], n[3], t[3], z[3], bm, bt;
    if (nid != -1)
    {
        const T dn = P.dx * (1 << (P.L - nlvl));
        const int code = nid - lvl_idx(nlvl);
        // the face centre and the neighbour's centre along the axis (a) and across it (c)
        const T a = x ? xc : yc, c = x ? yc : xc;
        const T an = cell_centre(compact(x ? code : code >> 1), dn), cn = cell_centre(compact(x ? code >> 1 : code), dn);
        const T a_face = a - dxl / T(2.0) + (high ? T(1.0) : T(0.0)) * dxl, c_face = c - dxl / T(2.0) + T(0.5) * dxl;
        bm = sqrt(T(3.0)) * (T(2.0) * ((a_face - (an - dn / T(2.0))) / dn) - T(1.0));
        bt = sqrt(T(3.0)) * (T(2.0) * ((c_face - (cn - dn / T(2.0))) / dn) - T(1.0));
        const T* const zm = x ? hr.s[3][1] : hr.s[3][2];
        const T* const zt = x ? hr.s[3][2] : hr.s[3][1];
        const T* const ht = x ? hr.s[0][2] : hr.s[0][1];
        const T* const nt = x ? hr.s[1][2] : hr.s[2][1];
        const T* const tt = x ? hr.s[2][2] : hr.s[1][1];
        z[0] = hr.s[3][0][nid]; z[1] = zm[nid]; z[2] = zt[nid];
        h[0] = A.h0[nid] - z[0]; h[1] = A.hm[nid] - z[1]; h[2] = ht[nid] - z[2];
        n[0] = A.n0[nid]; n[1] = A.nm[nid]; n[2] = nt[nid];
        t[0] = A.t0[nid]; t[1] = A.tm[nid]; t[2] = tt[nid];
    }
    else
    {
        bm = bt = T(0.0);
        z[0] = z0; h[0] = gh; n[0] = gn; t[0] = gt;
        z[1] = z[2] = h[1] = h[2] = n[1] = n[2] = t[1] = t[2] = T(0.0);
    }
    if (fric)
    {
        T rn = n[0], rt = t[0];
        friction_axis(x, h[0], rn, rt, P, dt);
        // points along the face only where the basis there is not zero (a neighbour of
        // another size): the slope they give is otherwise multiplied by zero
        if (bm != T(0.0)) friction_slope(x, h[0], n[0], t[0], h[1], n[1], t[1], P, dt);
        if (bt != T(0.0)) friction_slope(x, h[0], n[0], t[0], h[2], n[2], t[2], P, dt);
        n[0] = rn; t[0] = rt;
    }
    NbFace<T> r;
    r.h0 = h[0]; r.n0 = n[0]; r.t0 = t[0]; r.z0 = z[0];
    // modes in the order 0, 1x, 1y, as the reference sums them, both products fused (stated,
    // since the selects may otherwise keep the compiler from it)
    const T bx = x ? bm : bt, by = x ? bt : bm;
    auto at = [&](const T (&v)[3]) { return fma(x ? v[2] : v[1], by, fma(x ? v[1] : v[2], bx, v[0])); };
    r.hf = at(h); r.nf = at(n); r.tf = at(t); r.zf = at(z);
    const T e[3] = {z[0] + h[0], z[1] + h[1], z[2] + h[2]};
    r.etaf = at(e);
    return r;
}

// Limited slope of one field along the lane's axis (operators/get_limited_slopes.cuh:10-78):
// u0, um the own coefficients; hf, lf and h0, l0 the high and low neighbours' face values and
// mode 0. The x differences are divided by sqrt(3), as the reference does.
template <typename T>
__device__ __forceinline__ T limited_slope(bool x, T u0, T um, T hf, T lf, T h0, T l0, T dxf, T tolK)
{
    const T s3 = sqrt(T(3.0));
    const T jh = fabs(hf - (u0 + um * s3)), jl = fabs((u0 - um * s3) - lf);
    const T norm = fmax(fabs(u0 - um), fabs(u0 + um));
    const T dh = (norm > T(1e-12)) ? jh / (T(0.5) * dxf * norm) : T(0.0);
    const T dl = (norm > T(1e-12)) ? jl / (T(0.5) * dxf * norm) : T(0.0);
    T a = u0 - l0, b = h0 - u0;
    if (x) { a = a / s3; b = b / s3; }
    return fmax(dh, dl) < tolK ? um : minmod(um, a, b);
}

// Leaf state u (h, qx, qy by mode, the layout of Leaves::un) into the hierarchy at `a`,
// depths as surface elevations eta = h + z (mra/reinsert_assem_sol.cu:3-32).
template <typename T>
__device__ __forceinline__ void put_leaf(const Hier<T>& hr, int a, const T (&u)[9], const T (&z)[3], uint32_t mark = 0)
{
#pragma unroll
    for (int m = 0; m < 3; ++m)
    {
        hr.s[0][m][a] = u[m] + z[m];
        hr.s[1][m][a] = u[3 + m];
        hr.s[2][m][a] = u[6 + m];
    }
    if (hr.tag) hr.tag[a] = mark;   // the stage hierarchy of the keep-values decode
}

// Running maxima of the state at the end of a step, as the next step's
// mra/get_max_scale_coeffs.cu:3-27 reads them (|eta|, |h0|, |qx0|, |z0|; the reference
// also uses qx0 for the qy maximum).
template <typename T> struct StateMax
{
    T eta = T(0), h = T(0), qx = T(0), z = T(0);
    __device__ __forceinline__ void add(T h0, T qx0, T z0)
    {
        const T e = h0 + z0;
        eta = fmax(eta, fabs(e));
        h = fmax(h, fabs(h0));
        qx = fmax(qx, fabs(qx0));
        z = fmax(z, fabs(z0));
    }
    __device__ __forceinline__ void flush(Scalars<T>* sc)
    {
        T v[4] = {eta, h, qx, z};
        T* const dst[4] = {&sc->next_max[0], &sc->next_max[1], &sc->next_max[2], &sc->next_max[3]};
        block_max_atomic<T, 4>(v, dst);
    }
};

// The FV1 result of a leaf into the other of the two alternating hierarchy buffers at the
// leaf's own index (the re-insertion of mra/reinsert_assem_sol.cu:3-32, eta = h + z), and
// into the maxima the next step's thresholds use (mra/get_max_scale_coeffs.cu:3-27).
template <typename T>
__device__ __forceinline__ void put_leaf_fv1(const Hier<T>& hout, int a, T h, T qx, T qy, T z, StateMax<T>& mx)
{
    hout.s[0][0][a] = h + z;
    hout.s[1][0][a] = qx;
    hout.s[2][0][a] = qy;
    mx.add(h, qx, z);
}

// Wet test of one RK stage: a leaf is dry when its own depth and its four neighbours' (after
// ghost cells) are all below tol_h, and is then not updated, limited or rubbed. Wet leaves are
// appended to `wet` (warp-aggregated) for k_mwdg2_stage<.., LIST=true> (a NaN depth is not
// below tol_h, so a NaN leaf is listed and the stage kernel reports it), dry ones marked in
// `dry` for k_stage_dry, which then runs beside the wet-list kernel (the two touch disjoint
// leaves). Stage 1 also keeps a dry leaf's depth after ghost cells in U^n (un[0]); stage 2
// reports initial_tstep as the CFL step of dry leaves (dg2_update.cu:61).
template <typename T, int STAGE>
__device__ __forceinline__ void k_stage_wet_body(int bid, int nb, Leaves<T> lf, Hier<T> hin, Scalars<T>* sc, Params<T> P,
                                                   const StepArgs<T>* args, uint8_t* dry, int32_t* wet,
                                                   const uint8_t* dry1 = nullptr, uint32_t* clean_tag = nullptr)
{
    const T dt = args->dt;
    const Bnd<T>& B = args->B;
    const int n = sc->n_leaves;
    bool any_dry = false;
    for (int i0 = bid * blockDim.x; i0 < n; i0 += nb * blockDim.x)
    {
        const int i = i0 + threadIdx.x;
        bool is_wet = false;
        if (i < n)
        {
            const int a = lf.act[i];
            int32_t nid[4];
#pragma unroll
            for (int d = 0; d < 4; ++d) nid[d] = lf.nb[d][i];
            // own and neighbour loads issued together (almost every leaf is dry here); the
            // level and the discharges only enter the ghost cells of faces on the border
            // (ghost_pass)
            const bool border = (nid[0] == -1) | (nid[1] == -1) | (nid[2] == -1) | (nid[3] == -1);
            const int level = border ? lf.lvl[i] : 0;
            const T e0 = hin.s[0][0][a], z0 = hin.s[3][0][a];
            const T qx0 = border ? hin.s[1][0][a] : T(0.0), qy0 = border ? hin.s[2][0][a] : T(0.0);
            T nbh[4];
#pragma unroll
            for (int d = 0; d < 4; ++d)
                nbh[d] = (nid[d] != -1) ? hin.s[0][0][nid[d]] - hin.s[3][0][nid[d]] : T(0.0);
            T h0 = e0 - z0;
            T gh[4], gqx[4], gqy[4];
            ghost_pass(h0, qx0, qy0, z0, nid, level, a, P, B, dt, gh, gqx, gqy);
            bool is_dry = h0 < P.tol_h;
#pragma unroll
            for (int d = 0; d < 4; ++d) is_dry = is_dry && ((nid[d] != -1) ? nbh[d] : gh[d]) < P.tol_h;
            is_wet = !is_dry;
            any_dry |= is_dry;
            dry[i] = is_dry ? 1 : 0;
            if (STAGE == 1 && is_dry) lf.un[0][i] = h0;
            if (STAGE == 2 && clean_tag && is_dry && dry1[i]) clean_tag[a] = sc->step_tag;
        }
        // warp-aggregated append
        const unsigned mask = __ballot_sync(0xffffffffu, is_wet);
        const int lane = threadIdx.x & 31;
        int base = 0;
        if (lane == 0 && mask) base = atomicAdd(&sc->wet[STAGE - 1], __popc(mask));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (is_wet) wet[base + __popc(mask & ((1u << lane) - 1u))] = i;
    }
    if (STAGE == 2 && __syncthreads_or(any_dry) && threadIdx.x == 0) atomic_min_nn(&sc->dt_min, P.initial_tstep);
}
template <typename T, int STAGE>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 8 : 4) k_stage_wet(Leaves<T> lf, Hier<T> hin, Scalars<T>* sc, Params<T> P,
                                                   const StepArgs<T>* args, uint8_t* dry, int32_t* wet,
                                                   const uint8_t* dry1 = nullptr, uint32_t* clean_tag = nullptr)
{
    k_stage_wet_body<T, STAGE>(blockIdx.x, gridDim.x, lf, hin, sc, P, args, dry, wet, dry1, clean_tag);
}

// The dry leaves of one RK stage, marked by k_stage_wet (bandwidth-bound; it runs beside
// the latency-bound wet-list kernel). Stage 1 (hin: hierarchy, hout: stage hierarchy): U^n
// is the leaf's state with the discharge cleared by friction (depth after ghost cells as
// k_stage_wet left it in un[0]) and U* equals it. Stage 2 (hout: hierarchy): the leaf keeps
// U^n, which is re-inserted into the hierarchy and enters the next step's maxima.
// pm (learned refinement proposal, applied steps with both stages over the wet list): a
// leaf inside a subtree the proposal left out (its subtree's encode and decode are skipped
// too) keeps its state as it stands in the hierarchy where nothing has changed it. With the
// keep-values decode, which rewrites no leaf that persists, pm leaves out every subtree but
// those holding point sources.
// Stage 1 leaves such a dry leaf's U* in the stage hierarchy as it stands when the leaf was
// a leaf dry in both stages of the last step (clean_tag[a], at its hierarchy index, is the
// last step's tag: written by that step's stage-2 wet test; null when that step did not
// record it): U* is then still the one written when the leaf last changed. Its U^n copy
// (un, by leaf position) is rewritten only where the position now holds another leaf than
// in the last step (lf.same). Stage 1 marks the leaves it freezes (dry[i] = 2); stage 2
// writes nothing for such a leaf that is dry in stage 2 as well (dry1: stage 1's marks) and
// only adds it to the maxima, so a leaf's state is re-inserted at least once after it last
// changed.
template <typename T, int STAGE>
__device__ __forceinline__ void k_stage_dry_body(int bid, int nb, Leaves<T> lf, Hier<T> hin, Hier<T> hout, Scalars<T>* sc, Params<T> P,
                                                   bool friction, uint8_t* dry, const uint8_t* dry1, PropMask pm,
                                                   const uint32_t* clean_tag = nullptr)
{
    const uint32_t last_tag = sc->step_tag - 1u;
    const uint32_t wmark = (sc->step_tag << 1) | 1u;   // a written stage-hierarchy slot (Hier::tag)
    const int n = sc->n_leaves;
    const int stride = nb * blockDim.x;
    StateMax<T> mx;
    unsigned frozen = 0;
    // software pipeline: the next leaf's mark and hierarchy index are loaded while this
    // leaf's gathers at its index are in flight (one dependent round trip per leaf, not two)
    int i = bid * blockDim.x + threadIdx.x;
    bool dry_next = i < n && dry[i];
    int a_next = i < n ? lf.act[i] : 0;
    for (; i < n; i += stride)
    {
        const bool is_dry = dry_next;
        const int a = a_next;
        if (i + stride < n)
        {
            dry_next = dry[i + stride];
            a_next = lf.act[i + stride];
        }
        if (!is_dry) continue;
        bool keep_ustar = false;
        if (pm.prop && (STAGE == 2 || clean_tag))
        {
            const int lv = lf.lvl[i];
            const bool left_out = lv >= pm.level && pm_out(pm, (a - lvl_idx(lv)) >> (2 * (lv - pm.level)));
            if (STAGE == 1 && left_out && clean_tag[a] == last_tag)
            {
                dry[i] = 2;
                ++frozen;
                if (hout.tag) hout.tag[a] = wmark & ~1u;   // U* stands
                if (lf.same[i]) continue;
                keep_ustar = true;   // un only
            }
            if (STAGE == 2 && left_out && dry1[i] == 2)
            {
                mx.add(lf.un[0][i], lf.un[3][i], hin.s[3][0][a]);
                if (P.dt_leaf) P.dt_leaf[i] = P.initial_tstep;
                continue;
            }
        }
        const T z[3] = {hin.s[3][0][a], hin.s[3][1][a], hin.s[3][2][a]};
        T u[9];
        if (STAGE == 1)
        {
            u[0] = lf.un[0][i];
            u[3] = friction ? T(0.0) : hin.s[1][0][a];
            u[6] = friction ? T(0.0) : hin.s[2][0][a];
#pragma unroll
            for (int m = 1; m < 3; ++m)
            {
                u[m] = hin.s[0][m][a] - z[m];
                u[3 + m] = hin.s[1][m][a];
                u[6 + m] = hin.s[2][m][a];
            }
#pragma unroll
            for (int k = 1; k < 9; ++k) lf.un[k][i] = u[k];
            if (keep_ustar) continue;
        }
        else
        {
#pragma unroll
            for (int k = 0; k < 9; ++k) u[k] = lf.un[k][i];
            mx.add(u[0], u[3], z[0]);
            if (P.dt_leaf) P.dt_leaf[i] = P.initial_tstep;
        }
        put_leaf(hout, a, u, z, wmark);
    }
    if (STAGE == 2) mx.flush(sc);
    if (STAGE == 1 && pm.prop)
    {
        frozen = __reduce_add_sync(0xffffffffu, frozen);
        if ((threadIdx.x & 31) == 0 && frozen) atomicAdd(&sc->prop_frozen, frozen);
    }
}
template <typename T, int STAGE>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 8 : 5) k_stage_dry(Leaves<T> lf, Hier<T> hin, Hier<T> hout, Scalars<T>* sc, Params<T> P,
                                                   bool friction, uint8_t* dry, const uint8_t* dry1, PropMask pm,
                                                   const uint32_t* clean_tag = nullptr)
{
    k_stage_dry_body<T, STAGE>(blockIdx.x, gridDim.x, lf, hin, hout, sc, P, friction, dry, dry1, pm, clean_tag);
}

// ---------------------------------------------------------------- RK stages in place
//
// Steps whose two stages take the wet list (reference decode, no proposal): U* of a leaf stands
// in the hierarchy itself. Almost every leaf is dry and ends both stages as it started, so
// it is left alone: the wet test checks that the stage would put the same elevations back
// (eta = (eta - z) + z), and with friction k_apply clears its mode-0 discharge, which the decode
// left as rounding noise. The wet list's kernel, and the test for the few dry leaves that do
// change, write their results to the leaf's slot of the stage hierarchy, and k_apply copies them
// into the hierarchy once no leaf reads the old state any more. Neighbours that are significant parents (Leaves::par) take
// their U* from the stage hierarchy, where the scale re-encode puts it.
// Marks of stage 1 (`mark`): 0 wet, 1 dry and standing, 2 dry and changed. A standing leaf's
// U^n is not stored: it is the hierarchy's own value (k_fill_un writes it where a getter needs it).
// It replaces two writers of the dry leaves that moved 30 + 21 values a leaf. 4096^2 catchment,
// 1 % wet, FP32 (ncu, per launch, stage 1 / 2): wet test 34 / 33 and dry writer 126 / 91 us
// beside the wet list's kernel -> wet test 44 / 46, wet list 23 / 22, k_apply 19 / 6 us one after
// another; step 0.637 -> 0.492 ms, FP64 (dry start) 0.911 -> 0.693 ms.

// Position in a list of `n` entries for each lane with `in`, one atomic per warp.
__device__ __forceinline__ int list_slot(bool in, int32_t* n)
{
    const unsigned mask = __ballot_sync(0xffffffffu, in);
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (mask)
    {
        if (lane == 0) base = atomicAdd(n, __popc(mask));
        base = __shfl_sync(0xffffffffu, base, 0);
    }
    return base + __popc(mask & ((1u << lane) - 1u));
}

// Wet test of one in-place stage (the rule of k_stage_wet): wet leaves to `wet`, dry leaves
// whose state changes to a second list that fills the same array from its end (`fix`, its last
// entry, backwards: no leaf is in both), their new values to their slots of hs.
// Stage 1 (marks -> mark): U* = U^n with the depth after ghost cells and no discharge under
// friction. Stage 2 (mark: stage 1's; marks -> mark2): U^{n+1} = U^n, which has to be put back
// only where stage 1 moved the leaf; dry leaves enter the next step's maxima and report
// initial_tstep as their CFL step.
template <typename T, int STAGE>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 6 : 4) k_inplace_wet(Leaves<T> lf, Hier<T> hr, Hier<T> hs, Scalars<T>* sc, Params<T> P,
                                                                        const StepArgs<T>* args, bool friction, uint8_t* mark,
                                                                        uint8_t* mark2, int32_t* wet, int32_t* fix)
{
    const T dt = args->dt;
    const Bnd<T>& B = args->B;
    const int n = sc->n_leaves;
    bool any_dry = false;
    StateMax<T> mx;
    for (int i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x)
    {
        const int i = i0 + threadIdx.x;
        bool is_wet = false, is_fix = false;
        if (i < n)
        {
            const int a = lf.act[i];
            int32_t nid[4];
#pragma unroll
            for (int d = 0; d < 4; ++d) nid[d] = lf.nb[d][i];
            const unsigned par = STAGE == 2 ? lf.par[i] >> 4 : 0u;
            const uint8_t m1 = STAGE == 2 ? mark[i] : 0;
            const bool border = (nid[0] == -1) | (nid[1] == -1) | (nid[2] == -1) | (nid[3] == -1);
            const int level = border ? lf.lvl[i] : 0;
            const T e0 = hr.s[0][0][a], z0 = hr.s[3][0][a];
            const T qx0 = border || (STAGE == 2 && !friction) ? hr.s[1][0][a] : T(0.0);
            const T qy0 = border ? hr.s[2][0][a] : T(0.0);
            T e1 = T(0.0), z1 = T(0.0), e2 = T(0.0), z2 = T(0.0);
            if (STAGE == 1) { e1 = hr.s[0][1][a]; z1 = hr.s[3][1][a]; e2 = hr.s[0][2][a]; z2 = hr.s[3][2][a]; }
            T nbh[4];
#pragma unroll
            for (int d = 0; d < 4; ++d)
            {
                const T* const eta = (par >> d) & 1u ? hs.s[0][0] : hr.s[0][0];
                nbh[d] = (nid[d] != -1) ? eta[nid[d]] - hr.s[3][0][nid[d]] : T(0.0);
            }
            T h0 = e0 - z0;
            T gh[4], gqx[4], gqy[4];
            ghost_pass(h0, qx0, qy0, z0, nid, level, a, P, B, dt, gh, gqx, gqy);
            bool is_dry = h0 < P.tol_h;
#pragma unroll
            for (int d = 0; d < 4; ++d) is_dry = is_dry && ((nid[d] != -1) ? nbh[d] : gh[d]) < P.tol_h;
            is_wet = !is_dry;
            any_dry |= is_dry;
            T u[9];
            if (STAGE == 1)
            {
                const T h1 = e1 - z1, h2 = e2 - z2;
                // (a depth that a boundary segment reset has to be the hierarchy's own as well: the
                // elevations alone may agree by rounding)
                const bool stands = h0 == e0 - z0 && h0 + z0 == e0 && h1 + z1 == e1 && h2 + z2 == e2;
                is_fix = is_dry && !stands;
                mark[i] = is_wet ? 0 : stands ? 1 : 2;
                if (is_fix)
                {
                    u[0] = h0; u[1] = h1; u[2] = h2;
                    u[3] = friction ? T(0.0) : hr.s[1][0][a];
                    u[6] = friction ? T(0.0) : hr.s[2][0][a];
#pragma unroll
                    for (int m = 1; m < 3; ++m) { u[3 + m] = hr.s[1][m][a]; u[6 + m] = hr.s[2][m][a]; }
#pragma unroll
                    for (int k = 0; k < 9; ++k) lf.un[k][i] = u[k];
                    const T z[3] = {z0, z1, z2};
                    put_leaf(hs, a, u, z);
                }
            }
            else
            {
                mark2[i] = (uint8_t)(par << 4 | (is_dry ? 1u : 0u));   // (lf.par, for the wet list)
                is_fix = is_dry && m1 == 0;
                if (is_dry)
                {
                    // U^n of a standing leaf is the hierarchy's own value
                    if (m1 == 1) mx.add(e0 - z0, friction ? T(0.0) : qx0, z0);
                    else mx.add(lf.un[0][i], lf.un[3][i], z0);
                    if (P.dt_leaf) P.dt_leaf[i] = P.initial_tstep;
                }
                if (is_fix)
                {
                    const T z[3] = {z0, hr.s[3][1][a], hr.s[3][2][a]};
#pragma unroll
                    for (int k = 0; k < 9; ++k) u[k] = lf.un[k][i];
                    put_leaf(hs, a, u, z);
                }
            }
        }
        int at = list_slot(is_wet, &sc->wet[STAGE - 1]);
        if (is_wet) wet[at] = i;
        at = list_slot(is_fix, &sc->fix[STAGE - 1]);
        if (is_fix) fix[-at] = i;
    }
    if (STAGE == 2)
    {
        mx.flush(sc);
        if (__syncthreads_or(any_dry) && threadIdx.x == 0) atomic_min_nn(&sc->dt_min, P.initial_tstep);
    }
}

// The listed leaves' results from their slots of the stage hierarchy into the hierarchy;
// mark (stage 1 with friction): also the standing leaves' mode-0 discharge cleared.
template <typename T>
__global__ void __launch_bounds__(256) k_apply(Leaves<T> lf, Hier<T> hs, Hier<T> hr, const Scalars<T>* sc, int stage, const int32_t* wet,
                                               const int32_t* fix, const uint8_t* mark)
{
    if (mark)
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < sc->n_leaves; i += gridDim.x * blockDim.x)
        {
            if (mark[i] != 1) continue;
            const int a = lf.act[i];
            hr.s[1][0][a] = T(0.0);
            hr.s[2][0][a] = T(0.0);
        }
    const int nw = sc->wet[stage - 1], n = nw + sc->fix[stage - 1];
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
    {
        const int a = lf.act[k < nw ? wet[k] : fix[nw - k]];
        T v[9];
#pragma unroll
        for (int j = 0; j < 9; ++j) v[j] = hs.s[j / 3][j % 3][a];
#pragma unroll
        for (int j = 0; j < 9; ++j) hr.s[j / 3][j % 3][a] = v[j];
    }
}

// U^n (the leaf state) of the leaves that stood through both stages of an in-place step.
template <typename T>
__global__ void __launch_bounds__(256) k_fill_un(Leaves<T> lf, Hier<T> hr, const Scalars<T>* sc, const uint8_t* mark, const uint8_t* mark2)
{
    const int n = sc->n_leaves;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        if (mark[i] != 1 || !(mark2[i] & 1)) continue;
        const int a = lf.act[i];
#pragma unroll
        for (int m = 0; m < 3; ++m)
        {
            lf.un[m][i] = hr.s[0][m][a] - hr.s[3][m][a];
            lf.un[3 + m][i] = hr.s[1][m][a];
            lf.un[6 + m][i] = hr.s[2][m][a];
        }
    }
}

// Resident blocks of k_mwdg2_stage per SM that its registers are held to (64 in FP32, 128 in
// FP64). Bytes of spill stores / loads by ptxas: FP32 stage 1 144 / 76, stage 2 112 / 108, stage 2
// in place 300 / 236 (each neighbour comes from one of two hierarchies); FP64 148 / 112, 96 / 120
// and 152 / 156. 8 / 4 blocks took 135.8 us for the dam-break step and 3.74 ms for the
// ensemble's where 6 / 3 took 148.6 us and 3.94 ms; 9 / 5 and 10 / 6 are within noise of it.
template <typename T> constexpr int kStageBlocks = sizeof(T) == 4 ? 8 : 4;

// One RK2 stage of MWDG2, reading the hierarchy `hin` and writing each leaf's result into
// the hierarchy `hout` at the leaf's own index (which no leaf reads in this stage).
// STAGE 1 (hin: hierarchy, hout: stage hierarchy): friction (once per step), limiter with
// the step's max depth, U* -> hout, U^n (after friction and limiter) -> un.
// STAGE 2 (hin: stage hierarchy, hout: hierarchy): limiter with the stage's max depth,
// U^{n+1} = (U** + U^n)/2 -> un and hout (the next step's re-insertion,
// mra/reinsert_assem_sol.cu), the next step's maxima, CFL dt. LIST: only the leaves in
// the wet list built by k_stage_wet; otherwise every leaf.
//
// What bounds it: few wet leaves, one leaf's serial latency; many, instruction issue (IEEE
// divisions, square roots and pow of the friction and the fluxes). Two lanes per leaf halve the
// chain of a leaf's faces, and need about half the registers of a thread that holds all four. What
// concerns the leaf as a whole both lanes evaluate: its mean friction point, the speed test's
// divisions, the cell's centre, the mode-0 update, sqrt(g h), the ghost cells of a border leaf.
// Against one thread per leaf (ncu, per launch, stage 1 / 2): 256^2 dam break FP64, every leaf
// wet, 33.3 / 33.7 -> 15.3 / 17.6 us; 1000 x 700 flood FP64 54.8 / 28.8 -> 34.5 / 23.1 us; wet
// list of the 2048^2 urban case FP32 86.2 / 58.5 -> 74.9 / 56.3 us; step of eight ensemble
// members FP32 3.90 -> 3.52 ms. Four lanes per leaf (a face each) evaluated too much twice
// (dam break step 142 -> 158 us, ensemble 4.37 -> 4.96 ms where this form takes 3.74).
// INPL (stage 2 of an in-place step, mark: stage 1's marks): hin is the hierarchy, whose
// significant parents' U* stands in hout, the stage hierarchy, which also takes the results.
template <typename T, int STAGE, bool LIST, bool INPL = false>
__device__ __forceinline__ void k_mwdg2_stage_body(int bid, int nb, Leaves<T> lf, Hier<T> hin, Hier<T> hout, Scalars<T>* sc,
                                                                Params<T> P, const StepArgs<T>* args, bool friction,
                                                                const int32_t* wet, const uint8_t* mark = nullptr)
{
    const T dt = args->dt;
    const Hier<T>& hr = hin;
    StateMax<T> mx;
    const int nl = LIST ? sc->wet[STAGE - 1] : sc->n_leaves;
    T dt_loc = (sizeof(T) == 8) ? T(1.0e308) : T(3.0e38);
    bool nan_seen = false;
    unsigned n_wet = 0;
    const T max_h = (STAGE == 1) ? fmax(T(1.0), sc->max_h) : sc->max_h2;
    const uint32_t wmark = (sc->step_tag << 1) | 1u;   // a written stage-hierarchy slot (Hier::tag)
    const bool x = (threadIdx.x & 1) != 0;
    const unsigned pair = 3u << (threadIdx.x & 30);
    const T s3 = sqrt(T(3.0));
    const Axis<T> A = axis_of(hr, x);
    const int32_t* const nb_hi = x ? lf.nb[1] : lf.nb[0];
    const int32_t* const nb_lo = x ? lf.nb[3] : lf.nb[2];
    const int per = blockDim.x >> 1;
    for (int k = bid * per + (threadIdx.x >> 1); k < nl; k += nb * per)
    {
        const int i = LIST ? wet[k] : k;
        const int a = lf.act[i];
        const int level = lf.lvl[i];
        const int id_hi = nb_hi[i], id_lo = nb_lo[i];
        const T z0 = hr.s[3][0][a], zm = (x ? hr.s[3][1] : hr.s[3][2])[a];
        T h0 = A.h0[a] - z0, hm = A.hm[a] - zm;
        T n0 = A.n0[a], nm = A.nm[a], t0 = A.t0[a], tm = A.tm[a];
        // a NaN depth anywhere in the state (a dry-looking NaN leaf is never updated below)
        nan_seen |= (h0 != h0);
        // ghost cells of border faces; a border segment may also reset the own depth, in the
        // order N, E, S, W, so both lanes of a border leaf walk all four faces
        T gh_hi = T(0.0), gn_hi = T(0.0), gt_hi = T(0.0), gh_lo = T(0.0), gn_lo = T(0.0), gt_lo = T(0.0);
        if (__ballot_sync(pair, id_hi == -1 || id_lo == -1))
        {
            const int o_hi = __shfl_xor_sync(pair, id_hi, 1), o_lo = __shfl_xor_sync(pair, id_lo, 1);
            const int32_t n4[4] = {x ? o_hi : id_hi, x ? id_hi : o_hi, x ? o_lo : id_lo, x ? id_lo : o_lo};
            T gh[4], gqx[4], gqy[4];
            ghost_pass(h0, x ? n0 : t0, x ? t0 : n0, z0, n4, level, a, P, args->B, dt, gh, gqx, gqy);
            gh_hi = x ? gh[1] : gh[0]; gn_hi = x ? gqx[1] : gqy[0]; gt_hi = x ? gqy[1] : gqx[0];
            gh_lo = x ? gh[3] : gh[2]; gn_lo = x ? gqx[3] : gqy[2]; gt_lo = x ? gqy[3] : gqx[2];
        }
        // A leaf whose own depth and neighbour depths (after ghost cells) are all below tol_h
        // is not updated (dg2_update.cu:36-50), is not limited (the limiter needs a depth
        // above 0.05 max_h) and, being below tol_h, gets no friction: it needs none of the
        // neighbours' other coefficients.
        bool dry = false;
        if (!LIST)
        {
            const T hh = id_hi != -1 ? hr.s[0][0][id_hi] - hr.s[3][0][id_hi] : gh_hi;
            const T hl = id_lo != -1 ? hr.s[0][0][id_lo] - hr.s[3][0][id_lo] : gh_lo;
            dry = __ballot_sync(pair, !(hh < P.tol_h) || !(hl < P.tol_h)) == 0 && h0 < P.tol_h;
            n_wet += (dry || x) ? 0 : 1;
        }
        // friction_implicit.cu:24-48: shallow or slow leaves lose their discharge and
        // skip friction (their neighbours' copies are then left untouched too)
        bool fric = false;
        if (STAGE == 1 && friction)
        {
            const bool below_depth = (h0 < P.tol_h);
            const T un = below_depth ? T(0.0) : n0 / h0;
            const T ut = below_depth ? T(0.0) : t0 / h0;
            const bool below_speed = (fabs(un) < P.tol_s && fabs(ut) < P.tol_s);
            if (below_depth || below_speed) { n0 = T(0.0); t0 = T(0.0); }
            fric = !(below_depth || below_speed);
            if (fric)
            {
                T rn = n0, rt = t0;
                friction_axis(x, h0, rn, rt, P, dt);
                friction_slope(x, h0, n0, t0, hm, nm, tm, P, dt);
                n0 = rn; t0 = rt;
            }
        }
        // leaf state in the lane's coefficients: the slopes by both lanes, mode 0 by lane 0
        auto put = [&](T uh0, T un0, T ut0, T uhm, T unm, T utm) {
            const Axis<T> O = axis_of(hout, x);
            O.hm[a] = uhm + zm; O.nm[a] = unm; O.tm[a] = utm;
            if (!x)
            {
                O.h0[a] = uh0 + z0; O.n0[a] = un0; O.t0[a] = ut0;
                if (hout.tag) hout.tag[a] = wmark;   // the stage hierarchy of the keep-values decode
            }
        };
        auto put_un = [&](T uh0, T un0, T ut0, T uhm, T unm, T utm) {
            const Axis<T> U = axis_of(lf, x);
            U.hm[i] = uhm; U.nm[i] = unm; U.tm[i] = utm;
            if (!x) { U.h0[i] = uh0; U.n0[i] = un0; U.t0[i] = ut0; }
        };
        if (dry)
        {
            if (STAGE == 1) { put_un(h0, n0, t0, hm, nm, tm); put(h0, n0, t0, hm, nm, tm); }
            else
            {
                const Axis<T> U = axis_of(lf, x);
                const T uh = U.h0[i], un = U.n0[i], ut = U.t0[i];
                if (!x)
                {
                    mx.add(uh, ut, z0);   // (t is qx in the y lane)
                    if (P.dt_leaf) P.dt_leaf[i] = P.initial_tstep;
                }
                put(uh, un, ut, U.hm[i], U.nm[i], U.tm[i]);
            }
            dt_loc = fmin(dt_loc, P.initial_tstep);
            continue;
        }
        const T dxl = P.dx * (1 << (P.L - level));
        const int code = a - lvl_idx(level);
        const T xc = cell_centre(compact(code), dxl), yc = cell_centre(compact(code >> 1), dxl);
        const bool in_extent = !((xc >= P.xsz * P.dx) || (yc >= P.ysz * P.dx));
        const unsigned par = INPL ? lf.par[i] >> (x ? 5 : 4) : 0u;   // bits 0 and 2: the lane's faces
        const bool p_hi = INPL && (par & 1u), p_lo = INPL && (par & 4u);
        const NbFace<T> H = neighbour(p_hi ? hout : hr, p_hi ? axis_of(hout, x) : A, x, true, id_hi, id_hi == -1 ? level : level_of(id_hi), gh_hi, gn_hi, gt_hi, z0, xc, yc,
                                      dxl, STAGE == 1 && fric, P, dt);
        const NbFace<T> W = neighbour(p_lo ? hout : hr, p_lo ? axis_of(hout, x) : A, x, false, id_lo, id_lo == -1 ? level : level_of(id_lo), gh_lo, gn_lo, gt_lo, z0, xc, yc,
                                      dxl, STAGE == 1 && fric, P, dt);
        // operators/copy_to_buf_assem_sol.cu: the stage-1 result of a leaf that is not
        // updated is its state before limiting
        const T pre_h = hm, pre_n = nm, pre_t = tm;
        // operators/limit_slopes.cu:3-238 (finest-level leaves inside the DEM only)
        if (P.limit && level == P.L && in_extent)
        {
            const T e = limited_slope(x, z0 + h0, zm + hm, H.etaf, W.etaf, H.z0 + H.h0, W.z0 + W.h0, P.dx, P.tol_Krivo);
            const T p = limited_slope(x, n0, nm, H.nf, W.nf, H.n0, W.n0, P.dx, P.tol_Krivo);
            const T q = limited_slope(x, t0, tm, H.tf, W.tf, H.t0, W.t0, P.dx, P.tol_Krivo);
            if (T(0.05) * max_h < fmin(h0, fmin(H.h0, W.h0))) { hm = e - zm; nm = p; tm = q; }
        }
        if (STAGE == 1) put_un(h0, n0, t0, hm, nm, tm);
        // operators/dg2_update.cu:31-79 (wet leaves, not high wall, inside the DEM)
        const bool highwall = (fabs(z0 - P.wall_height) < T(1e-10));
        const bool any = h0 >= P.tol_h || __ballot_sync(pair, H.h0 >= P.tol_h || W.h0 >= P.tol_h) != 0;
        T leaf_dt = P.initial_tstep;
        if (any && !highwall && in_extent)
        {
            // the leaf changes: the encode of the next step revisits its subtree
            if (!x && P.act && level >= P.act_level) P.act[(a - lvl_idx(level)) >> (2 * (level - P.act_level))] = 1;
            // operators/dg2_update.cu:160-334 along the axis
            const T g = P.g, tol_h = P.tol_h;
            const T hf_h = h0 + hm * s3, hf_l = h0 - hm * s3, zf_h = z0 + zm * s3, zf_l = z0 - zm * s3;
            const T zi_h = fmax(zf_h, H.zf), zi_l = fmax(zf_l, W.zf);
            const V3<T> s_h = star(V3<T>{hf_h, n0 + nm * s3, t0 + tm * s3}, zf_h, zi_h, tol_h);
            const V3<T> s_l = star(V3<T>{hf_l, n0 - nm * s3, t0 - tm * s3}, zf_l, zi_l, tol_h);
            // (the flux's tangential component changes sign with the tangential discharge, so
            // the y lane needs no rotation of its frame)
            // The fused products are stated: the one-thread form of this kernel, whose bits agree
            // with the reference's build, fused u q everywhere but for the neighbours' side of
            // the x faces (found by comparing all choices over dam breaks, catchments and floods
            // in both precisions; this one gives the same bits everywhere).
            const V3<T> F_h = flux_hll_x<T, true>(s_h, star(V3<T>{H.hf, H.nf, H.tf}, H.zf, zi_h, tol_h), tol_h, g, false, x);
            const V3<T> F_l = flux_hll_x<T, true>(star(V3<T>{W.hf, W.nf, W.tf}, W.zf, zi_l, tol_h), s_l, tol_h, g, x, false);
            const V3<T> U0 = (s_h + s_l) / T(2.0);
            const V3<T> U1 = (s_h - s_l) / (T(2.0) * s3);
            V3<T> L0 = (-T(1.0) * (F_h - F_l)) / dxl;
            V3<T> L1 = (-s3 / dxl) * (F_h + F_l - phys_flux_x(U0 - U1, tol_h, g) - phys_flux_x(U0 + U1, tol_h, g));
            // operators/get_bed_src.cuh:46-72
            const T zs_h = zi_h - fmax(T(0.0), -((hf_h + zf_h) - zi_h));
            const T zs_l = zi_l - fmax(T(0.0), -((hf_l + zf_l) - zi_l));
            const T z1 = (zs_h - zs_l) / (T(2.0) * s3);
            L0.qx = L0.qx + -T(2.0) * s3 * g * U0.h * z1 / dxl;
            L1.qx = L1.qx + -T(2.0) * s3 * g * U1.h * z1 / dxl;
            // coeffs += dt * (Lx + Ly): mode 0 takes both axes, a slope its own
            const T oh = __shfl_xor_sync(pair, L0.h, 1);
            const T on = __shfl_xor_sync(pair, L0.qy, 1), ot = __shfl_xor_sync(pair, L0.qx, 1);
            T uh0 = h0 + dt * (L0.h + oh), un0 = n0 + dt * (L0.qx + on), ut0 = t0 + dt * (L0.qy + ot);
            T uhm = hm + dt * L1.h, unm = nm + dt * L1.qx, utm = tm + dt * L1.qy;
            if (STAGE == 2 && INPL && mark[i] == 1)
            {
                // a leaf that stood in stage 1: U^n is U*
                uh0 = T(0.5) * (uh0 + (A.h0[a] - z0)); un0 = T(0.5) * (un0 + n0); ut0 = T(0.5) * (ut0 + t0);
                uhm = T(0.5) * (uhm + pre_h); unm = T(0.5) * (unm + pre_n); utm = T(0.5) * (utm + pre_t);
            }
            else if (STAGE == 2)
            {
                const Axis<T> U = axis_of(lf, x);
                uh0 = T(0.5) * (uh0 + U.h0[i]); un0 = T(0.5) * (un0 + U.n0[i]); ut0 = T(0.5) * (ut0 + U.t0[i]);
                uhm = T(0.5) * (uhm + U.hm[i]); unm = T(0.5) * (unm + U.nm[i]); utm = T(0.5) * (utm + U.tm[i]);
            }
            if (uh0 < tol_h) un0 = ut0 = unm = utm = T(0.0);
            else if (STAGE == 2)
                // (both directions give the same value but for their speeds: each lane its own)
                leaf_dt = P.CFL * dxl / (fabs(un0 / uh0) + sqrt(g * uh0));
            if (STAGE == 2)
            {
                leaf_dt = fmin(leaf_dt, __shfl_xor_sync(pair, leaf_dt, 1));
                // both lanes have read U^n mode 0 before lane 0 overwrites it
                __syncwarp(pair);
                put_un(uh0, un0, ut0, uhm, unm, utm);
                nan_seen |= (uh0 != uh0);
                if (!x) mx.add(uh0, ut0, z0);
            }
            put(uh0, un0, ut0, uhm, unm, utm);
        }
        else if (STAGE == 1) put(h0, n0, t0, pre_h, pre_n, pre_t);
        else if (INPL && mark[i] == 1)
        {
            const T uh = A.h0[a] - z0;
            put_un(uh, n0, t0, pre_h, pre_n, pre_t);
            if (!x) mx.add(uh, t0, z0);
            put(uh, n0, t0, pre_h, pre_n, pre_t);
        }
        else
        {
            const Axis<T> U = axis_of(lf, x);
            const T uh = U.h0[i], un = U.n0[i], ut = U.t0[i];
            if (!x) mx.add(uh, ut, z0);
            put(uh, un, ut, U.hm[i], U.nm[i], U.tm[i]);
        }
        if (!x && STAGE == 2 && P.dt_leaf) P.dt_leaf[i] = leaf_dt;
        dt_loc = fmin(dt_loc, leaf_dt);
    }
    if (!LIST)
    {
        const unsigned tot = __reduce_add_sync(0xffffffffu, n_wet);
        if ((threadIdx.x & 31) == 0 && tot) atomicAdd(&sc->wet[STAGE - 1], (int)tot);
    }
    if (STAGE == 2)
    {
        mx.flush(sc);
        dt_loc = warp_min(dt_loc);
        __shared__ T red[kSolverThreads / 32];
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        if (lane == 0) red[w] = dt_loc;
        __syncthreads();
        if (threadIdx.x == 0)
        {
            T m = red[0];
            for (int k = 1; k < (int)(blockDim.x >> 5); ++k) m = fmin(m, red[k]);
            atomic_min_nn(&sc->dt_min, m);
        }
        if (__syncthreads_or(nan_seen) && threadIdx.x == 0) atomicOr(&sc->status, 1);
    }
}
template <typename T, int STAGE, bool LIST>
__global__ void __launch_bounds__(kSolverThreads, kStageBlocks<T>) k_mwdg2_stage(Leaves<T> lf, Hier<T> hin, Hier<T> hout, Scalars<T>* sc,
                                                                Params<T> P, const StepArgs<T>* args, bool friction,
                                                                const int32_t* wet)
{
    k_mwdg2_stage_body<T, STAGE, LIST>(blockIdx.x, gridDim.x, lf, hin, hout, sc, P, args, friction, wet);
}

template <typename T>
__global__ void __launch_bounds__(kSolverThreads, kStageBlocks<T>) k_inplace_stage2(Leaves<T> lf, Hier<T> hr, Hier<T> hs, Scalars<T>* sc,
                                                                               Params<T> P, const StepArgs<T>* args, const int32_t* wet,
                                                                               const uint8_t* mark)
{
    k_mwdg2_stage_body<T, 2, true, true>(blockIdx.x, gridDim.x, lf, hr, hs, sc, P, args, false, wet, mark);
}

// max |h0| of the stage-2 leaf state after ghost cells (run_simulation.cu:613-620).
template <typename T>
__device__ __forceinline__ void k_stage2_maxh_body(int bid, int nb, Leaves<T> lf, Hier<T> hr, Scalars<T>* sc, Params<T> P,
                                                     const StepArgs<T>* args)
{
    const T dt = args->dt;
    const Bnd<T>& B = args->B;
    const int n = sc->n_leaves;
    T mh = T(0);
    for (int i = bid * blockDim.x + threadIdx.x; i < n; i += nb * blockDim.x)
    {
        const int a = lf.act[i];
        const T z0 = hr.s[3][0][a];
        T h0 = hr.s[0][0][a] - z0;
        int32_t nid[4];
        bool border = false;
#pragma unroll
        for (int d = 0; d < 4; ++d) { nid[d] = lf.nb[d][i]; border |= (nid[d] == -1); }
        if (border)
        {
            T gh[4], gqx[4], gqy[4];
            ghost_pass(h0, hr.s[1][0][a], hr.s[2][0][a], z0, nid, (int)lf.lvl[i], a, P, B, dt, gh, gqx, gqy);
        }
        mh = fmax(mh, fabs(h0));
    }
    T v[1] = {mh};
    T* const dst[1] = {&sc->max_h2};
    block_max_atomic<T, 1>(v, dst);
}
template <typename T>
__global__ void __launch_bounds__(256) k_stage2_maxh(Leaves<T> lf, Hier<T> hr, Scalars<T>* sc, Params<T> P,
                                                     const StepArgs<T>* args)
{
    k_stage2_maxh_body<T>(blockIdx.x, gridDim.x, lf, hr, sc, P, args);
}

// operators/fv1_update.cu:3-243 with friction and ghost cells fused. Reads the leaf and its
// neighbours from `hr` and writes the result into the leaf arrays and, at the leaf's own
// index, into `hout`, the other of two alternating hierarchy buffers (no leaf reads `hout`
// in this kernel), with the next step's maxima: the next step needs no re-insertion pass.
template <typename T>
__global__ void __launch_bounds__(kSolverThreads, sizeof(T) == 4 ? 6 : 3) k_hwfv1(Leaves<T> lf, Hier<T> hr, Hier<T> hout, Scalars<T>* sc,
                                                          Params<T> P, const StepArgs<T>* args, bool friction)
{
    const T dt = args->dt;
    const Bnd<T>& B = args->B;
    const int n = sc->n_leaves;
    T dt_loc = (sizeof(T) == 8) ? T(1.0e308) : T(3.0e38);
    bool nan_seen = false;
    StateMax<T> mx;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        const int a = lf.act[i];
        const int level = lf.lvl[i];
        int32_t nid[4];
#pragma unroll
        for (int d = 0; d < 4; ++d) nid[d] = lf.nb[d][i];
        Cell<T> own;
        load_cell(hr, a, own);
        // a NaN depth anywhere in the state (a NaN leaf with NaN neighbours is never updated)
        nan_seen |= (own.h[0] != own.h[0]);
        T gh[4], gqx[4], gqy[4];
        ghost_pass(own.h[0], own.qx[0], own.qy[0], own.z[0], nid, level, a, P, B, dt, gh, gqx, gqy);
        bool fric = false;
        if (friction)
        {
            const T h = own.h[0];
            const bool below_depth = (h < P.tol_h);
            const T ux = below_depth ? T(0.0) : own.qx[0] / h;
            const T uy = below_depth ? T(0.0) : own.qy[0] / h;
            const bool below_speed = (fabs(ux) < P.tol_s && fabs(uy) < P.tol_s);
            if (below_depth || below_speed) { own.qx[0] = T(0.0); own.qy[0] = T(0.0); }
            fric = !(below_depth || below_speed);
            if (fric) friction_cell<T>(own, P, dt);
        }
        T nbh[4];
#pragma unroll
        for (int d = 0; d < 4; ++d) nbh[d] = (nid[d] != -1) ? hr.s[0][0][nid[d]] - hr.s[3][0][nid[d]] : gh[d];
        if (own.h[0] < P.tol_h && nbh[0] < P.tol_h && nbh[1] < P.tol_h && nbh[2] < P.tol_h && nbh[3] < P.tol_h)
        {
            // dry leaf: not updated (fv1_update.cu:27-46), discharge zeroed by friction if enabled
            lf.un[0][i] = own.h[0];
            lf.un[3][i] = own.qx[0];
            lf.un[6][i] = own.qy[0];
            put_leaf_fv1(hout, a, own.h[0], own.qx[0], own.qy[0], own.z[0], mx);
            if (P.dt_leaf) P.dt_leaf[i] = P.initial_tstep;
            dt_loc = fmin(dt_loc, P.initial_tstep);
            continue;
        }
        V3<T> U[4];
        T zn[4];
#pragma unroll
        for (int d = 0; d < 4; ++d)
        {
            Cell<T> c;
            if (nid[d] != -1) load_cell(hr, nid[d], c);
            else { c.h[0] = gh[d]; c.qx[0] = gqx[d]; c.qy[0] = gqy[d]; c.z[0] = own.z[0]; }
            if (fric) friction_cell<T>(c, P, dt);
            U[d] = V3<T>{c.h[0], c.qx[0], c.qy[0]};
            zn[d] = c.z[0];
        }
        T h = own.h[0], qx = own.qx[0], qy = own.qy[0];
        const bool wet = (h >= P.tol_h || U[0].h >= P.tol_h || U[1].h >= P.tol_h || U[2].h >= P.tol_h || U[3].h >= P.tol_h);
        T leaf_dt = P.initial_tstep;
        if (wet)
        {
            const T dxl = P.dx * (1 << (P.L - level));
            const T z = own.z[0];
            const T eta_loc = h + z;
            const T zin = fmax(z, zn[0]), zie = fmax(z, zn[1]), zis = fmax(z, zn[2]), ziw = fmax(z, zn[3]);
            const V3<T> Uc = {h, qx, qy};
            const V3<T> Usnn = star(Uc, z, zin, P.tol_h), Usnp = star(U[0], zn[0], zin, P.tol_h);
            const V3<T> F_n = flux_hll_y(Usnn, Usnp, P.tol_h, P.g);
            const V3<T> Usen = star(Uc, z, zie, P.tol_h), Usep = star(U[1], zn[1], zie, P.tol_h);
            const V3<T> F_e = flux_hll_x(Usen, Usep, P.tol_h, P.g);
            const V3<T> Ussn = star(U[2], zn[2], zis, P.tol_h), Ussp = star(Uc, z, zis, P.tol_h);
            const V3<T> F_s = flux_hll_y(Ussn, Ussp, P.tol_h, P.g);
            const V3<T> Uswn = star(U[3], zn[3], ziw, P.tol_h), Uswp = star(Uc, z, ziw, P.tol_h);
            const V3<T> F_w = flux_hll_x(Uswn, Uswp, P.tol_h, P.g);
            // operators/get_bed_src.cuh:7-44
            const T zsw = ziw - fmax(T(0.0), -(eta_loc - ziw));
            const T zse = zie - fmax(T(0.0), -(eta_loc - zie));
            const T bx = P.g * T(0.5) * (Uswp.h + Usen.h) * (zse - zsw) / dxl;
            const T zss = zis - fmax(T(0.0), -(eta_loc - zis));
            const T zsn = zin - fmax(T(0.0), -(eta_loc - zin));
            const T by = P.g * T(0.5) * (Ussp.h + Usnn.h) * (zsn - zss) / dxl;
            h = h - dt * (F_e.h - F_w.h) / dxl;
            qx = qx - dt * ((F_e.qx - F_w.qx) / dxl + bx);
            qy = qy - dt * (F_e.qy - F_w.qy) / dxl;
            h = h - dt * (F_n.h - F_s.h) / dxl;
            qx = qx - dt * (F_n.qx - F_s.qx) / dxl;
            qy = qy - dt * ((F_n.qy - F_s.qy) / dxl + by);
            const bool below_depth = (h < P.tol_h);
            const bool below_disch = (fabs(qx) < P.tol_q && fabs(qy) < P.tol_q);
            if (below_depth || below_disch) { qx = T(0.0); qy = T(0.0); }
            if (!below_depth)
            {
                const T ux = qx / h, uy = qy / h;
                const T dtx = P.CFL * dxl / (fabs(ux) + sqrt(P.g * h));
                const T dty = P.CFL * dxl / (fabs(uy) + sqrt(P.g * h));
                leaf_dt = fmin(dtx, dty);
            }
            nan_seen |= (h != h);
        }
        lf.un[0][i] = h;
        lf.un[3][i] = qx;
        lf.un[6][i] = qy;
        put_leaf_fv1(hout, a, h, qx, qy, own.z[0], mx);
        if (P.dt_leaf) P.dt_leaf[i] = leaf_dt;
        dt_loc = fmin(dt_loc, leaf_dt);
    }
    mx.flush(sc);
    dt_loc = warp_min(dt_loc);
    __shared__ T red[kSolverThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) red[w] = dt_loc;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        T m = red[0];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) m = fmin(m, red[k]);
        atomic_min_nn(&sc->dt_min, m);
    }
    if (__syncthreads_or(nan_seen) && threadIdx.x == 0) atomicOr(&sc->status, 1);
}

// Leaf containing each finest cell code (search over the leaves' Z-order starts) and its
// depth eta0 - z0, discharges and bed (output/project_assem_sol.cu:3-77). One warp per
// point: lane j probes position lo + (j + 1) * step of the range [lo, hi] that holds the
// answer (the last leaf whose start is <= c; starts increase along the leaf list), and the
// ballot of the probes narrows the range 32-fold per round (two rounds for a tile's leaves).
// tile_offsets (the scanned leaf counts of the 4^5-cell tiles, ntiles of them; null before
// the first step) narrow the start: leaves are in Z order, so the leaf holding finest cell
// c is among the leaves of tile c >> 10, or is the last leaf before them when a coarser leaf
// covers the whole tile.
template <typename T>
__device__ __forceinline__ void k_sample_points_body(Leaves<T> lf, Hier<T> hr, Scalars<T>* sc, int L, const int32_t* codes, int np,
                                const int32_t* tile_offsets, int ntiles, T* out, const uint8_t* mark = nullptr,
                                const uint8_t* mark2 = nullptr)
{
    const int k = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (k >= np) return;   // the whole warp
    const int n = sc->n_leaves;
    const int c = codes[k];
    int lo = 0, hi = n - 1;
    if (tile_offsets)
    {
        const int t = c >> (2 * kTileDepth);
        lo = tile_offsets[t];
        hi = (t + 1 < ntiles ? tile_offsets[t + 1] : n) - 1;
        if (hi < lo) lo = hi = lo - 1;
    }
    while (lo < hi)
    {
        const int step = (hi - lo + 31) / 32;
        const int pos = min(hi, lo + (lane + 1) * step);
        const int l = lf.lvl[pos];
        const bool le = ((lf.act[pos] - lvl_idx(l)) << (2 * (L - l))) <= c;
        const int t = __popc(__ballot_sync(0xffffffffu, le));   // probes 0..t-1 start at or before c
        const int nlo = t == 0 ? lo : min(hi, lo + t * step);
        const int nhi = t == 32 ? hi : min(hi, lo + (t + 1) * step) - 1;
        lo = nlo;
        hi = nhi;
    }
    if (lane != 0) return;
    const int a = lf.act[lo];
    const T z0 = hr.s[3][0][a];
    // mark, mark2 (in-place steps): a leaf that stood through both stages has its state in hr
    const bool stood = mark && mark[lo] == 1 && (mark2[lo] & 1);
    const T eta = stood ? hr.s[0][0][a] : lf.un[0][lo] + z0;
    out[4 * k + 0] = eta - z0;
    out[4 * k + 1] = stood ? hr.s[1][0][a] : lf.un[3][lo];
    out[4 * k + 2] = stood ? hr.s[2][0][a] : lf.un[6][lo];
    out[4 * k + 3] = z0;
}
template <typename T>
__global__ void k_sample_points(Leaves<T> lf, Hier<T> hr, Scalars<T>* sc, int L, const int32_t* codes, int np,
                                const int32_t* tile_offsets, int ntiles, T* out, const uint8_t* mark = nullptr,
                                const uint8_t* mark2 = nullptr)
{
    k_sample_points_body<T>(lf, hr, sc, L, codes, np, tile_offsets, ntiles, out, mark, mark2);
}

// Leaf state with the bed coefficients gathered from the hierarchy, 12 rows of n values.
// Water volume of the leaf state in cell units: sum over leaves of h0 x 4^(L - level), each
// term exact in FP64 (a power-of-two scaling of the leaf's depth) and summed in FP64 whatever
// the state's precision; times dx^2 it is the volume in m^3. One atomic per block.
template <typename T> __global__ void __launch_bounds__(256) k_volume(Leaves<T> lf, const Scalars<T>* sc, int L, double* out)
{
    const int n = sc->n_leaves;
    double v = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        v += ldexp((double)lf.un[0][i], 2 * (L - (int)lf.lvl[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __shared__ double red[8];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        atomicAdd(out, t);
    }
}

template <typename T> __global__ void k_gather_state(Leaves<T> lf, Hier<T> hr, Scalars<T>* sc, bool mw, double* out)
{
    const int n = sc->n_leaves;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        const int a = lf.act[i];
        const size_t N = (size_t)n;
        out[0 * N + i] = lf.un[0][i];
        out[1 * N + i] = lf.un[3][i];
        out[2 * N + i] = lf.un[6][i];
        out[3 * N + i] = hr.s[3][0][a];
        out[4 * N + i] = mw ? (double)lf.un[1][i] : 0.0;
        out[5 * N + i] = mw ? (double)lf.un[4][i] : 0.0;
        out[6 * N + i] = mw ? (double)lf.un[7][i] : 0.0;
        out[7 * N + i] = mw ? (double)hr.s[3][1][a] : 0.0;
        out[8 * N + i] = mw ? (double)lf.un[2][i] : 0.0;
        out[9 * N + i] = mw ? (double)lf.un[5][i] : 0.0;
        out[10 * N + i] = mw ? (double)lf.un[8][i] : 0.0;
        out[11 * N + i] = mw ? (double)hr.s[3][2][a] : 0.0;
    }
}

} // namespace mw
