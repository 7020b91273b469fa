// vphys_tracers.cuh -- implicit vertical diffusion of every tracer with the KPP
// non-local tendency fused into the store (rdb_ocean_vdiff.F90:1107-1414,
// rdb_ocean_vmix.F90:1605-1714).
//
// One thread per cell column; a block's columns are consecutive in i,
// so every per-level access of a warp is one coalesced 256-B segment.
//
// * Only the column's live span [k_lo, k_hi] (first live layer from the bed,
//   first live layer from the surface) is solved: every row outside it is an
//   identity row of the reference's matrix (both couplings gated to zero by
//   H_VANISHED), whose solution is its input, its budget increment zero and
//   its non-local deposit refused -- the values are unchanged (up to the sign
//   of a zero), so those cells are neither read nor written.  Land columns
//   cost one scan of h.
// * The matrix is factorised once per diffusivity (kt, and ks when it differs)
//   in the same upward pass that forward-sweeps every tracer.  The pivots'
//   c' live in shared memory; the forward-swept right-hand sides are written
//   in place into the tracer arrays with an L2 evict_last hint and read back
//   by the downward pass, so the round trip stays in L2 and HBM sees each
//   tracer value read once and written once.
// * Loads are issued a block of levels ahead of the arithmetic, and a block's
//   quotients do not branch (quot, vphys_device.cuh), so the levels and the
//   tracers of a block overlap under the serial Thomas recurrence, whose
//   latency at eleven warps an SM is the bound (issue 42 %, DRAM 40 %).
// * Handles with more than five tracers are solved in even groups of at most
//   five, each with its own factorisation (shallow columns in one).
#pragma once
#include "vphys_device.cuh"
#include "vphys_kernels.cuh"

// Blocks of 64 columns, two levels a block upward and downward with the
// deposit, four without it, at most five tracers a thread (1440x1080x75 with 4
// tracers / 600x451x75 with 10, the fused solve): 1.83 / 0.87 ms.  128 columns
// 1.93 / 1.00, 32 1.89 / 0.99; one level upward 2.56 / 1.17, three 1.86 / 0.89;
// eight levels without the deposit 2.16 / 1.00; four tracers a thread - / 0.97.
// (All sixteen tracers in one thread, divisions branching: 3.54 / 1.65.)
#ifndef VPHYS_TR_THREADS
#define VPHYS_TR_THREADS 64
#endif
#ifndef VPHYS_TR_U
#define VPHYS_TR_U 2
#endif
#ifndef VPHYS_TR_UB
#define VPHYS_TR_UB 2
#endif
#ifndef VPHYS_TR_UP
#define VPHYS_TR_UP 4
#endif
#ifndef VPHYS_TR_GROUP
#define VPHYS_TR_GROUP 5
#endif

namespace vphys {

// The columns of one warp: column (i, j) on this lane, `tid` its slot in the
// block's shared memory of `bs` columns; the tracers t0 .. t0 + nt - 1 (nt < 0:
// all).  CI: with the diffusion, the compensated column content before it
// (terms bottom-up, in the upward pass) and after it (top-down, in the
// downward pass) into p.content_old / _new.
template <int NTR, bool TWO, bool DEF, bool CI = false>
__device__ __forceinline__ void tracer_columns(const Params &p, double dt, int diffuse, int nonlocal, int i, int j,
                                               double *smem, int tid, int bs, int t0 = 0, int nt = -1)
{
    constexpr bool WIDE = NTR > VPHYS_TR_GROUP;         // shallow columns (tracer_groups): one level a block
    constexpr int TR_U = WIDE ? 1 : VPHYS_TR_U;         // levels per block of the upward pass
    constexpr int TR_UB = WIDE ? 1 : VPHYS_TR_UB;       // levels per load block of the downward pass
    constexpr int TR_UP = WIDE ? 1 : VPHYS_TR_UP;       // the same below the boundary layer
    constexpr int TR_US = 8;                            // levels per load block of the span scans
    vphys_config cd = p.cfg;   // DEF: the default knobs folded in (is_default_tracer_knobs)
    if (DEF) default_tracer_knobs(cd);
    const vphys_config &c = cd;
    const int nx = p.nx, nz = p.nz, ntr = nt < 0 ? p.ntr : nt;
    const size_t P = p.plane;
    const bool in_grid = i < nx;
    const size_t col = (size_t)(in_grid ? i : 0) + (size_t)nx * j;
    const double *__restrict__ hp = p.h + col;
    const int iT = c.idx_temperature - t0, iS = c.idx_salinity - t0, iPS = c.idx_pseudo_salt - t0;
    double *cpA = smem + tid;                       // cpA[(k-1)*bs]
    double *cpB = smem + (size_t)nz * bs + tid;     // only when TWO
    const unsigned long long pol_keep = l2_policy_evict_last();
    const unsigned long long pol_once = l2_policy_evict_first();

    // ---- this column's live span; rows outside it are identity rows.  The
    //      scans read TR_US levels per wait, so a land column costs 10 waits on
    //      memory at nz = 75, not 75 ----
    int k_lo = 0, k_hi = 0;
    double h_lo = 0.0, h_hi = 0.0;
    if (in_grid) {
        for (int k0 = 1; k0 <= nz && k_lo == 0; k0 += TR_US) {
            double hv[TR_US];
#pragma unroll
            for (int u = 0; u < TR_US; ++u) hv[u] = (k0 + u <= nz) ? __ldg(hp + P * (size_t)(k0 + u - 1)) : 0.0;
#pragma unroll
            for (int u = TR_US - 1; u >= 0; --u)
                if (hv[u] > H_VANISHED) {
                    k_lo = k0 + u;
                    h_lo = hv[u];
                }
        }
        if (k_lo > 0) {
            for (int k0 = nz; k0 >= k_lo && k_hi == 0; k0 -= TR_US) {
                double hv[TR_US];
#pragma unroll
                for (int u = 0; u < TR_US; ++u) hv[u] = (k0 - u >= k_lo) ? __ldg(hp + P * (size_t)(k0 - u - 1)) : 0.0;
#pragma unroll
                for (int u = TR_US - 1; u >= 0; --u)
                    if (hv[u] > H_VANISHED) {
                        k_hi = k0 - u;
                        h_hi = hv[u];
                    }
            }
        }
    }
    const bool live = k_lo > 0;
    const unsigned rows = live ? (unsigned)(k_hi - k_lo + 1) : 0u;   // level k is in the span: (unsigned)(k - k_lo) < rows
    // the warp sweeps the union of its lanes' spans with a uniform k, so its
    // loads stay coalesced and the row-type branches stay uniform; a lane
    // outside its own span is predicated off (no load, no store)
    const unsigned full = 0xffffffffu;
    const int w_lo = __reduce_min_sync(full, live ? k_lo : 0x7fffffff);
    const int w_hi = __reduce_max_sync(full, live ? k_hi : 0);
    if (w_hi == 0) {   // no live layer anywhere in this warp
        if (CI && diffuse && in_grid)
            for (int t = 0; t < ntr; ++t)
                p.content_old[col + P * (size_t)(t0 + t)] = p.content_new[col + P * (size_t)(t0 + t)] = 0.0;
        return;
    }
    double c_old[NTR], e_old[NTR], c_new[NTR], e_new[NTR];   // CI: Neumaier sums and their compensations
#pragma unroll
    for (int t = 0; t < NTR; ++t) c_old[t] = e_old[t] = c_new[t] = e_new[t] = 0.0;

    double *trc[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t) trc[t] = (t < ntr) ? p.tr[t0 + t] + col : nullptr;
    // With heat/salt budgets the reference needs h*c_new - h*c_old, so the
    // forward-swept values of T and S go to a scratch plane instead of over
    // the input (rbuf); every other tracer is swept in place.
    double *heat = (c.budgets && diffuse && iT >= 0 && iT < ntr) ? p.heat_budget + col : nullptr;
    double *salt = (c.budgets && diffuse && iS >= 0 && iS < ntr) ? p.salt_budget + col : nullptr;
    double *rbuf[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t) {
        rbuf[t] = trc[t];
        if (t < ntr && heat && t == iT) rbuf[t] = p.budget_scratch + col;
        if (t < ntr && salt && t == iS) rbuf[t] = p.budget_scratch + P * (size_t)nz + col;
    }

    if (diffuse) {
        // ---- upward pass: rows, factorisation, forward sweep of every tracer.
        //      Rows are branch-free: outside a lane's span h is taken as 0, which
        //      gates both couplings of build_factorize_tracer_matrix's row
        //      (rdb_ocean_vdiff.F90:1285-1341) off, and nothing is stored ----
        const double *__restrict__ KA = p.kt + col;
        const double *__restrict__ KB = p.ks + col;
        double h_c = (k_lo == w_lo) ? h_lo : 0.0;
        double cpA_prev = 0.0, cpB_prev = 0.0, beA = 0.0, beB = 0.0;   // be*: the row's coupling to the row below
        double r_prev[NTR];
#pragma unroll
        for (int t = 0; t < NTR; ++t) r_prev[t] = 0.0;
        // row k reads its tracers and h, K one level up; the loads of block
        // k0 + TR_U are issued before block k0 is computed (two register
        // buffers; the block's stores go to its own levels).  Loading into one
        // set of registers as the block frees them saves the copies but leaves
        // the latency uncovered: 1.99 against 1.83 ms at 1440x1080x75.
        auto load_up = [&](int k0, double (&xs_)[TR_U][NTR], double (&hps_)[TR_U], double (&kap_)[TR_U],
                           double (&kbp_)[TR_U]) {
#pragma unroll
            for (int u = 0; u < TR_U; ++u) {
                const bool act = (unsigned)(k0 + u - k_lo) < rows, up = (unsigned)(k0 + u + 1 - k_lo) < rows;
                const size_t off = P * (size_t)(k0 + u - 1);
                hps_[u] = up ? __ldg(hp + off + P) : 0.0;
                kap_[u] = up ? ld_hint(KA + off + P, pol_once) : 0.0;
                kbp_[u] = (TWO && up) ? ld_hint(KB + off + P, pol_once) : 0.0;
#pragma unroll
                for (int t = 0; t < NTR; ++t) xs_[u][t] = (act && t < ntr) ? trc[t][off] : 0.0;
            }
        };
        double xs[TR_U][NTR], hps[TR_U], kap[TR_U], kbp[TR_U];
        load_up(w_lo, xs, hps, kap, kbp);
        for (int k0 = w_lo; k0 <= w_hi; k0 += TR_U) {
            double xs_n[TR_U][NTR], hps_n[TR_U], kap_n[TR_U], kbp_n[TR_U];
            load_up(k0 + TR_U, xs_n, hps_n, kap_n, kbp_n);
            // (1) the couplings of the interfaces above the block's rows: alA of
            // row k and beA of row k + 1, every quotient of the block free of branches
            double alA[TR_U], bnA[TR_U], alB[TR_U], bnB[TR_U];
            Ranges rc;
            auto couple = [&](auto div) {
                double hl = h_c;
#pragma unroll
                for (int u = 0; u < TR_U; ++u) {
                    const double hc = fmx(hl, H_VANISHED), hu = fmx(hps[u], H_VANISHED);
                    const double dz = face_thick(hc, hu, c.use_harmonic);
                    const bool both = hl > H_VANISHED && hps[u] > H_VANISHED;
                    const double dl = hc * dz, du = hu * dz, nA = dt * kap[u];
                    const double a = div(nA, dl), b = div(nA, du);
                    alA[u] = both ? a : 0.0;
                    bnA[u] = both ? b : 0.0;
                    if (TWO) {
                        const double nB = dt * kbp[u];
                        const double aB = div(nB, dl), bB = div(nB, du);
                        alB[u] = both ? aB : 0.0;
                        bnB[u] = both ? bB : 0.0;
                    }
                    hl = hps[u];
                }
            };
            couple([&](double n, double d) {
                rc.num(n);
                rc.den(d);
                return quot(n, d, rcp2(d));
            });
            if (!rc.ok()) couple([](double n, double d) { return xdiv(n, d); });
            // (2) the recurrences: c' and every tracer's forward-swept value
            const double cA0 = cpA_prev, cB0 = cpB_prev, beA0 = beA, beB0 = beB;
            double rr[TR_U][NTR], cpa[TR_U], cpb[TR_U];
            Ranges rg;
#pragma unroll
            for (int u = 0; u < TR_U; ++u) {
                const double dA = (1.0 + alA[u] + beA) + beA * cpA_prev;
                const double yA = rcp2(dA);
                const double nA = -alA[u];
                rg.den(dA);
                rg.num(nA);
                cpA_prev = quot(nA, dA, yA);
                cpa[u] = cpA_prev;
                double dB = dA, yB = yA;
                if (TWO) {
                    dB = (1.0 + alB[u] + beB) + beB * cpB_prev;
                    yB = rcp2(dB);
                    const double nB = -alB[u];
                    rg.den(dB);
                    rg.num(nB);
                    cpB_prev = quot(nB, dB, yB);
                    cpb[u] = cpB_prev;
                }
#pragma unroll
                for (int t = 0; t < NTR; ++t) {
                    const bool useA = !TWO || (t == iT);
                    const double num = xs[u][t] + (useA ? beA : beB) * ((u == 0) ? r_prev[t] : rr[u > 0 ? u - 1 : 0][t]);
                    rg.num(num);
                    rr[u][t] = quot(num, useA ? dA : dB, useA ? yA : yB);
                }
                beA = bnA[u];
                if (TWO) beB = bnB[u];
            }
            if (!rg.ok()) {
                cpA_prev = cA0;
                cpB_prev = cB0;
                beA = beA0;
                beB = beB0;
#pragma unroll
                for (int u = 0; u < TR_U; ++u) {
                    const Rcp denA = rcp_of((1.0 + alA[u] + beA) + beA * cpA_prev);
                    cpA_prev = qdiv(-alA[u], denA);
                    cpa[u] = cpA_prev;
                    Rcp denB = denA;
                    if (TWO) {
                        denB = rcp_of((1.0 + alB[u] + beB) + beB * cpB_prev);
                        cpB_prev = qdiv(-alB[u], denB);
                        cpb[u] = cpB_prev;
                    }
#pragma unroll
                    for (int t = 0; t < NTR; ++t) {
                        const bool useA = !TWO || (t == iT);
                        rr[u][t] = qdiv(xs[u][t] + (useA ? beA : beB) * ((u == 0) ? r_prev[t] : rr[u > 0 ? u - 1 : 0][t]),
                                        useA ? denA : denB);
                    }
                    beA = bnA[u];
                    if (TWO) beB = bnB[u];
                }
            }
#pragma unroll
            for (int u = 0; u < TR_U; ++u) {
                const int k = k0 + u;
                if ((unsigned)(k - k_lo) < rows) {
                    const size_t off = P * (size_t)(k - 1);
                    cpA[(size_t)(k - 1) * bs] = cpa[u];
                    if (TWO) cpB[(size_t)(k - 1) * bs] = cpb[u];
#pragma unroll
                    for (int t = 0; t < NTR; ++t)
                        if (t < ntr) {
                            st_hint(rbuf[t] + off, rr[u][t], pol_keep);
                            if (CI) neumaier_add(c_old[t], e_old[t], h_c * xs[u][t]);
                        }
                }
                h_c = hps[u];
            }
#pragma unroll
            for (int t = 0; t < NTR; ++t) r_prev[t] = rr[TR_U - 1][t];
#pragma unroll
            for (int u = 0; u < TR_U; ++u) {
                hps[u] = hps_n[u];
                kap[u] = kap_n[u];
                kbp[u] = kbp_n[u];
#pragma unroll
                for (int t = 0; t < NTR; ++t) xs[u][t] = xs_n[u][t];
            }
        }
    }

    // ---- non-local column scalars, recomputed exactly as KPP pass 2 ----
    const bool do_nl = nonlocal && c.use_kpp;
    bool nl = do_nl && live;
    double h_b = 0.0, q_T_kin = 0.0, q_S_kin = 0.0;
    if (nl) {
        const double rho0 = c.rho0;
        h_b = p.bl_depth[col];
        const double u_star = sqrt(xdiv(p.stress_mag[col], rho0));
        // the heat flux pass 2 charged (shortwave: what passes h_b, or the
        // surface layer k_hi)
        q_T_kin = kpp_q_t_kin(c, p.q_heat[col], p.sw_src + col, p.sw_kappa, col, p.plane, h_b, h_hi);
        q_S_kin = xdiv(p.q_salt[col], rho0);
        // with "eos" coefficients or shortwave B0 is the assembly's (pass 2
        // stored it before the solve changed the surface T and S); otherwise
        // the same number recomputed
        const double B_0 = (c.buoyancy_coeffs || c.sw_pen_frac != 0.0)
                               ? p.b0[col]
                               : (GRAVITY / rho0) * (c.alpha_T * q_T_kin - c.beta_S * q_S_kin);
        const double wstar3 = fmx(0.0, -B_0) * h_b;
        const double w_star = sm_cbrt(wstar3);
        const double w_s = sqrt(u_star * u_star + w_star * w_star);
        nl = (h_b > 0.0 && w_s > 0.0 && B_0 < 0.0);
    }

    // ---- downward pass: back-substitution, budgets, non-local deposit and
    //      the store (the reference's k_sfc is this column's k_hi) ----
    double x_above[NTR];
#pragma unroll
    for (int t = 0; t < NTR; ++t) x_above[t] = 0.0;
    double gT_above = 0.0, gS_above = 0.0;
    double d_run = 0.0;
    double h_c = h_hi, h_a = 0.0;   // layer above k_hi is vanished: its flux is closed
    // sigma = d_run / h_b with one reciprocal per column (qdiv: the quotient bit for bit)
    const Rcp r_hb = rcp_of(nl ? h_b : 1.0);
    // the loads of block k0 - TR_UB are issued before block k0 is computed
    auto load_down = [&](int k0, double (&rs_)[TR_UB][NTR], double (&hbs_)[TR_UB]) {
#pragma unroll
        for (int u = 0; u < TR_UB; ++u) {
            const int k = k0 - u;
            const bool act = (unsigned)(k - k_lo) < rows;
            const size_t off = P * (size_t)(k - 1);
            hbs_[u] = (act && k > 1) ? __ldg(hp + off - P) : 0.0;
#pragma unroll
            for (int t = 0; t < NTR; ++t)
                rs_[u][t] = (act && t < ntr && (diffuse || t == iT || t == iS || t == iPS))
                                ? ld_hint((diffuse ? rbuf[t] : trc[t]) + off, pol_keep)
                                : 0.0;
        }
    };
    // Below the boundary layer every term of the deposit is an exact zero: once
    // no lane of the warp is inside (its last flux, one level down, spent),
    // the walk goes on without it and without h.  Budgets and the column
    // content read h to the bed.
    const bool to_bed = heat || salt || (CI && diffuse);
    int k0 = w_hi;
    double rs[TR_UB][NTR], hbs[TR_UB];
    load_down(w_hi, rs, hbs);
    for (; k0 >= w_lo; k0 -= TR_UB) {
        if (!to_bed) {
            const bool in_bl = nl && (d_run < h_b || gT_above != 0.0 || gS_above != 0.0);
            if (!__reduce_max_sync(full, in_bl ? 1 : 0)) break;
        }
        double rs_n[TR_UB][NTR], hbs_n[TR_UB];
        load_down(k0 - TR_UB, rs_n, hbs_n);
#pragma unroll
        for (int u = 0; u < TR_UB; ++u) {
            const int k = k0 - u;
            if (k < w_lo) break;
            const bool act = (unsigned)(k - k_lo) < rows;
            if (act) {
                const size_t off = P * (size_t)(k - 1);
                const double h_bl = hbs[u];
                double gT = 0.0, gS = 0.0;
                if (nl) {
                    d_run = d_run + h_c;
                    if (k > 1 && d_run < h_b) {
                        const double sigma = qdiv(d_run, r_hb);
                        const double g_shape = sigma * (1.0 - sigma) * (1.0 - sigma);
                        const double gamma_factor = c.cs_nonlocal * g_shape;
                        gT = gamma_factor * q_T_kin;
                        gS = gamma_factor * q_S_kin;
                    }
                }
                double fT = 0.0, fS = 0.0;
                if (do_nl) {
                    double fT_up = 0.0, fT_dn = 0.0, fS_up = 0.0, fS_dn = 0.0;
                    if (k < nz) {
                        fT_up = nonlocal_face_flux(gT_above, h_c, h_a);
                        fS_up = nonlocal_face_flux(gS_above, h_c, h_a);
                    }
                    if (k > 1) {
                        fT_dn = nonlocal_face_flux(gT, h_bl, h_c);
                        fS_dn = nonlocal_face_flux(gS, h_bl, h_c);
                    }
                    fT = dt * (fT_up - fT_dn);
                    fS = dt * (fS_up - fS_dn);
                }
                // conc_add_source's quotients src / (h + H_DIV_EPS), one reciprocal for
                // the layer (salinity and pseudo-salt share fS); a zero source adds
                // itself, as xdiv(+-0, b > 0) = +-0
                double incT = fT, incS = fS;
                if (do_nl && (fT != 0.0 || fS != 0.0)) {
                    const Rcp r_h = rcp_of(h_c + H_DIV_EPS);
                    if (fT != 0.0) incT = qdiv(fT, r_h);
                    if (fS != 0.0) incS = qdiv(fS, r_h);
                }
#pragma unroll
                for (int t = 0; t < NTR; ++t) {
                    if (t < ntr && (diffuse || t == iT || t == iS || t == iPS)) {
                        double x = rs[u][t];
                        if (diffuse) {
                            const bool useA = !TWO || (t == iT);
                            const double cpk = useA ? cpA[(size_t)(k - 1) * bs] : cpB[(size_t)(k - 1) * bs];
                            x = x - cpk * x_above[t];   // x_above = 0 at k_hi: the top row
                            x_above[t] = x;
                            if ((t == iT && heat) || (t == iS && salt)) {
                                double *bud = (t == iT) ? heat : salt;
                                const double x_old = trc[t][off];
                                const double p_new = h_c * x, p_old = h_c * x_old;
                                bud[off] = bud[off] + (p_new - p_old);
                            }
                        }
                        if (do_nl && h_c > H_VANISHED) {
                            if (t == iT) x = x + incT;
                            else if (t == iS || t == iPS) x = x + incS;
                        }
                        if (CI && diffuse) neumaier_add(c_new[t], e_new[t], h_c * x);
                        trc[t][off] = x;
                    }
                }
                gT_above = gT;
                gS_above = gS;
                h_a = h_c;
                h_c = h_bl;
            }
        }
#pragma unroll
        for (int u = 0; u < TR_UB; ++u) {
            hbs[u] = hbs_n[u];
#pragma unroll
            for (int t = 0; t < NTR; ++t) rs[u][t] = rs_n[u][t];
        }
    }
    if (diffuse && k0 >= w_lo) {
        auto load_plain = [&](int kt, double (&r_)[TR_UP][NTR]) {
#pragma unroll
            for (int u = 0; u < TR_UP; ++u) {
                const int k = kt - u;
                const bool act = (unsigned)(k - k_lo) < rows;
#pragma unroll
                for (int t = 0; t < NTR; ++t)
                    r_[u][t] = (act && t < ntr) ? ld_hint(trc[t] + P * (size_t)(k - 1), pol_keep) : 0.0;
            }
        };
        double r[TR_UP][NTR];
        load_plain(k0, r);
        for (; k0 >= w_lo; k0 -= TR_UP) {
            double r_n[TR_UP][NTR];
            load_plain(k0 - TR_UP, r_n);
#pragma unroll
            for (int u = 0; u < TR_UP; ++u) {
                const int k = k0 - u;
                if ((unsigned)(k - k_lo) < rows) {
                    const double cA = cpA[(size_t)(k - 1) * bs], cB = TWO ? cpB[(size_t)(k - 1) * bs] : cA;
#pragma unroll
                    for (int t = 0; t < NTR; ++t)
                        if (t < ntr) {
                            const double x = r[u][t] - ((!TWO || t == iT) ? cA : cB) * x_above[t];
                            x_above[t] = x;
                            trc[t][P * (size_t)(k - 1)] = x;
                        }
                }
            }
#pragma unroll
            for (int u = 0; u < TR_UP; ++u)
#pragma unroll
                for (int t = 0; t < NTR; ++t) r[u][t] = r_n[u][t];
        }
    }
    if (CI && diffuse && in_grid) {
#pragma unroll
        for (int t = 0; t < NTR; ++t)
            if (t < ntr) {
                p.content_old[col + P * (size_t)(t0 + t)] = c_old[t] + e_old[t];
                p.content_new[col + P * (size_t)(t0 + t)] = c_new[t] + e_new[t];
            }
    }
}

// blockIdx.x: the tracer groups of a column block side by side (so h and K,
// read by each, come from L2 after the first), group g holding
// ntr / ngroups tracers and one more in the first ntr % ngroups groups.
template <int NTR, bool TWO, bool DEF, bool CI>
__global__ void __launch_bounds__(128) k_tracers(const Params p, double dt, int diffuse, int nonlocal, int ngroups)
{
    extern __shared__ double smem[];
    const int g = blockIdx.x % ngroups, b = blockIdx.x / ngroups;
    const int nt = p.ntr / ngroups, more = p.ntr % ngroups;
    tracer_columns<NTR, TWO, DEF, CI>(p, dt, diffuse, nonlocal, b * blockDim.x + threadIdx.x, blockIdx.y, smem,
                                      threadIdx.x, blockDim.x, g * nt + min(g, more), nt + (g < more ? 1 : 0));
}

template <int NTR, bool TWO>
static void launch_tracers_n(const Params &p, double dt, bool diffuse, bool nonlocal, int ngroups, cudaStream_t stream)
{
    // two factorisations keep two c' arrays: halve the block to stay within
    // the 227 KB of shared memory per block at nz = VPHYS_NZ_MAX
    const int bs = TWO ? VPHYS_TR_THREADS / 2 : VPHYS_TR_THREADS;
    const size_t smem = (size_t)p.nz * bs * sizeof(double) * (TWO ? 2 : 1);
    static bool attr_set = false;
    if (!attr_set) {
        const int mx = (int)((size_t)VPHYS_NZ_MAX * bs * sizeof(double) * (TWO ? 2 : 1));
        cudaFuncSetAttribute(k_tracers<NTR, TWO, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
        cudaFuncSetAttribute(k_tracers<NTR, TWO, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
        cudaFuncSetAttribute(k_tracers<NTR, TWO, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
        attr_set = true;
    }
    dim3 grid((p.nx + bs - 1) / bs * ngroups, p.ny);
    if (is_default_tracer_knobs(p.cfg))
        k_tracers<NTR, TWO, true, false><<<grid, bs, smem, stream>>>(p, dt, diffuse ? 1 : 0, nonlocal ? 1 : 0, ngroups);
    else if (p.content_old && diffuse)
        k_tracers<NTR, TWO, false, true><<<grid, bs, smem, stream>>>(p, dt, 1, nonlocal ? 1 : 0, ngroups);
    else
        k_tracers<NTR, TWO, false, false><<<grid, bs, smem, stream>>>(p, dt, diffuse ? 1 : 0, nonlocal ? 1 : 0, ngroups);
}

}  // namespace vphys
