// Adjoint of the thermal-water transport part of one substep, the companion of
// bk_substep_adjoint: the forward transport phase (physics/thermal_water.py:77-190 -- surface
// areas, scalar P2G, diffusion) and the scalar G2P with its water stress and mass
// (thermal_water.py:193-229, 248-253) and, in gas mode, its local gas source and gas-pressure
// stress (thermal_water.py:232-245, physics/materials/gas.py:16-35) reversed, given the substep's
// grid with its transport fields
// kept (BkSubstepParams.keep_transport_fields) and the adjoints the mechanics adjoint produced for
// the stress, particle mass and material temperature that P2G and the return map used.
//
// Order, all per substep:
//   prepare          T_mat = T + sum w dT, mass = dry + W', stress tau + J (p_amb - p) I
//                    - J c (s - s0) I: the inputs bk_substep_adjoint needs (call before it)
//   scalar_chain     dL/d(T', W', N', T_mat, mass, stress) -> dL/d(T, W, N, n, F, x, alpha) and
//                    the node adjoints of (dT, dW/W)
//   diffuse          node gather: dL/d(dT, dW/W) -> dL/d(volume, capacity, energy, water, heat, loss)
//   scatter          particle gather of the node-field adjoints -> dL/d(F, T, W, x)
//   owners           surface heat/loss of face-owning particles -> dL/d(T, W, F, x, h) and the
//                    face-vertex adjoints
//   vertices         mesh-vertex adjoints -> dL/d(x, F) of the bound particles
//   clear            zero the kept fields and every node scratch array over the active box
// Node scratch arrays start at zero and are left at zero. Discrete switches (tray contact test,
// nodes without capacity, the stability flags) carry no gradient.
#include <climits>
#include <cstdio>

#include "baking_b200.h"
#include "bk_common.h"
#include "bk_device.cuh"
#include "bk_launch.cuh"
#include "bk_scatter.cuh"

using namespace bk;

namespace {

constexpr int kThreads = 128;

// The forward substep's transport node fields (volume, capacity, energy, water, heat, loss,
// exchange) and the node adjoint scratch arrays.
struct BkGridFields {
    double* fields[7];
    double* field_bar[6];
    double2* dTr_bar;
};

struct TParams {
    int64_t n, pitch;
    int R;
    float origin[3], dx, rec_dx, dt;
    double rho_w, s0, c_water, kc, kw, cell;
    int water_enabled;
    double oven, tray, tray_transfer, surface_loss, latent;
    double contact_limit;  // floor height + contact distance, summed in float as the forward does
    int gas, settling;
    double ambient, peak, width, source_scale;  // gas: ambient pressure, source peak/width, dt * density
};

__device__ __forceinline__ void add_det_grad(float* Fb, int64_t i, int64_t pitch, const M3& F, float scale) {
    // d det(F) / dF = det(F) F^-T; adds scale * det(F) F^-T
    const M3 inv = inverse3(F);
    const float J = det3(F);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) Fb[(3 * r + c) * pitch + i] += scale * J * inv.m[3 * c + r];
}

// Gas content after this substep's local source (thermal_water.py:238-245):
// N' = N + dt rho alpha exp(-z^2), z = ((T + T')/2 - T_peak) / width; no source while settling.
// `ez`, `z` (may be NULL) return exp(-z^2) and z.
__device__ __forceinline__ double source_moles(const TParams& P, const BkState& in, const BkConstants& cst, int64_t i,
                                               double T, double Tn, double* ez, double* z) {
    double N = in.gas_moles[i];
    if (!P.settling) {
        const double zz = (0.5 * (T + Tn) - P.peak) / P.width;
        const double e = exp(-(zz * zz));
        N += P.source_scale * (double)cst.gas_rate[cst.gas_rate_per_particle ? i : 0] * e;
        if (ez) *ez = e;
        if (z) *z = zz;
    }
    return N;
}

// ------------------------------------------------------------------ prepare
__global__ void k_tadj_prepare(TParams P, BkState in, BkConstants cst, const double2* dTr,
                               float* __restrict__ T_mat, float* __restrict__ mass, float* __restrict__ tau_eff) {
    pdl_enter();
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    const int64_t pitch = P.pitch;
    Stencil st = make_stencil(load_v3(in.x, i, pitch), P.origin, P.dx, P.R, P.rec_dx);
    if (!st.valid) return;
    double dTp, ratio;
    gather_scalars(st, dTr, P.R, dTp, ratio);
    const double T = in.temperature[i];
    const double Tn = T + dTp, Wn = in.water[i] * (1.0 + ratio);
    T_mat[i] = (float)Tn;
    mass[i] = (float)(cst.dry_mass[i] + Wn);
    const M3 F = load_m3(in.F, i, pitch);
    const float J = det3(F);
    M3 tau = load_m3(in.tau, i, pitch);
    if (P.gas) {
        const float n = in.porosity[i];
        if (n > 0.0f && n < 1.0f && isfinite(n) && J > 0.0f) {
            const float p = (float)gas_pressure(source_moles(P, in, cst, i, T, Tn, nullptr, nullptr), (float)Tn, J, n);
            const float iso = J * ((float)P.ambient - p);
#pragma unroll
            for (int e = 0; e < 9; ++e) tau.m[e] += (e % 4) == 0 ? iso : 0.0f;
        }
    }
    const double sat = Wn * reciprocal_newton(P.rho_w * (double)cst.volume[i] * (double)J);
    const float iso = J * (float)P.c_water * ((float)sat - (float)P.s0);
#pragma unroll
    for (int e = 0; e < 9; ++e) tau.m[e] -= (e % 4) == 0 ? iso : 0.0f;
    store_m3(tau_eff, i, pitch, tau);
}

// ------------------------------------------------------------- scalar chain
// Node adjoints of (dT, dW/W) are scattered like the forward's scalar P2G (bk_scatter.cuh). The gather
// needs sum w (dT, r) for T' and W' and sum grad w (dT, r), which does not depend on the adjoints, for
// the weight gradients of x: both in float64, axis by axis. 1M particles: 173 us with a weight product,
// its gradients and a block tile per node and particle, now 133; it waits for memory (long_scoreboard 12
// of 17 cycles an issue at 4 blocks per SM), so eight blocks per SM with a few spilled registers are faster.
__global__ void __launch_bounds__(kThreads, 8) k_tadj_scalar(TParams P, BkState in, BkConstants cst,
                                                        const double2* dTr, BkAdjointTransport a,
                                                        const BkAdjointState adj, double2* __restrict__ dTr_bar) {
    __shared__ ScalarRecord<2> sm[kThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + tid;
    const int64_t pitch = P.pitch;
    prefetch_planes(i, P.n, pitch, in.F, 9, adj.F, 9, adj.x, 3);
    pdl_enter();
    double rate_b = 0.0;  // dL/d(gas source rate) through this particle
    double Tnb = 0.0, ratiob = 0.0;
    Stencil st;
    st.valid = false;
    st.b[0] = st.b[1] = st.b[2] = 0;
    if (i < P.n) st = make_stencil(load_v3(in.x, i, pitch), P.origin, P.dx, P.R, P.rec_dx);
    const bool valid = i < P.n && st.valid;
    if (i < P.n && !st.valid) {
        a.temperature_in[i] = 0.0;
        a.water_in[i] = 0.0;
        if (P.gas) a.gas_moles_in[i] = 0.0;
    } else if (valid) {
        double dTp = 0.0, ratio = 0.0;
        double gT[3] = {0.0, 0.0, 0.0}, gr[3] = {0.0, 0.0, 0.0};  // times dx
        const double2* nodes = dTr + node_index(st.b[0], st.b[1], st.b[2], P.R);
        const int64_t R = P.R;
#pragma unroll 1
        for (int ox = 0; ox < 3; ++ox) {
            const double wx = (double)pick3(st.w[0], ox), gx = (double)qweight_grad(st.l[0], ox);
            double tx = 0.0, rx = 0.0, tgy = 0.0, rgy = 0.0, tgz = 0.0, rgz = 0.0;
#pragma unroll
            for (int oy = 0; oy < 3; ++oy) {
                const double wy = (double)st.w[1][oy], gy = (double)qweight_grad(st.l[1], oy);
                double ty = 0.0, ry = 0.0, tg = 0.0, rg = 0.0;
#pragma unroll
                for (int oz = 0; oz < 3; ++oz) {
                    const double wz = (double)st.w[2][oz], gz = (double)qweight_grad(st.l[2], oz);
                    const double2 d = nodes[(ox * R + oy) * R + oz];
                    ty = fma(wz, d.x, ty);
                    ry = fma(wz, d.y, ry);
                    tg = fma(gz, d.x, tg);
                    rg = fma(gz, d.y, rg);
                }
                tx = fma(wy, ty, tx);
                rx = fma(wy, ry, rx);
                tgy = fma(gy, ty, tgy);
                rgy = fma(gy, ry, rgy);
                tgz = fma(wy, tg, tgz);
                rgz = fma(wy, rg, rgz);
            }
            dTp = fma(wx, tx, dTp);
            ratio = fma(wx, rx, ratio);
            gT[0] = fma(gx, tx, gT[0]);
            gr[0] = fma(gx, rx, gr[0]);
            gT[1] = fma(wx, tgy, gT[1]);
            gr[1] = fma(wx, rgy, gr[1]);
            gT[2] = fma(wx, tgz, gT[2]);
            gr[2] = fma(wx, rgz, gr[2]);
        }
        const double T = in.temperature[i], Tn = T + dTp;
        const double W = in.water[i];
        const double Wn = W * (1.0 + ratio);
        const M3 F = load_m3(in.F, i, pitch);
        const float Jf = det3(F);
        const double J = (double)Jf;
        const double V0 = (double)cst.volume[i];
        const double i_J = reciprocal_newton(J), i_full = i_J * reciprocal_newton(P.rho_w * V0);
        const double sat = Wn * i_full;
        // adjoints arriving at T', W', T_mat, mass and the P2G stress
        Tnb = a.temperature_out[i] + (double)adj.temperature[i];
        double Wnb = a.water_out[i] + (double)adj.mass[i];
        const double trace = (double)adj.tau[i] + (double)adj.tau[4 * pitch + i] + (double)adj.tau[8 * pitch + i];
        // stress -= iso I, iso = J c (s - s0)
        const double isob = -trace;
        double Jb = isob * P.c_water * (sat - P.s0);
        const double satb = isob * J * P.c_water;
        Wnb += satb * i_full;
        Jb -= satb * sat * i_J;
        double Tb_direct = 0.0;  // through the source's mean temperature, besides T'
        if (P.gas) {
            double ez = 0.0, z = 0.0;
            const double Np = source_moles(P, in, cst, i, T, Tn, &ez, &z);
            double Npb = a.gas_moles_out[i];
            const float n = in.porosity[i];
            if (n > 0.0f && n < 1.0f && isfinite(n) && Jf > 0.0f) {
                // stress += J (p_amb - p) I, p = N' R T_mat / (J n) (gas.py:11-13, 27-29)
                const float Tm = (float)Tn;
                const double pg = (double)(float)gas_pressure(Np, Tm, Jf, n);
                Jb += trace * (P.ambient - pg);
                const double pb = -trace * J;
                const double i_n = reciprocal_newton((double)n);
                Npb += pb * kGasConstant * (double)Tm * (i_J * i_n);
                Tnb += pb * pg * reciprocal_newton((double)Tm);
                Jb -= pb * pg * i_J;
                adj.porosity[i] += (float)(-pb * pg * i_n);
            }
            a.gas_moles_in[i] = Npb;
            if (!P.settling) {
                const double rate = (double)cst.gas_rate[cst.gas_rate_per_particle ? i : 0];
                rate_b = Npb * P.source_scale * ez;
                const double zb = Npb * P.source_scale * rate * ez * (-2.0 * z);
                Tnb += zb * 0.5 / P.width;
                Tb_direct = zb * 0.5 / P.width;
            }
        }
        // W' = W (1 + sum w r), T' = T + sum w dT
        ratiob = Wnb * W;
        a.water_in[i] = Wnb * (1.0 + ratio);
        a.temperature_in[i] = Tnb + Tb_direct;
        // weight gradients: x_bar += sum_j grad w_j (dT_j T'_bar + r_j ratio_bar)
#pragma unroll
        for (int c = 0; c < 3; ++c) adj.x[c * pitch + i] += (float)((gT[c] * Tnb + gr[c] * ratiob) * (double)P.rec_dx);
        add_det_grad(adj.F, i, pitch, F, (float)Jb);
    }
    // ---- scatter w (T'_bar, ratio_bar) into the node adjoints
    const double val[2] = {Tnb, ratiob};
    scatter_scalars<2, 2>(sm[tid >> 5], valid, st, val, {&dTr_bar->x, &dTr_bar->y}, P.R, group_lanes(P.n, P.R));
    if (P.gas && a.gas_rate) {
        if (cst.gas_rate_per_particle) {
            if (i < P.n) a.gas_rate[i] += rate_b;
        } else {
            // one shared rate: a warp sum, then one atomic per warp
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) rate_b += __shfl_xor_sync(0xffffffffu, rate_b, o);
            if (lane == 0 && rate_b != 0.0) atomicAdd(a.gas_rate, rate_b);
        }
    }
}

// ------------------------------------------------------------------ diffuse
// For node i with capacity: T_i = E_i / c_i, s_i = W_i / (rho_w v_i); heat rate
// H_i + sum_j kc fill_ij (T_j - T_i); water rate -Lo_i + sum_j mob_ij (s_j - s_i) with
// mob_ij = kw fill_ij (T_i + T_j)(s_i + s_j) / 4, fill_ij = 2 v_i v_j / ((v_i + v_j) cell);
// dT_i = dt heat_i / c_i, (dW/W)_i = dt water_i / W_i. Node i gathers the adjoints of its own rates
// and of its 6 neighbours' rates (which use its T, s, v), so no atomics are needed.
struct NodeVals {
    double v, c, T, s, W;
    bool live;
};

__device__ __forceinline__ NodeVals node_vals(const TParams& P, double* const* f, int64_t i) {
    NodeVals n;
    n.c = f[1][i];
    n.live = n.c > 0.0;
    n.v = f[0][i];
    n.W = f[3][i];
    n.T = n.live ? f[2][i] / n.c : 0.0;
    n.s = n.live ? n.W / (P.rho_w * n.v) : 0.0;
    return n;
}

__global__ void k_tadj_diffuse(TParams P, BkGridFields g, const int32_t* box) {
    pdl_enter();
    int lo[3], ext[3];
    int64_t count = 1;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int l = max(box[k], 0), h = min(box[3 + k], P.R - 1);
        if (l > h) return;
        lo[k] = l;
        ext[k] = h - l + 1;
        count *= ext[k];
    }
    const int R = P.R;
    const double dt = (double)P.dt;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < count; t += (int64_t)gridDim.x * blockDim.x) {
        int c[3];
        c[2] = lo[2] + (int)(t % ext[2]);
        c[1] = lo[1] + (int)((t / ext[2]) % ext[1]);
        c[0] = lo[0] + (int)(t / ((int64_t)ext[2] * ext[1]));
        const int64_t i = node_index(c[0], c[1], c[2], R);
        const NodeVals ni = node_vals(P, g.fields, i);
        double vb = 0.0, cb = 0.0, Eb = 0.0, Wb = 0.0, Hb = 0.0, Lb = 0.0, Tb = 0.0, sb = 0.0;
        if (ni.live) {
            const double2 ob = g.dTr_bar[i];
            // own outputs
            const double heat_b = ob.x * dt / ni.c;
            double heat_rate = g.fields[4][i], water_rate = -g.fields[5][i];
            // rates are needed for the c_i and W_i terms: recompute them below with the neighbours
            const double water_b = ni.W > 0.0 ? ob.y * dt / ni.W : 0.0;
            Hb = heat_b;
            Lb = -water_b;
#pragma unroll
            for (int axis = 0; axis < 3; ++axis)
#pragma unroll
                for (int side = 0; side < 2; ++side) {
                    int o[3] = {c[0], c[1], c[2]};
                    o[axis] += 2 * side - 1;
                    if (o[axis] < 0 || o[axis] >= R) continue;
                    const int64_t j = node_index(o[0], o[1], o[2], R);
                    const NodeVals nj = node_vals(P, g.fields, j);
                    if (!nj.live) continue;
                    const double sum = ni.v + nj.v;
                    const double fill = 2.0 * ni.v * nj.v / sum / P.cell;
                    const double dfill_i = 2.0 * nj.v * nj.v / (sum * sum) / P.cell;  // d fill / d v_i
                    const double hc = P.kc * fill;
                    heat_rate += hc * (nj.T - ni.T);
                    // the neighbour's heat-rate adjoint
                    const double2 jb = g.dTr_bar[j];
                    const double heat_bj = jb.x * dt / nj.c;
                    // own rate: hc (T_j - T_i); neighbour's rate: hc (T_i - T_j)
                    Tb += -heat_b * hc + heat_bj * hc;
                    vb += (heat_b * (nj.T - ni.T) + heat_bj * (ni.T - nj.T)) * P.kc * dfill_i;
                    if (P.water_enabled) {
                        const double water_bj = nj.W > 0.0 ? jb.y * dt / nj.W : 0.0;
                        const double q = P.kw * fill * 0.25;
                        const double mob = q * (ni.T + nj.T) * (ni.s + nj.s);
                        water_rate += mob * (nj.s - ni.s);
                        // own: mob (s_j - s_i); neighbour's: mob (s_i - s_j)
                        const double ds_own = nj.s - ni.s, ds_nb = ni.s - nj.s;
                        sb += water_b * (-mob + ds_own * q * (ni.T + nj.T)) + water_bj * (mob + ds_nb * q * (ni.T + nj.T));
                        Tb += (water_b * ds_own + water_bj * ds_nb) * q * (ni.s + nj.s);
                        vb += (water_b * ds_own + water_bj * ds_nb) * (mob / fill) * dfill_i;
                    }
                }
            // dT_i = dt heat_rate / c_i, ratio_i = dt water_rate / W_i
            cb -= ob.x * dt * heat_rate / (ni.c * ni.c);
            if (ni.W > 0.0) Wb -= ob.y * dt * water_rate / (ni.W * ni.W);
            // T_i = E_i / c_i, s_i = W_i / (rho_w v_i)
            Eb += Tb / ni.c;
            cb -= Tb * ni.T / ni.c;
            Wb += sb / (P.rho_w * ni.v);
            vb -= sb * ni.s / ni.v;
        }
        g.field_bar[0][i] = vb;
        g.field_bar[1][i] = cb;
        g.field_bar[2][i] = Eb;
        g.field_bar[3][i] = Wb;
        g.field_bar[4][i] = Hb;
        g.field_bar[5][i] = Lb;
    }
}

// ------------------------------------------------------------------ scatter
// Node fields (volume V0 det F, capacity, capacity T, W) += w (...) for every particle: the
// reverse of that scatter is a 27-node gather of the four field adjoints. The block first stages
// the adjoints of its particles' node box in shared memory (when the box fits kScatterTile nodes),
// so that the gathers read shared memory. 1M particles: 141 us with the weight products and their
// gradients formed per node and field, now 116 (seven blocks per SM for the same reason as above).
constexpr int kScatterTile = 512;

__global__ void __launch_bounds__(kThreads, 7) k_tadj_scatter(TParams P, BkState in, BkConstants cst, BkGridFields g_bar,
                                                         BkAdjointTransport a, const BkAdjointState adj) {
    __shared__ double s_bar[4][kScatterTile];
    __shared__ int s_box[6];
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + tid;
    const int64_t pitch = P.pitch;
    prefetch_planes(i, P.n, pitch, in.F, 9, adj.F, 9, adj.x, 3);
    pdl_enter();
    Stencil st;
    st.valid = false;
    st.b[0] = st.b[1] = st.b[2] = 0;
    if (i < P.n) st = make_stencil(load_v3(in.x, i, pitch), P.origin, P.dx, P.R, P.rec_dx);
    const bool valid = i < P.n && st.valid;
    // the block's node box
    if (tid < 6) s_box[tid] = tid < 3 ? INT_MAX : INT_MIN;
    __syncthreads();
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const int lo = __reduce_min_sync(0xffffffffu, valid ? st.b[ax] : INT_MAX);
        const int hi = __reduce_max_sync(0xffffffffu, valid ? st.b[ax] + 2 : INT_MIN);
        if (lane == 0 && lo != INT_MAX) {
            atomicMin(&s_box[ax], lo);
            atomicMax(&s_box[3 + ax], hi);
        }
    }
    __syncthreads();
    int lo[3] = {0, 0, 0}, ext[3] = {1, 1, 1};
    int count = 0;
    if (s_box[0] != INT_MAX) {
        long long c = 1;
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            lo[ax] = s_box[ax];
            ext[ax] = s_box[3 + ax] - s_box[ax] + 1;
            c *= ext[ax];
        }
        count = c <= kScatterTile ? (int)c : 0;
    }
    for (int t = tid; t < count; t += kThreads) {
        const int z = t % ext[2], y = (t / ext[2]) % ext[1], x = t / (ext[2] * ext[1]);
        const int64_t node = node_index(lo[0] + x, lo[1] + y, lo[2] + z, P.R);
#pragma unroll
        for (int f = 0; f < 4; ++f) s_bar[f][t] = g_bar.field_bar[f][node];
    }
    __syncthreads();  // uniform: every thread reaches it
    if (!valid) return;
    const M3 F = load_m3(in.F, i, pitch);
    const double vol = (double)cst.volume[i] * (double)det3(F);
    const double cap = cst.capacity[i], T = in.temperature[i], W = in.water[i];
    const double* const bar[4] = {g_bar.field_bar[0], g_bar.field_bar[1], g_bar.field_bar[2], g_bar.field_bar[3]};
    // sums of w f0, w f2 and w f3, and the weight gradients of the cofactor, axis by axis
    const double capT = cap * T;
    double v0 = 0.0, v2 = 0.0, v3 = 0.0, g[3] = {0.0, 0.0, 0.0};
    const int row = count > 0 ? ext[2] : P.R;
    const int64_t plane = count > 0 ? (int64_t)ext[1] * ext[2] : (int64_t)P.R * P.R;
    const int64_t corner = count > 0 ? ((int64_t)(st.b[0] - lo[0]) * ext[1] + (st.b[1] - lo[1])) * ext[2] + (st.b[2] - lo[2])
                                     : node_index(st.b[0], st.b[1], st.b[2], P.R);
    auto gather = [&](auto field) {
#pragma unroll 1
        for (int ox = 0; ox < 3; ++ox) {
            double x0 = 0.0, x2 = 0.0, x3 = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
#pragma unroll
            for (int oy = 0; oy < 3; ++oy) {
                double y0 = 0.0, y2 = 0.0, y3 = 0.0, s0 = 0.0, s1 = 0.0;
                const int64_t at = corner + ox * plane + oy * row;
#pragma unroll
                for (int oz = 0; oz < 3; ++oz) {
                    const double f0 = field(0, at + oz), f1 = field(1, at + oz), f2 = field(2, at + oz), f3 = field(3, at + oz);
                    const double w = (double)st.w[2][oz];
                    const double s = fma(vol, f0, fma(cap, f1, fma(capT, f2, W * f3)));
                    y0 = fma(w, f0, y0);
                    y2 = fma(w, f2, y2);
                    y3 = fma(w, f3, y3);
                    s0 = fma(w, s, s0);
                    s1 = fma((double)qweight_grad(st.l[2], oz), s, s1);
                }
                const double w = (double)st.w[1][oy];
                x0 = fma(w, y0, x0);
                x2 = fma(w, y2, x2);
                x3 = fma(w, y3, x3);
                gx = fma(w, s0, gx);
                gy = fma((double)qweight_grad(st.l[1], oy), s0, gy);
                gz = fma(w, s1, gz);
            }
            const double w = (double)pick3(st.w[0], ox);
            v0 = fma(w, x0, v0);
            v2 = fma(w, x2, v2);
            v3 = fma(w, x3, v3);
            g[0] = fma((double)qweight_grad(st.l[0], ox), gx, g[0]);
            g[1] = fma(w, gy, g[1]);
            g[2] = fma(w, gz, g[2]);
        }
    };
    if (count > 0) gather([&](int f, int64_t t) { return s_bar[f][t]; });
    else gather([&](int f, int64_t t) { return bar[f][t]; });
    const double volb = v0, Tb = cap * v2, Wb = v3;
    float xg[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) xg[c] = (float)(g[c] * (double)P.rec_dx);
    a.temperature_in[i] += Tb;
    a.water_in[i] += Wb;
#pragma unroll
    for (int c = 0; c < 3; ++c) adj.x[c * pitch + i] += xg[c];
    add_det_grad(adj.F, i, pitch, F, (float)(volb * (double)cst.volume[i]));
}

// ---------------------------------------------------------------- surface
// Mesh vertex positions of this substep (geometry/mesh_tracking.py:13-38) into surface.vertices,
// as the forward's transport phase computes them: a block of 128 or 256 threads per vertex of a coarse
// mesh, a warp per vertex of a fine one (kBlock = 32), kVertexWarps to a block.
constexpr int kVertexWarps = 4;
template <int kBlock>
constexpr int vertex_threads() { return kBlock == 32 ? 32 * kVertexWarps : kBlock; }

template <int kBlock>
__global__ void __launch_bounds__(vertex_threads<kBlock>()) k_tadj_vertex_positions(TParams P, const float* x,
                                                                                const float* F, BkSurface sf) {
    pdl_enter();
    if constexpr (kBlock == 32) {
        const int64_t k = (int64_t)blockIdx.x * kVertexWarps + (threadIdx.x >> 5);
        if (k >= sf.vertex_count) return;  // whole warps
        const int vid = sf.vertex_ids[k];
        const float v = vertex_warp(sf.binding_offsets, sf.binding_particles, sf.binding_weights, sf.reference_offsets,
                                    sf.binding_pitch, sf.reference_vertices, sf.vertex_pitch, x, F, P.pitch, vid);
        const int lane = threadIdx.x & 31;
        if (lane < 3) sf.vertices[lane * sf.vertex_pitch + vid] = v;
    } else {
        const int vid = sf.vertex_ids[blockIdx.x];
        const float v = vertex_block<kBlock>(sf.binding_offsets, sf.binding_particles, sf.binding_weights,
                                               sf.reference_offsets, sf.binding_pitch, sf.reference_vertices,
                                               sf.vertex_pitch, x, F, P.pitch, vid);
        if (threadIdx.x < 3) sf.vertices[threadIdx.x * sf.vertex_pitch + vid] = v;
    }
}

__device__ __forceinline__ void face_vertices(const BkSurface& sf, int f, double q[3][3], int vid[3]) {
    const int64_t vp = sf.vertex_pitch;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        vid[k] = sf.faces[3 * f + k];
#pragma unroll
        for (int a = 0; a < 3; ++a) q[k][a] = (double)sf.vertices[a * vp + vid[k]];
    }
}

// Owner o (particle p): its rates' adjoints to the state and to the face vertices; returns the
// heat-transfer parameter's.
__device__ __forceinline__ double owner_reverse(const TParams& P, const BkState& in, const BkConstants& cst, const BkSurface& sf,
                                                const BkGridFields& g, const BkAdjointTransport& a, const BkAdjointState& adj,
                                                int64_t o, int p, const Stencil& st) {
    const int64_t pitch = P.pitch;
    // recompute the owner's exposed and tray-contact areas
    double exposed = 0.0, contact = 0.0;
    const int f0 = sf.owner_face_offsets[o], f1 = sf.owner_face_offsets[o + 1];
    for (int f = f0; f < f1; ++f) {
        double q[3][3];
        int vid[3];
        face_vertices(sf, f, q, vid);
        const double e1[3] = {q[1][0] - q[0][0], q[1][1] - q[0][1], q[1][2] - q[0][2]};
        const double e2[3] = {q[2][0] - q[0][0], q[2][1] - q[0][1], q[2][2] - q[0][2]};
        const double nr[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
        const double len = sqrt(nr[0] * nr[0] + nr[1] * nr[1] + nr[2] * nr[2]);
        const double cy = (q[0][1] + q[1][1] + q[2][1]) / 3.0;
        if (cy <= P.contact_limit && nr[1] < -0.2 * len) contact += 0.5 * len;
        else exposed += 0.5 * len;
    }
    const M3 F = load_m3(in.F, p, pitch);
    const double vol = (double)cst.volume[p] * (double)det3(F);
    const double T = in.temperature[p], W = in.water[p];
    const double sat = W / (P.rho_w * vol);
    const double h = (double)cst.heat_parameter[0];
    const double loss = P.water_enabled ? P.surface_loss * T * sat * exposed : 0.0;
    const double heat = h * exposed * (P.oven - T) + P.tray_transfer * contact * (P.tray - T) - P.latent * loss;
    // gather the heat and loss adjoints from the owner's stencil
    double heatb = 0.0, lossb = 0.0, gs[3] = {0.0, 0.0, 0.0};
    const int64_t R = P.R, corner = node_index(st.b[0], st.b[1], st.b[2], P.R);
#pragma unroll
    for (int ox = 0; ox < 3; ++ox) {
        double hx = 0.0, lx = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
#pragma unroll
        for (int oy = 0; oy < 3; ++oy) {
            double hy = 0.0, ly = 0.0, s1 = 0.0;
#pragma unroll
            for (int oz = 0; oz < 3; ++oz) {
                const int64_t node = corner + (ox * R + oy) * R + oz;
                const double fh = g.field_bar[4][node], fl = g.field_bar[5][node];
                hy = fma((double)st.w[2][oz], fh, hy);
                ly = fma((double)st.w[2][oz], fl, ly);
                s1 = fma((double)qweight_grad(st.l[2], oz), heat * fh + loss * fl, s1);
            }
            const double w = (double)st.w[1][oy], s0 = heat * hy + loss * ly;
            hx = fma(w, hy, hx);
            lx = fma(w, ly, lx);
            gx = fma(w, s0, gx);
            gy = fma((double)qweight_grad(st.l[1], oy), s0, gy);
            gz = fma(w, s1, gz);
        }
        const double w = (double)st.w[0][ox];
        heatb = fma(w, hx, heatb);
        lossb = fma(w, lx, lossb);
        gs[0] = fma((double)qweight_grad(st.l[0], ox), gx, gs[0]);
        gs[1] = fma(w, gy, gs[1]);
        gs[2] = fma(w, gz, gs[2]);
    }
    float xg[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) xg[c] = (float)(gs[c] * (double)P.rec_dx);
#pragma unroll
    for (int c = 0; c < 3; ++c) adj.x[c * pitch + p] += xg[c];
    const double lossb_all = lossb - P.latent * heatb;
    double Tb = heatb * (-h * exposed - P.tray_transfer * contact);
    double exposedb = heatb * h * (P.oven - T), contactb = heatb * P.tray_transfer * (P.tray - T);
    if (P.water_enabled) {
        Tb += lossb_all * P.surface_loss * sat * exposed;
        exposedb += lossb_all * P.surface_loss * T * sat;
        const double satb = lossb_all * P.surface_loss * T * exposed;
        a.water_in[p] += satb / (P.rho_w * vol);
        const double volb = -satb * sat / vol;
        add_det_grad(adj.F, p, pitch, F, (float)(volb * (double)cst.volume[p]));
    }
    a.temperature_in[p] += Tb;
    const double hb = heatb * exposed * (P.oven - T);
    // face areas -> vertex adjoints
    const int64_t vp = sf.vertex_pitch;
    for (int f = f0; f < f1; ++f) {
        double q[3][3];
        int vid[3];
        face_vertices(sf, f, q, vid);
        const double e1[3] = {q[1][0] - q[0][0], q[1][1] - q[0][1], q[1][2] - q[0][2]};
        const double e2[3] = {q[2][0] - q[0][0], q[2][1] - q[0][1], q[2][2] - q[0][2]};
        const double nr[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
        const double len = sqrt(nr[0] * nr[0] + nr[1] * nr[1] + nr[2] * nr[2]);
        if (!(len > 0.0)) continue;
        const double cy = (q[0][1] + q[1][1] + q[2][1]) / 3.0;
        const bool is_contact = cy <= P.contact_limit && nr[1] < -0.2 * len;
        const double areab = is_contact ? contactb : exposedb;
        // area = |e1 x e2| / 2: nbar = areab n / (2 |n|); e1bar = e2 x nbar, e2bar = nbar x e1
        const double k = areab * 0.5 / len;
        const double nb[3] = {k * nr[0], k * nr[1], k * nr[2]};
        const double e1b[3] = {e2[1] * nb[2] - e2[2] * nb[1], e2[2] * nb[0] - e2[0] * nb[2], e2[0] * nb[1] - e2[1] * nb[0]};
        const double e2b[3] = {nb[1] * e1[2] - nb[2] * e1[1], nb[2] * e1[0] - nb[0] * e1[2], nb[0] * e1[1] - nb[1] * e1[0]};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            atomicAdd(&a.vertices[c * vp + vid[0]], -(e1b[c] + e2b[c]));
            atomicAdd(&a.vertices[c * vp + vid[1]], e1b[c]);
            atomicAdd(&a.vertices[c * vp + vid[2]], e2b[c]);
        }
    }
    return hb;
}

__global__ void k_tadj_owners(TParams P, BkState in, BkConstants cst, BkSurface sf, BkGridFields g,
                              BkAdjointTransport a, const BkAdjointState adj) {
    pdl_enter();
    const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t pitch = P.pitch;
    const bool mine = o < sf.owner_count;
    const int p = mine ? sf.owners[o] : 0;
    double hb = 0.0;
    Stencil st;
    st.valid = false;
    if (mine) st = make_stencil(load_v3(in.x, p, pitch), P.origin, P.dx, P.R, P.rec_dx);
    if (mine && st.valid) hb = owner_reverse(P, in, cst, sf, g, a, adj, o, p, st);
    // One shared parameter: a warp's sum in one atomic (an atomic per owner queued tens of thousands of
    // them on one address: 85 us for a ball of 100k particles, 18 with this and the gather in columns).
    if (a.heat_parameter) {
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) hb += __shfl_xor_sync(0xffffffffu, hb, k);
        if ((threadIdx.x & 31) == 0 && hb != 0.0) atomicAdd(a.heat_parameter, hb);
    }
}

// One block (kBlock = 32: one warp) per surface vertex: its adjoint to the bound particles' x and F,
// then zeroed.
template <int kBlock>
__global__ void __launch_bounds__(vertex_threads<kBlock>()) k_tadj_vertices(TParams P, BkSurface sf, BkAdjointTransport a,
                                                                        const BkAdjointState adj) {
    pdl_enter();
    __shared__ float s_w[kBlock / 32];
    const int64_t k = kBlock == 32 ? (int64_t)blockIdx.x * kVertexWarps + (threadIdx.x >> 5) : (int64_t)blockIdx.x;
    if (k >= sf.vertex_count) return;  // whole warps, or the whole block
    const int vid = sf.vertex_ids[k];
    const int t = threadIdx.x % kBlock;
    const int64_t vp = sf.vertex_pitch, bp = sf.binding_pitch, pitch = P.pitch;
    const double vb[3] = {a.vertices[vid], a.vertices[vp + vid], a.vertices[2 * vp + vid]};
    if constexpr (kBlock == 32) __syncwarp();
    else __syncthreads();
    if (t < 3) a.vertices[t * vp + vid] = 0.0;
    const int b0 = sf.binding_offsets[vid], b1 = sf.binding_offsets[vid + 1];
    if (b0 == b1 || (vb[0] == 0.0 && vb[1] == 0.0 && vb[2] == 0.0)) return;  // the same for the whole block or warp
    // v = (1 - sum_b w_b) pred_b0 + sum_b w_b pred_b
    float wsum = 0.f;
    for (int b = b0 + t; b < b1; b += kBlock) wsum += sf.binding_weights[b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
    if constexpr (kBlock > 32) {
        if ((t & 31) == 0) s_w[t >> 5] = wsum;
        __syncthreads();
        wsum = 0.f;
        for (int w = 0; w < kBlock / 32; ++w) wsum += s_w[w];
    }
    for (int b = b0 + t; b < b1; b += kBlock) {
        const float c = sf.binding_weights[b] + (b == b0 ? 1.f - wsum : 0.f);
        const int p = sf.binding_particles[b];
        const float o[3] = {sf.reference_offsets[b], sf.reference_offsets[bp + b], sf.reference_offsets[2 * bp + b]};
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const float pb = (float)(c * vb[r]);
            atomicAdd(&adj.x[r * pitch + p], pb);
#pragma unroll
            for (int k2 = 0; k2 < 3; ++k2) atomicAdd(&adj.F[(3 * r + k2) * pitch + p], pb * o[k2]);
        }
    }
}

// ------------------------------------------------------------------- clear
__global__ void k_tadj_clear(TParams P, BkGridFields g, const int32_t* box) {
    pdl_enter();
    int lo[3], ext[3];
    int64_t count = 1;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int l = max(box[k], 0), h = min(box[3 + k], P.R - 1);
        if (l > h) return;
        lo[k] = l;
        ext[k] = h - l + 1;
        count *= ext[k];
    }
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < count; t += (int64_t)gridDim.x * blockDim.x) {
        const int c2 = lo[2] + (int)(t % ext[2]);
        const int c1 = lo[1] + (int)((t / ext[2]) % ext[1]);
        const int c0 = lo[0] + (int)(t / ((int64_t)ext[2] * ext[1]));
        const int64_t i = node_index(c0, c1, c2, P.R);
#pragma unroll
        for (int k = 0; k < 7; ++k) g.fields[k][i] = 0.0;
#pragma unroll
        for (int k = 0; k < 6; ++k) g.field_bar[k][i] = 0.0;
        g.dTr_bar[i] = make_double2(0.0, 0.0);
    }
}

TParams tparams(const BkSubstepParams& p, const BkSurface* sf) {
    TParams t;
    t.n = p.n; t.pitch = p.pitch; t.R = p.resolution;
    for (int k = 0; k < 3; ++k) t.origin[k] = p.origin[k];
    t.dx = p.spacing; t.rec_dx = 1.0f / p.spacing; t.dt = p.time_step;
    t.rho_w = p.scalar.water_density;
    t.s0 = p.initial_saturation;
    t.c_water = p.water_stress;
    t.kc = (double)(p.conductivity * p.spacing);
    t.kw = (double)(p.diffusivity * p.scalar.water_density * p.spacing);
    t.cell = (double)(p.spacing * p.spacing * p.spacing);
    t.water_enabled = p.scalar.water_enabled;
    t.oven = p.scalar.oven_temperature; t.tray = p.scalar.tray_temperature;
    t.tray_transfer = p.scalar.tray_transfer; t.surface_loss = p.scalar.surface_loss; t.latent = p.scalar.latent_heat;
    t.contact_limit = sf ? (double)(sf->floor_height + sf->contact_distance) : 0.0;
    t.gas = p.gas;
    t.settling = p.settling;
    t.ambient = p.gas_ambient_pressure;
    t.peak = p.gas_peak;
    t.width = p.gas_width;
    t.source_scale = (double)(p.time_step * p.density);
    return t;
}

unsigned blocks(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

extern "C" {

int bk_transport_adjoint_prepare(const BkSubstepParams* params, const BkState* in, const BkConstants* constants,
                                 const double* node_dT_ratio, float* material_temperature, float* mass,
                                 float* stress, void* stream) {
    if (!params || !in || !constants || !node_dT_ratio || !material_temperature || !mass || !stress)
        return fail(BK_ERR_ARGUMENT, "bk_transport_adjoint_prepare: null argument");
    const BkSubstepParams& p = *params;
    if (!p.transport || p.material != 1 || !in->temperature || !in->water || !in->tau || !constants->dry_mass)
        return fail(BK_ERR_ARGUMENT, "bk_transport_adjoint_prepare: needs the Ding model with transport");
    if (p.gas && (!in->gas_moles || !in->porosity || !constants->gas_rate))
        return fail(BK_ERR_ARGUMENT, "bk_transport_adjoint_prepare: gas mode needs the gas arrays");
    if (p.n == 0) return BK_OK;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const cudaError_t e = launch_chained(k_tadj_prepare, blocks(p.n, 256), 256, 0, s, tparams(p, nullptr), *in, *constants,
                                         reinterpret_cast<const double2*>(node_dT_ratio), material_temperature, mass,
                                         stress);
    return check_chained(e, "bk_transport_adjoint_prepare");
}

int bk_transport_adjoint(const BkSubstepParams* params, const BkState* in, const BkConstants* constants,
                         const BkGrid* grid, const BkSurface* surface, const BkAdjointState* mechanics,
                         BkAdjointTransport* adjoint, void* stream) {
    if (!params || !in || !constants || !grid || !surface || !mechanics || !adjoint)
        return fail(BK_ERR_ARGUMENT, "bk_transport_adjoint: null argument");
    const BkSubstepParams& p = *params;
    if (!p.transport || p.material != 1)
        return fail(BK_ERR_UNSUPPORTED, "bk_transport_adjoint: the Ding model with transport");
    if (p.gas && (!in->gas_moles || !in->porosity || !constants->gas_rate || !adjoint->gas_moles_out ||
                  !adjoint->gas_moles_in || !mechanics->porosity))
        return fail(BK_ERR_ARGUMENT, "bk_transport_adjoint: gas mode needs the gas arrays and their adjoints");
    const BkAdjointTransport& a = *adjoint;
    if (!a.temperature_out || !a.water_out || !a.temperature_in || !a.water_in || !a.node_dT_ratio || !a.vertices ||
        !mechanics->tau || !mechanics->mass || !mechanics->temperature || !mechanics->x || !mechanics->F)
        return fail(BK_ERR_ARGUMENT, "bk_transport_adjoint: missing adjoint arrays");
    for (int k = 0; k < 6; ++k)
        if (!a.node_fields[k]) return fail(BK_ERR_ARGUMENT, "bk_transport_adjoint: missing node-field adjoint");
    for (int k = 0; k < 7; ++k)
        if (!grid->fields[k]) return fail(BK_ERR_ARGUMENT, "bk_transport_adjoint: missing node field");
    if (p.n == 0) return BK_OK;
    const TParams P = tparams(p, surface);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    BkGridFields g;
    for (int k = 0; k < 7; ++k) g.fields[k] = grid->fields[k];
    for (int k = 0; k < 6; ++k) g.field_bar[k] = a.node_fields[k];
    g.dTr_bar = reinterpret_cast<double2*>(a.node_dT_ratio);
    const int32_t* box = grid->bounds + 6;
    int device = 0, sms = 148;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const unsigned box_blocks = node_box_blocks(p.n, p.resolution, sms);
    cudaError_t e = launch_chained(k_tadj_scalar, blocks(p.n, kThreads), kThreads, 0, s, P, *in, *constants,
                                   reinterpret_cast<const double2*>(grid->node_dT_ratio), a, *mechanics, g.dTr_bar);
    if (int rc = check_chained(e, "bk_transport_adjoint/scalar")) return rc;
    e = launch_chained(k_tadj_diffuse, box_blocks, 256, 0, s, P, g, box);
    if (int rc = check_chained(e, "bk_transport_adjoint/diffuse")) return rc;
    e = launch_chained(k_tadj_scatter, blocks(p.n, kThreads), kThreads, 0, s, P, *in, *constants, g, a, *mechanics);
    if (int rc = check_chained(e, "bk_transport_adjoint/scatter")) return rc;
    const unsigned nv = (unsigned)surface->vertex_count;
    const int vertex_block_size = vertex_block_threads(surface->vertex_count, surface->binding_count);
    if (nv > 0) {
        if (vertex_block_size == 256)
            e = launch_chained(k_tadj_vertex_positions<256>, nv, 256, 0, s, P, in->x, in->F, *surface);
        else if (vertex_block_size == 128)
            e = launch_chained(k_tadj_vertex_positions<128>, nv, 128, 0, s, P, in->x, in->F, *surface);
        else
            e = launch_chained(k_tadj_vertex_positions<32>, blocks(nv, kVertexWarps), 32 * kVertexWarps, 0, s, P, in->x,
                               in->F, *surface);
        if (int rc = check_chained(e, "bk_transport_adjoint/vertex_positions")) return rc;
    }
    if (surface->owner_count > 0) {
        e = launch_chained(k_tadj_owners, blocks(surface->owner_count, 64), 64, 0, s, P, *in, *constants, *surface, g, a,
                           *mechanics);
        if (int rc = check_chained(e, "bk_transport_adjoint/owners")) return rc;
    }
    if (nv > 0) {
        if (vertex_block_size == 256) e = launch_chained(k_tadj_vertices<256>, nv, 256, 0, s, P, *surface, a, *mechanics);
        else if (vertex_block_size == 128)
            e = launch_chained(k_tadj_vertices<128>, nv, 128, 0, s, P, *surface, a, *mechanics);
        else
            e = launch_chained(k_tadj_vertices<32>, blocks(nv, kVertexWarps), 32 * kVertexWarps, 0, s, P, *surface, a,
                               *mechanics);
        if (int rc = check_chained(e, "bk_transport_adjoint/vertices")) return rc;
    }
    e = launch_chained(k_tadj_clear, box_blocks, 256, 0, s, P, g, box);
    return check_chained(e, "bk_transport_adjoint/clear");
}

}  // extern "C"
