// Internal-mode (baroclinic) kernels of oce_timestep case(3)
// (src/fv_main.F90:1983-2070):
//   pressure_col : densityJM + hydrostatic prefix sum per node column
//   bpg_elem     : baroclinic_pressure_gradient_3D per element column
//   velgrad3d    : vel_gradients (least squares, free slip) per (elem, level)
//   adv3_edge    : upwind horizontal momentum flux per (internal edge, level)
//   velrhs       : compute_vel_rhs up to the AB combine, per (elem, level):
//                  pressure force, Coriolis/AB2 history, the edge momentum
//                  fluxes gathered in edge order, filter viscosity, QUICK
//                  vertical advection
//   implvisc     : implicit vertical viscosity per element column
//                  (momentum_vert_impl_visc_tmp / momentum_vert_impl_visc)
//   update3d     : update_3D_vel per element column; stores the new Je, Ze, ZBe
//   wvel         : vert_vel_sigma per node column (edge gather + reverse scan)
//   jac_swap     : last elevation rotation of the sub-cycle, jacobian elevation
//   je_elem      : Je, Ze, ZBe at init
#include "device_common.cuh"

FESOMC_PREC_BEGIN

// Column blocks: B consecutive entities per block, one thread per (entity,
// level), levels on consecutive threads (coalesced column access).  Level
// sums / scans that the reference does sequentially go through shared memory
// (one row of L per entity, odd row stride) and are done by one thread per
// entity, in level order.
struct ColBlock {
    int L, B, jl, z;
    __device__ ColBlock(const Dev &d)
        : L(d.L), B(d.by_L.div(blockDim.x)), jl(d.by_L.div(threadIdx.x)), z((int)threadIdx.x - jl * d.L) {}
};

// ---------------------------------------------------------------------------
// pressure (fv_pressure_new.F90:91-107): density per (node, level), the
// hydrostatic sum per node in level order
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) k_pressure_col(Dev d) {
    pdl_enter();
    extern __shared__ __align__(16) unsigned char sm_raw[];
    real *sm = reinterpret_cast<real *>(sm_raw);
    const real gd0 = kG / d.density_0;
    const int L = d.L, NS = d.NS;
    const ColBlock cb(d);
    const int S = L | 1;
    for (long long nb = (long long)blockIdx.x * cb.B; nb < d.N; nb += (long long)gridDim.x * cb.B) {
        const long long n_ = nb + cb.jl;
        const bool act = cb.jl < cb.B && n_ < d.N;
        if (act) {
            const int n = (int)n_;
            const real a = jac_a(d, d.eta_jac, n);
            const size_t i = (size_t)n * L + cb.z;
            const real rho = density_jm(d.TF[i], d.SF[i], -z_of(d, a, cb.z), d.density_0);
            d.rho_c[i] = rho;
            sm[cb.jl * S + cb.z] = rho * jc_of(d, a, cb.z) * gd0;
        }
        __syncthreads();
        if ((int)threadIdx.x < cb.B && nb + threadIdx.x < d.N) {
            real *row = sm + threadIdx.x * S;
            real hp = real(0.0);
            for (int k = 0; k < L; ++k) {
                hp = hp + row[k];
                row[k] = hp;
            }
        }
        __syncthreads();
        if (act) {
            const size_t bs = (size_t)n_ * NS;
            d.hpressure[bs + cb.z + 1] = sm[cb.jl * S + cb.z];
            if (cb.z == 0) d.hpressure[bs] = real(0.0);
        }
        __syncthreads();
    }
}

// What the level threads of a column block need of their element, staged in
// shared memory by four lanes per element, one per node, before the level
// phase: the level threads otherwise load nodes, geometry and elevations (24
// of bpg_elem's 33 loads, the same for all levels of an element) each for
// itself.  kEsReals values per element.
constexpr int kEsW = 0, kEsGx = 4, kEsGy = 8, kEsAn = 12, kEsA = 16, kEsX = 20, kEsReals = 24;
// lanes of the caller's warp that take part in a phase of the block's first
// 'count' threads
__device__ __forceinline__ unsigned lanes_below(int count) {
    const int n = count - (int)(threadIdx.x & ~31u);
    return n >= 32 ? kFull : (1u << n) - 1u;
}

// baroclinic_pressure_gradient_3D (fv_pressure_new.F90:146-221) per
// (element, level); Bar_pr_2D as a level-ordered sum per element.  Also the
// element's surface pressure force of compute_vel_rhs (fv_3D_vel.F90:60-75),
// the same for every level.  Column blocks reach 1024 threads (B * L), so
// the kernel is bounded to 64 registers.
// Bound by the latency of its loads between barriers, by its loads' number
// before the staging.  FP32 (48 registers, 8 blocks of 160 threads per SM)
// has the level loads in flight during the staging; FP64 has no registers
// for that.  1.05 M nodes FP64 0.838 -> 0.762 ms (with the early loads 0.85),
// 232 k FP32 0.195 -> 0.109, 40 k, 30 layers 0.058 as before.
#if FESOMC_FP32
#define BPG_BOUNDS __maxnreg__(48)
constexpr bool kBpgEarly = true;
#else
#define BPG_BOUNDS __launch_bounds__(1024)
constexpr bool kBpgEarly = false;
#endif
__global__ void BPG_BOUNDS k_bpg_elem(Dev d) {
    pdl_enter();
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const int L = d.L, NS = d.NS;
    const ColBlock cb(d);
    const int S = 2 * L + 1, B = cb.B;
    real *const es = reinterpret_cast<real *>(sm_raw);    // kEsReals per element
    real *const ex = es + B * kEsReals;                   // 12 per element: dh, depth, pressure of its nodes
    real *const sm = ex + B * 12;
    for (long long eb = (long long)blockIdx.x * B; eb < d.E; eb += (long long)gridDim.x * B) {
        // the level loads first: they are in flight during the staging
        const long long e_ = eb + cb.jl;
        const bool act = cb.jl < B && e_ < d.E;
        real je = real(1.0), hu[4], hl[4];
        if (kBpgEarly) {
            if (act) {
                const int4 en = d.elem_nodes[e_];
                const int nd[4] = {en.x, en.y, en.z, en.w};
                je = d.Je[(size_t)e_ * L + cb.z];
                for (int k = 0; k < 4; ++k) {
                    hu[k] = d.hpressure[(size_t)nd[k] * NS + cb.z];
                    hl[k] = d.hpressure[(size_t)nd[k] * NS + cb.z + 1];
                }
            }
        }
        if ((int)threadIdx.x < 4 * B) {
            const int j = threadIdx.x >> 2, k = threadIdx.x & 3;
            const int e = (int)(eb + j < d.E ? eb + j : d.E - 1);
            const int nd = reinterpret_cast<const int *>(d.elem_nodes)[4 * (size_t)e + k];
            const real4 g = (k & 1) ? d.gs_y[e] : d.gs_x[e];
            real *const o = es + j * kEsReals, *const x = ex + j * 12;
            x[k] = d.depth[nd] + d.eta_n[nd];
            x[4 + k] = d.depth[nd];
            x[8 + k] = -kG * (d.atp1[nd] * d.eta_n[nd] - d.atp2[nd] * d.ssh_gp[nd]);
            o[kEsAn + k] = jac_a(d, d.eta_jac, nd);
            const real4 w = d.w_cv[e];
            if (k == 2) { o[kEsW] = w.x; o[kEsW + 1] = w.y; o[kEsW + 2] = w.z; o[kEsW + 3] = w.w; }
            if (k < 2) {
                real *const go = o + (k ? kEsGy : kEsGx);
                go[0] = g.x; go[1] = g.y; go[2] = g.z; go[3] = g.w;
            }
            if (k == 3) o[kEsX] = d.elem_bpfac[e];
            __syncwarp(lanes_below(4 * B));
            // Ax, Ay, Bx, By: gradients of the total depth and of the depth
            const real *v = x + (k < 2 ? 0 : 4);
            o[kEsA + k] = wsum(g, v[0], v[1], v[2], v[3]);
            if (k < 2) {
                real pr[4] = {x[8], x[9], x[10], x[11]};
                if (d.key_atm) {
                    // sea-level pressure and E - P of the element (fv_3D_vel.F90:40-53)
                    const int4 en = d.elem_nodes[e];
                    const real d0i = real(1.0) / d.density_0;
                    const real atm_mean = wsum(w, (real)d.mslp[en.x], (real)d.mslp[en.y], (real)d.mslp[en.z], (real)d.mslp[en.w]);
                    const real emp_mean = wsum(w, (real)d.emp[en.x], (real)d.emp[en.y], (real)d.emp[en.z], (real)d.emp[en.w]);
                    for (int q = 0; q < 4; ++q)
                        pr[q] = pr[q] - (real(kPref) - atm_mean) * d0i + kG * emp_mean * d0i;
                }
                if (eb + j < d.E)
                    reinterpret_cast<real *>(d.Fp)[2 * (size_t)e + k] = wsum(g, pr[0], pr[1], pr[2], pr[3]) * d.elem_area[e];
            }
        }
        __syncthreads();
        if (act) {
            const int e = (int)e_, z = cb.z;
            const real *const o = es + cb.jl * kEsReals;
            real pre[4];
            if (!kBpgEarly) {
                const int4 en = d.elem_nodes[e_];
                const int nd[4] = {en.x, en.y, en.z, en.w};
                je = d.Je[(size_t)e_ * L + cb.z];
                for (int k = 0; k < 4; ++k) {
                    hu[k] = d.hpressure[(size_t)nd[k] * NS + cb.z];
                    hl[k] = d.hpressure[(size_t)nd[k] * NS + cb.z + 1];
                }
            }
            for (int k = 0; k < 4; ++k) pre[k] = real(0.5) * (hu[k] + hl[k]) * jc_of(d, o[kEsAn + k], z);
            const real4 w = make_real4(o[kEsW], o[kEsW + 1], o[kEsW + 2], o[kEsW + 3]);
            const real4 gx = make_real4(o[kEsGx], o[kEsGx + 1], o[kEsGx + 2], o[kEsGx + 3]);
            const real4 gy = make_real4(o[kEsGy], o[kEsGy + 1], o[kEsGy + 2], o[kEsGy + 3]);
            const real accJe_inv = -o[kEsX] / je;
            const real qd_up = wsum(w, hu[0], hu[1], hu[2], hu[3]);
            const real qd_low = wsum(w, hl[0], hl[1], hl[2], hl[3]);
            const real sx = wsum(gx, pre[0], pre[1], pre[2], pre[3]);
            const real sy = wsum(gy, pre[0], pre[1], pre[2], pre[3]);
            const real s0 = __ldg(d.sig + z), s1 = __ldg(d.sig + z + 1);
            const real Ax = o[kEsA], Ay = o[kEsA + 1], Bx = o[kEsA + 2], By = o[kEsA + 3];
            const real bu = accJe_inv * (sx + qd_low * (s1 * Ax - Bx) - qd_up * (s0 * Ax - Bx));
            const real bv = accJe_inv * (sy + qd_low * (s1 * Ay - By) - qd_up * (s0 * Ay - By));
            d.Bar_pru[(size_t)e * L + z] = bu;
            d.Bar_prv[(size_t)e * L + z] = bv;
            sm[cb.jl * S + z] = bu * je;
            sm[cb.jl * S + L + z] = bv * je;
        }
        __syncthreads();
        // one thread per (element, component): the level sums in level order
        if ((int)threadIdx.x < 2 * B && eb + (threadIdx.x >> 1) < d.E) {
            const int j = threadIdx.x >> 1, c = threadIdx.x & 1;
            const real *row = sm + j * S + c * L;
            real b = real(0.0);
            for (int k = 0; k < L; ++k) b = b + row[k];
            reinterpret_cast<real *>(d.Bar_pr_2D)[2 * (eb + j) + c] = b;
        }
        __syncthreads();
    }
}

// vel_gradients (fv_gradients.F90:2-93), one thread per (element, level).
// FP64: 64 registers: 32 resident warps per SM instead of 24 (11 % faster; 48:
// 0.380 against 0.373 ms at 1.05 M nodes).  FP32: 32 registers, 232 k nodes
// 0.074 -> 0.052 ms.
__global__ void __maxnreg__(FESOMC_FP32 ? 32 : 64) k_velgrad3d(Dev d) {
    pdl_enter();
    const unsigned total = (unsigned)d.E * d.L;
    GRID_LOOP(ii, total) {
        const int e = d.by_L.div(ii);
        const int z = (int)ii - e * d.L;
        const int L = d.L;
        const int4 en = d.elem_nodes[e];
        const int4 nb = d.elem_nb[e];
        const int4 ee = d.elem_edges[e];
        const int nbs[4] = {nb.x, nb.y, nb.z, nb.w};
        const int eds[4] = {ee.x, ee.y, ee.z, ee.w};
        const real4 gx = d.gv_x[e], gy = d.gv_y[e];
        const real gxa[4] = {gx.x, gx.y, gx.z, gx.w};
        const real gya[4] = {gy.x, gy.y, gy.z, gy.w};
        const int jend = (en.x == en.w) ? 3 : 4;
        const real u0 = d.U_n[ii], v0 = d.V_n[ii];
        real a1 = real(0.0), a2 = real(0.0), a3 = real(0.0), a4 = real(0.0);
        for (int j = 0; j < jend; ++j) {
            const int e2 = nbs[j];
            if (e2 >= 0) {
                const real u2 = d.U_n[(size_t)e2 * L + z], v2 = d.V_n[(size_t)e2 * L + z];
                a1 = a1 + gxa[j] * (u2 - u0);
                a2 = a2 + gya[j] * (u2 - u0);
                a3 = a3 + gxa[j] * (v2 - v0);
                a4 = a4 + gya[j] * (v2 - v0);
            } else {
                const real2 dxy = d.edge_dxdy[eds[j]];
                const real zc1 = dxy.x * d.elem_cos[e], zc2 = dxy.y;
                const real un = -real(2.0) * (u0 * zc2 - v0 * zc1) / (zc1 * zc1 + zc2 * zc2);
                a1 = a1 + gxa[j] * un * zc2;
                a2 = a2 + gya[j] * un * zc2;
                a3 = a3 - gxa[j] * un * zc1;
                a4 = a4 - gya[j] * un * zc1;
            }
        }
        d.vgux[ii] = a1;
        d.vguy[ii] = a2;
        d.vgvx[ii] = a3;
        d.vgvy[ii] = a4;
    }
}

// w-weighted element mean of a node column value: SUM(w_cv*X(k,nodes))
__device__ __forceinline__ real wsum_col(const real4 &w, const real *X, int stride, const int4 &en, int k) {
    return wsum(w, X[(size_t)en.x * stride + k], X[(size_t)en.y * stride + k], X[(size_t)en.z * stride + k],
                X[(size_t)en.w * stride + k]);
}
__device__ __forceinline__ real wsum_zbar(const Dev &d, const real4 &w, const real4 &a, int k) {
    return wsum(w, zbar_of(d, a.x, k), zbar_of(d, a.y, k), zbar_of(d, a.z, k), zbar_of(d, a.w, k));
}
__device__ __forceinline__ real wsum_z(const Dev &d, const real4 &w, const real4 &a, int k) {
    return wsum(w, z_of(d, a.x, k), z_of(d, a.y, k), z_of(d, a.z, k), z_of(d, a.w, k));
}

// Vertical momentum flux uvertAB(:,k) of momentum_vert_adv_upwind at interface
// k (0-based, 0..NS-1) of element e (fv_advection.F90:389-443); the element
// means of Z and zbar come from the stored Ze / ZBe.
__device__ __forceinline__ void uvert_at(const Dev &d, int e, int k, const real4 &w, const int4 &en, real ar,
                                         real &fu, real &fv) {
    const int L = d.L, NS = d.NS;
    const real *U = d.U_n + (size_t)e * L;
    const real *V = d.V_n + (size_t)e * L;
    if (k == NS - 1) { fu = real(0.0); fv = real(0.0); return; }
    const real wv = wsum_col(w, d.Wvel, NS, en, k) * ar;
    if (k == 0) { fu = -wv * U[0]; fv = -wv * V[0]; return; }
    const int nz = k + 1;  // 1-based interface index, 2..NS-1
    const real *ZE = d.Ze + (size_t)e * L;   // ZE[m-1] = SUM(w*Z(m))
    const real *ZB = d.ZBe + (size_t)e * L;  // ZB[m-1] = SUM(w*zbar(m))
    real umean = real(0.0), vmean = real(0.0);
    // U_n(m) 1-based  ->  U[m-1]
    if (wv >= real(0.0)) {
        if (nz == NS - 1) {
            umean = real(0.5) * (U[nz - 2] + U[nz - 1]);
            vmean = real(0.5) * (V[nz - 2] + V[nz - 1]);
        } else {
            const real Z1 = ZB[nz - 1];
            const real aa = Z1 - ZE[nz - 2];
            const real bb = ZE[nz - 1] - Z1;
            const real cc = ZE[nz] - Z1;
            const real dd = (cc + aa) * (bb * bb - aa * aa) - (cc * cc - aa * aa) * (bb + aa);
            const real dg = aa * bb * (aa + bb) / dd;
            const real db = -aa * cc * (aa + cc) / dd;
            const real da = real(1.0) - dg - db;
            umean = U[nz - 2] * da + U[nz - 1] * db + U[nz] * dg;
            vmean = V[nz - 2] * da + V[nz - 1] * db + V[nz] * dg;
        }
    }
    if (wv < real(0.0)) {
        if (nz == 2) {
            umean = real(0.5) * (U[nz - 2] + U[nz - 1]);
            vmean = real(0.5) * (V[nz - 2] + V[nz - 1]);
        } else {
            const real Z1 = ZB[nz - 1];
            const real aa = ZE[nz - 1] - Z1;
            const real bb = Z1 - ZE[nz - 2];
            const real cc = Z1 - ZE[nz - 3];
            const real dd = (cc + aa) * (bb * bb - aa * aa) - (cc * cc - aa * aa) * (bb + aa);
            const real dg = aa * bb * (aa + bb) / dd;
            const real db = -aa * cc * (aa + cc) / dd;
            const real da = real(1.0) - dg - db;
            umean = U[nz - 1] * da + U[nz - 2] * db + U[nz - 3] * dg;
            vmean = V[nz - 1] * da + V[nz - 2] * db + V[nz - 3] * dg;
        }
    }
    fu = -umean * wv;
    fv = -vmean * wv;
}

// Upwind horizontal momentum flux of one (internal edge, level)
// (momentum_adv_upwind, fv_advection.F90:114-188), computed once and gathered
// by the edge's two elements in velrhs.  Thread per (edge, level), levels on
// consecutive threads.
__global__ void k_adv3_edge(Dev d) {
    pdl_enter();
    const unsigned total = (unsigned)d.Ed_in * d.L;
    const int L = d.L;
    GRID_LOOP(ii, total) {
        const int ed = d.by_L.div(ii);
        const int z = (int)ii - ed * L;
        const int2 nn = d.edge_nodes[ed];
        const int2 et = d.edge_tri[ed];
        const real acc = real(0.5) * (d.ac[nn.x] + d.ac[nn.y]);
        const real4 X = d.edge_cross[ed];
        const size_t i1 = (size_t)et.x * L + z, i2 = (size_t)et.y * L + z;
        const real u1 = d.U_n[i1] - d.vgux[i1] * X.x - d.vguy[i1] * X.y;
        const real v1 = d.V_n[i1] - d.vgvx[i1] * X.x - d.vgvy[i1] * X.y;
        const real u2 = d.U_n[i2] - d.vgux[i2] * X.z - d.vguy[i2] * X.w;
        const real v2 = d.V_n[i2] - d.vgvx[i2] * X.z - d.vgvy[i2] * X.w;
        const real jd = real(0.5) * (jc_of(d, jac_a(d, d.eta_jac, nn.x), z) + jc_of(d, jac_a(d, d.eta_jac, nn.y), z));
        const real2 dxy = d.edge_dxdy[ed];
        const real un = real(0.5) * kREarth * jd *
                          ((u1 + u2) * dxy.y - (v1 * d.elem_cos[et.x] + v2 * d.elem_cos[et.y]) * dxy.x);
        real uu, vv;
        if (un >= real(0.0)) { uu = u1 * un * acc; vv = v1 * un * acc; }
        else { uu = u2 * un * acc; vv = v2 * un * acc; }
        d.adv3[ii] = make_real2(uu, vv);
    }
}

// ---------------------------------------------------------------------------
// biharmonic_viscosity (fv_viscosity.F90:104-334) and its sub-step-1 twin
// biharmonic_viscosity_3D_to_2D (:964-1219): two Laplacians of a velocity,
// each an edge flux of the normal velocity gradient (the mean of the two
// elements' gradients with its tangential part replaced by the difference
// quotient), gathered per element in edge order (internal edges, then
// boundary edges).
// bih_edge: the flux of every (edge, level); mode 0 times Jd, mode 1 times
// Jd and the edge's sponge factor, mode 2 plain.
// bih_uc: U_c = Ah * sum of the mode-0 fluxes; Ah = -Abh0 sqrt(area/s)/s
// (mode 0), -acc Abh0 sqrt(area/s)/s (mode 1, the 3D-to-2D form; its Visc
// term is zero on this path, h_viscosity only runs with the sediment model).
// bih_grad: vel_lapl_gradients (fv_gradients.F90:327-402) of U_c into the
// velocity-gradient arrays.  velgrad_puls: vel_gradients_puls
// (fv_gradients.F90:404-496, free slip) of U_puls.
// velrhs gathers the mode-1 fluxes into U_rhs after the filter viscosity;
// p1_elem gathers the mode-2 fluxes, times Je, into U_rhs_2D_3D.
// bih_geom, once per model: what the passes of both biharmonic operators need
// of an edge and an element beside the fields.  The square root and the two
// divisions of the unit vector, and the square root and two divisions of Ah,
// were formed again for every level: 42 k nodes, 20 layers, FP64: biharmonic
// 0.129 -> 0.097 ms, biharmonic_2d 0.147 -> 0.116.
// ---------------------------------------------------------------------------
__global__ void k_bih_geom(Dev d) {
    pdl_enter();
    GRID_LOOP(ii, d.Ed) {
        const int ed = (int)ii;
        const int2 et = d.edge_tri[ed];
        const real2 dxy = d.edge_dxdy[ed];
        const real ye = dxy.y * kREarth;
        real xe, tx = real(0.0), ty = real(0.0), tl = real(1.0);
        if (ed < d.Ed_in) {
            const real4 X = d.edge_cross[ed];
            xe = dxy.x * kREarth * real(0.5) * (d.elem_cos[et.x] + d.elem_cos[et.y]);
            tx = -X.x + X.z;
            ty = -X.y + X.w;
            tl = sqrt(tx * tx + ty * ty);
            tx = tx / tl;
            ty = ty / tl;
        } else {
            xe = dxy.x * kREarth * d.elem_cos[et.x];
        }
        d.bih_dir[ed] = make_real4(xe, ye, tx, ty);
        d.bih_len[ed] = tl;
    }
    GRID_LOOP(ii, d.E) {
        const int e = (int)ii;
        const real sa = scale_area_of(d, e);
        d.bih_ah[e] = make_real2(-d.Abh0 * sqrt(d.elem_area[e] / sa) / sa,
                                 -d.elem_acc[e] * d.Abh0 * sqrt(d.elem_area[e] / sa) / sa);
    }
}

__global__ void k_bih_edge(Dev d, const real *U, const real *V, int mode) {
    pdl_enter();
    const unsigned total = (unsigned)d.Ed * d.L;
    const int L = d.L;
    GRID_LOOP(ii, total) {
        const int ed = d.by_L.div(ii);
        const int z = (int)ii - ed * L;
        const int2 nn = d.edge_nodes[ed];
        const int2 et = d.edge_tri[ed];
        const real4 G = d.bih_dir[ed];
        const real xe = G.x, ye = G.y;
        const size_t i1 = (size_t)et.x * L + z;
        real u1, v1;
        if (ed < d.Ed_in) {
            const size_t i2 = (size_t)et.y * L + z;
            const real tx = G.z, ty = G.w, tl = d.bih_len[ed];
            real g1 = real(0.5) * (d.vgux[i1] + d.vgux[i2]);
            real g2 = real(0.5) * (d.vguy[i1] + d.vguy[i2]);
            real tt = g1 * tx + g2 * ty - (U[i2] - U[i1]) / tl;
            g1 = g1 - tx * tt;
            g2 = g2 - ty * tt;
            u1 = (g1 * ye - g2 * xe);
            g1 = real(0.5) * (d.vgvx[i1] + d.vgvx[i2]);
            g2 = real(0.5) * (d.vgvy[i1] + d.vgvy[i2]);
            tt = g1 * tx + g2 * ty - (V[i2] - V[i1]) / tl;
            g1 = g1 - tx * tt;
            g2 = g2 - ty * tt;
            v1 = (g1 * ye - g2 * xe);
        } else {
            u1 = (d.vgux[i1]) * ye - (d.vguy[i1]) * xe;
            v1 = (d.vgvx[i1]) * ye - (d.vgvy[i1]) * xe;
        }
        real fu = u1, fv = v1;
        if (mode != 2) {
            const real jd = real(0.5) * (jc_of(d, jac_a(d, d.eta_jac, nn.x), z) + jc_of(d, jac_a(d, d.eta_jac, nn.y), z));
            fu = u1 * jd;
            fv = v1 * jd;
            if (mode == 1) {
                const real acc = (d.ac[nn.x] + d.ac[nn.y]) / real(2.0);
                fu = fu * acc;
                fv = fv * acc;
            }
        }
        d.bihfl[ii] = make_real2(fu, fv);
    }
}

__global__ void k_bih_uc(Dev d, int mode) {
    pdl_enter();
    const unsigned total = (unsigned)d.E * d.L;
    const int L = d.L;
    GRID_LOOP(ii, total) {
        const int e = d.by_L.div(ii);
        const int z = (int)ii - e * L;
        const real2 c = bih_gather(d, e, z);
        const real2 ah = d.bih_ah[e];
        const real Ah = mode == 0 ? ah.x : ah.y;
        d.bihU[ii] = c.x * (Ah);
        d.bihV[ii] = c.y * (Ah);
    }
}

// least-squares gradients of (U, V) per (element, level); the boundary
// neighbour is -2 U (vel_lapl_gradients) or the free-slip mirror
// (vel_gradients_puls)
template <bool FREE_SLIP>
__global__ void k_bih_grad(Dev d, const real *U, const real *V) {
    pdl_enter();
    const unsigned total = (unsigned)d.E * d.L;
    const int L = d.L;
    GRID_LOOP(ii, total) {
        const int e = d.by_L.div(ii);
        const int z = (int)ii - e * L;
        const int4 en = d.elem_nodes[e];
        const int4 nb = d.elem_nb[e];
        const int4 ee = d.elem_edges[e];
        const int nbs[4] = {nb.x, nb.y, nb.z, nb.w};
        const int eds[4] = {ee.x, ee.y, ee.z, ee.w};
        const real4 gx = d.gv_x[e], gy = d.gv_y[e];
        const real gxa[4] = {gx.x, gx.y, gx.z, gx.w};
        const real gya[4] = {gy.x, gy.y, gy.z, gy.w};
        const int jend = (en.x == en.w) ? 3 : 4;
        const real u0 = U[ii], v0 = V[ii];
        real a1 = real(0.0), a2 = real(0.0), a3 = real(0.0), a4 = real(0.0);
        for (int j = 0; j < jend; ++j) {
            const int e2 = nbs[j];
            real u, v;
            if (e2 >= 0) {
                u = U[(size_t)e2 * L + z] - u0;
                v = V[(size_t)e2 * L + z] - v0;
            } else if (FREE_SLIP) {
                const real2 dxy = d.edge_dxdy[eds[j]];
                const real zc1 = dxy.x * d.elem_cos[e], zc2 = dxy.y;
                const real un = -real(2.0) * (u0 * zc2 - v0 * zc1) / (zc1 * zc1 + zc2 * zc2);
                const real ua = u0 + un * zc2;
                const real va = v0 - un * zc1;
                u = ua - u0;
                v = va - v0;
            } else {
                u = -real(2.0) * u0;
                v = -real(2.0) * v0;
            }
            a1 = a1 + gxa[j] * u;
            a2 = a2 + gya[j] * u;
            a3 = a3 + gxa[j] * v;
            a4 = a4 + gya[j] * v;
        }
        d.vgux[ii] = a1;
        d.vguy[ii] = a2;
        d.vgvx[ii] = a3;
        d.vgvy[ii] = a4;
    }
}

// viscosity_filt2x_3D (fv_viscosity.F90:570-670), first half: U_c of every
// (element, level) from the differences of U*Je with its neighbours
// (neighbour 4 only when it differs from neighbour 1), times K_bi.  velrhs
// forms UV_rhs from the neighbours' U_c.
__global__ void k_filt2x_uc(Dev d) {
    pdl_enter();
    const unsigned total = (unsigned)d.E * d.L;
    const int L = d.L;
    const real tau_inv = d.dt * d.tau_c / real(3600.0) / real(24.0);
    GRID_LOOP(ii, total) {
        const int e = d.by_L.div(ii);
        const int z = (int)ii - e * L;
        const int4 nb = d.elem_nb[e];
        const int nbs[4] = {nb.x, nb.y, nb.z, nb.w};
        const real K_bi = tau_inv * sqrt(scale_area_of(d, e) / d.elem_area[e]);
        const real uj = d.U_n[ii] * d.Je[ii], vj = d.V_n[ii] * d.Je[ii];
        real uc = real(0.0), vc = real(0.0);
        for (int j = 0; j < 4; ++j) {
            const int ne = nbs[j];
            if (!(ne >= 0 && (j < 3 || ne != nbs[0]))) continue;
            const size_t i2 = (size_t)ne * L + z;
            if (j == 0) {
                uc = uj - d.U_n[i2] * d.Je[i2];
                vc = vj - d.V_n[i2] * d.Je[i2];
            } else {
                uc = uc + uj - d.U_n[i2] * d.Je[i2];
                vc = vc + vj - d.V_n[i2] * d.Je[i2];
            }
        }
        d.f2U[ii] = uc * K_bi;
        d.f2V[ii] = vc * K_bi;
    }
}

// ---------------------------------------------------------------------------
// velrhs: compute_vel_rhs (fv_3D_vel.F90:1-180), one thread per (element,
// level) with levels on consecutive lanes.  Each warp takes 31 outputs and
// its lane 31 forms the vertical flux at its own index, the interface below
// lane 30's layer, so the flux at interface z+1 comes from the next lane
// for every output and no lane forms a second flux.
// ff = 1 on the very first call (lfirst), 1.5+epsilon afterwards.
// (Sharing the fluxes across the block through shared memory was measured
// 16 % slower than recomputing them: the block-wide barrier costs more.)
// The gathers of the edge fluxes and of the neighbours' velocities load all
// four before any is used; behind the tests of the sides one came after the
// other: 1.05 M nodes 1.36 -> 1.27 ms, 232 k FP32 0.257 -> 0.230, 42 k 0.098 ->
// 0.091.
// ---------------------------------------------------------------------------
// FP64: 4 resident blocks (at most 64 registers): the few spilled registers
// cost less than the lost warps (11 % faster than 3 blocks at 80 registers; 5
// blocks: 1.25 ms at 1.05 M nodes against 1.27, but 0.021 against 0.019 at 16
// k).  FP32: 8 blocks (32 registers), 232 k nodes 0.230 -> 0.160 ms; its
// latency is hidden by warps alone.
__global__ void __launch_bounds__(256, FESOMC_FP32 ? 8 : 4) k_velrhs(Dev d, real ff) {
    pdl_enter();
    const unsigned total = (unsigned)d.E * d.L;
    const int lane = threadIdx.x & 31;
    const unsigned nwarp = gridDim.x * (blockDim.x >> 5);
    for (unsigned c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c * 31 < total; c += nwarp) {
        const unsigned iw = c * 31 + lane;
        const bool valid = lane < 31 && iw < total;
        const unsigned ii = iw < total ? iw : total - 1;
        const int e = d.by_L.div(ii);
        const int z = (int)ii - e * d.L;
        const int L = d.L;
        const int4 en = d.elem_nodes[e];
        const real4 w = d.w_cv[e];
        const real ar = d.elem_area[e];
        const real je = d.Je[ii];
        // pressure force from eta_n (per element, from bpg_elem)
        const real2 F = d.Fp[e];
        const real Fx = F.x, Fy = F.y;
        const real un0 = d.U_n[ii], vn0 = d.V_n[ii];
        real ur = -(real(0.5) + d.epsilon) * d.U_rhsAB[ii] + Fx * je;
        real vr = -(real(0.5) + d.epsilon) * d.V_rhsAB[ii] + Fy * je;
        const real cor = d.coriolis[e];
        real uab = vn0 * cor * ar * je;
        real vab = -un0 * cor * ar * je;
        // horizontal upwind momentum advection (fv_advection.F90:114-188):
        // edge fluxes in edge order
        if (d.mom_adv_3D == 1) {
            const int4 il = d.elem_iedges[e];
            const int codes[4] = {il.x, il.y, il.z, il.w};   // absent ones (-1) last
            real2 f[4];   // loaded together, not one after the other behind the tests
#pragma unroll
            for (int c = 0; c < 4; ++c) {
#if FESOMC_FP32   // an edge again (adv3 holds one at least): 0.242 -> 0.230 ms at 232 k nodes
                f[c] = d.adv3[(size_t)(max(codes[c] < 0 ? codes[0] : codes[c], 0) >> 1) * L + z];
#else
                f[c] = codes[c] >= 0 ? d.adv3[(size_t)(codes[c] >> 1) * L + z] : make_real2(real(0.0), real(0.0));
#endif
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (codes[c] < 0) continue;
                if (codes[c] & 1) { uab = uab + f[c].x; vab = vab + f[c].y; }
                else { uab = uab - f[c].x; vab = vab - f[c].y; }
            }
        }
        // filter viscosity (fv_viscosity.F90:842-860)
        if (d.filt_3D) {
            const int4 nb = d.elem_nb[e];
            const int nbs[4] = {nb.x, nb.y, nb.z, nb.w};
            const int jend = (en.x == en.w) ? 3 : 4;
            real u1 = real(0.0), v1 = real(0.0);
            real un[4], vn[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const size_t i2 = nbs[j] >= 0 ? (size_t)nbs[j] * L + z : ii;
                un[j] = d.U_n[i2];
                vn[j] = d.V_n[i2];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (nbs[j] >= 0 && j < jend) {
                    u1 = u1 + un[j] - un0;
                    v1 = v1 + vn[j] - vn0;
                }
            ur = ur + d.tau_inv_filt * u1 * ar * je;
            vr = vr + d.tau_inv_filt * v1 * ar * je;
        }
        // biharmonic viscosity (fv_viscosity.F90:248-330): the pass-2 edge
        // fluxes in edge order, internal edges then boundary edges
        if (d.bih_3D) {
            const int4 se = d.elem_sedges[e];
            const int codes[4] = {se.x, se.y, se.z, se.w};
            for (int c = 0; c < 4; ++c) {
                const int code = codes[c];
                if (code < 0) break;
                const real2 f = d.bihfl[(size_t)(code >> 1) * L + z];
                if (code & 1) { ur = ur - f.x; vr = vr - f.y; }
                else { ur = ur + f.x; vr = vr + f.y; }
            }
        }
        // vertical advection (fv_advection.F90:354-469): flux at interface z
        // here, at z+1 from the next lane (same element) or computed
        const real mwd = d.mask_wd[e];
        if (d.vert_adv == 1) {
            real fu0, fv0;
            uvert_at(d, e, z, w, en, ar, fu0, fv0);
            real fu1 = __shfl_down_sync(kFull, fu0, 1), fv1 = __shfl_down_sync(kFull, fv0, 1);
            if (z == L - 1) { fu1 = real(0.0); fv1 = real(0.0); }   // the bottom interface carries no flux
            if (mwd != real(0.0)) {
                const real acc = d.elem_acc[e];
                uab = uab + (fu0 - fu1) * acc;
                vab = vab + (fv0 - fv1) * acc;
            } else {
                uab = real(0.0);
                vab = real(0.0);
            }
        }
        if (valid) {
            d.U_rhsAB[ii] = uab;
            d.V_rhsAB[ii] = vab;
            const real area_inv = real(1.0) / ar;
            const real dt = d.dt;
            // UV_rhs of viscosity_filt2x_3D (zero when it is off)
            real uvx = real(0.0), uvy = real(0.0);
            if (d.filt_bi_3D) {
                const int4 nb = d.elem_nb[e];
                const int nbs[4] = {nb.x, nb.y, nb.z, nb.w};
                const real uc = d.f2U[ii], vc = d.f2V[ii];
                for (int j = 0; j < 4; ++j) {
                    const int ne = nbs[j];
                    if (!(ne >= 0 && (j < 3 || ne != nbs[0]))) continue;
                    const size_t i2 = (size_t)ne * L + z;
                    if (j == 0) { uvx = -uc + d.f2U[i2]; uvy = -vc + d.f2V[i2]; }
                    else { uvx = uvx - uc + d.f2U[i2]; uvy = uvy - vc + d.f2V[i2]; }
                }
            }
            d.U_rhs[ii] = mwd * (un0 + d.Bar_pru[ii] * dt + (dt * (ur + uab * ff) * area_inv + uvx) / je);
            d.V_rhs[ii] = mwd * (vn0 + d.Bar_prv[ii] * dt + (dt * (vr + vab * ff) * area_inv + uvy) / je);
        }
    }
}

// ---------------------------------------------------------------------------
// implvisc: momentum_vert_impl_visc (fv_viscosity.F90:1266-1371), thread per
// column; the fic variant is k_implvisc_fic_tile or k_implvisc_fic_reg.
// ---------------------------------------------------------------------------
template <int MAXL>
__global__ void k_implvisc(Dev d) {
    pdl_enter();
    GRID_LOOP(ii, d.E) {
        const int e = (int)ii;
        const int L = d.L, NS = d.NS;
        real *ur = d.U_rhs + (size_t)e * L;
        real *vr = d.V_rhs + (size_t)e * L;
        const real *Av = d.Av + (size_t)e * NS;
        const real mwd = d.mask_wd[e];
        const real dt = d.dt;
        const real ub = d.U_n[(size_t)e * L + L - 1], vb = d.V_n[(size_t)e * L + L - 1];
        const real a_Cd = d.C_d * ((real(1.0) - d.elem_acc[e]) * d.Cd_bz + real(1.0));
        const real *je = d.Je + (size_t)e * L;
        real a[MAXL], b[MAXL], c[MAXL], cp[MAXL], up[MAXL], vp[MAXL], uu[MAXL], vv[MAXL];
        const real *zc = d.Ze + (size_t)e * L;
        for (int z = 1; z <= L - 2; ++z) {
            const real zinv = dt / je[z];
            a[z] = -Av[z] / (zc[z] - zc[z - 1]) * zinv;
            c[z] = -Av[z + 1] / (zc[z + 1] - zc[z]) * zinv;
            b[z] = -a[z] - c[z] + real(1.0);
        }
        real zinv = dt / je[L - 1];
        a[L - 1] = -Av[L - 1] / (zc[L - 1] - zc[L - 2]) * zinv;
        b[L - 1] = -a[L - 1] + real(1.0);
        c[L - 1] = real(0.0);
        zinv = dt / je[0];
        c[0] = -Av[1] / (zc[1] - zc[0]) * zinv;
        a[0] = real(0.0);
        b[0] = -c[0] + real(1.0);
        for (int z = 0; z < L; ++z) { uu[z] = ur[z]; vv[z] = vr[z]; }
        uu[0] = uu[0] + zinv * d.taux[e] / d.density_0;
        vv[0] = vv[0] + zinv * d.tauy[e] / d.density_0;
        zinv = dt / je[L - 1];
        const real friction = -a_Cd * sqrt(ub * ub + vb * vb);
        uu[L - 1] = uu[L - 1] + zinv * friction * ub;
        vv[L - 1] = vv[L - 1] + zinv * friction * vb;
        // the recurrences carry their last value in registers
        real cpv = c[0] / b[0], upv = uu[0] / b[0], vpv = vv[0] / b[0];
        cp[0] = cpv;
        up[0] = upv;
        vp[0] = vpv;
        for (int z = 1; z < L; ++z) {
            const real az = a[z];
            const real m = b[z] - cpv * az;
            cpv = c[z] / m;
            upv = (uu[z] - upv * az) / m;
            vpv = (vv[z] - vpv * az) / m;
            cp[z] = cpv;
            up[z] = upv;
            vp[z] = vpv;
        }
        real un = upv, vn = vpv;
        uu[L - 1] = un;
        vv[L - 1] = vn;
        for (int z = L - 2; z >= 0; --z) {
            un = up[z] - cp[z] * un;
            vn = vp[z] - cp[z] * vn;
            uu[z] = un;
            vv[z] = vn;
        }
        for (int z = 0; z < L; ++z) { ur[z] = uu[z] * mwd; vr[z] = vv[z] * mwd; }
    }
}

// after the sub-cycle: the last sub-step's rotation of the elevation's time
// levels (fv_main.F90:1547-1551; those before it are made by the next
// sub-step's ssh_node), and the elevation of the jacobian call
// (fv_main.F90:2050)
__global__ void k_jac_swap(Dev d) {
    pdl_enter();
    GRID_LOOP(ii, d.N) {
        const double e0 = d.eta_n[ii], e1 = d.eta_n_1[ii], en = d.eta_new[ii];
        d.eta_n_2[ii] = e1;
        d.eta_n_1[ii] = e0;
        d.eta_n[ii] = en;
        d.eta_jac[ii] = en;
    }
}

// Je, Ze, ZBe of every (element, level) from eta_jac (jacobian,
// fv_main.F90:1208-1267); at init, afterwards refreshed by update3d
__global__ void k_je_elem(Dev d) {
    pdl_enter();
    const unsigned total = (unsigned)d.E * d.L;
    GRID_LOOP(ii, total) {
        const int e = d.by_L.div(ii);
        const int z = (int)ii - e * d.L;
        const real4 w = d.w_cv[e];
        const real4 a = elem_jac_a(d, d.eta_jac, d.elem_nodes[e]);
        d.Je[ii] = je_of(d, w, a, z);
        d.Ze[ii] = wsum_z(d, w, a, z);
        d.ZBe[ii] = wsum_zbar(d, w, a, z);
    }
}

// update_3D_vel (fv_3D_vel.F90:201-255) with the U_filt averaging of
// oce_barotropic_timestep (fv_main.F90:1670-1677) folded in; column block
// per element.  Runs right after the jacobian call: the stored Je still holds
// the previous jacobian (Jc_old), and is replaced here by the new Je / Ze /
// ZBe.
// FP64: 48 registers (40: 0.62 ms, 32: 0.70 against 0.60 at 1.05 M nodes); FP32:
// 32, 232 k nodes 0.095 -> 0.087.
// The element's scalars are formed by four lanes per element, one per node.
// Blocks of 160 threads: 1.05 M nodes 0.80 -> 0.60 ms, 232 k FP32 0.131 ->
// 0.095, 40 k, 30 layers 0.059 -> 0.039 (one lane per element formed them, 320
// threads).
constexpr int kU3Sc = 16;  // per element: w_cv(4), a(4), U2p, V2p, uf, vf, U_n_2D(2), dmean_inv; then dh(4)
__global__ void __maxnreg__(FESOMC_FP32 ? 32 : 48) k_update3d(Dev d, real Mt_inv) {
    pdl_enter();
    extern __shared__ __align__(16) unsigned char sm_raw[];
    real *sm = reinterpret_cast<real *>(sm_raw);
    const int L = d.L;
    const ColBlock cb(d);
    const int S = 2 * L + 1, B = cb.B;
    real *const sc = sm + (size_t)B * S, *const dhs = sc + (size_t)B * kU3Sc;
    for (long long eb = (long long)blockIdx.x * B; eb < d.E; eb += (long long)gridDim.x * B) {
        const long long e_ = eb + cb.jl;
        const bool act = cb.jl < B && e_ < d.E;
        const size_t i = (size_t)e_ * L + cb.z;
        real a_old = real(0.0), ur = real(0.0), vr = real(0.0);
        if (act) {
            a_old = d.Je[i];
            ur = d.U_rhs[i];
            vr = d.V_rhs[i];
        }
        // the element's scalars, here rather than in the serial sum or the
        // level loop, so that both read shared memory only
        if ((int)threadIdx.x < 4 * B) {
            const int j = threadIdx.x >> 2, k = threadIdx.x & 3;
            const int e = (int)(eb + j < d.E ? eb + j : d.E - 1);
            const int n = reinterpret_cast<const int *>(d.elem_nodes)[4 * (size_t)e + k];
            real *o = sc + kU3Sc * j;
            o[k] = reinterpret_cast<const real *>(d.w_cv)[4 * (size_t)e + k];
            dhs[4 * j + k] = d.depth[n] + d.eta_n[n];
            o[4 + k] = jac_a(d, d.eta_jac, n);
            if (k < 2) o[12 + k] = reinterpret_cast<const real *>(d.U_n_2D)[2 * (size_t)e + k];
            __syncwarp(lanes_below(4 * B));
            if (k < 2 && eb + j < d.E) {
                const real4 w = make_real4(o[0], o[1], o[2], o[3]);
                const real dmean_inv = real(1.0) / dmax(d.Dmin, wsum(w, dhs[4 * j], dhs[4 * j + 1], dhs[4 * j + 2], dhs[4 * j + 3]));
                real *const F = k ? d.V_filt_2D : d.U_filt_2D;
                const real f = (F[e] * Mt_inv) * dmean_inv;
                F[e] = f;
                o[10 + k] = f;
                if (k == 0) o[14] = dmean_inv;
            }
        }
        if (act) {
            sm[cb.jl * S + cb.z] = ur * a_old;
            sm[cb.jl * S + L + cb.z] = vr * a_old;
        }
        __syncthreads();
        // one thread per (element, component): the level sums in level order
        if ((int)threadIdx.x < 2 * B && eb + (threadIdx.x >> 1) < d.E) {
            const int j = threadIdx.x >> 1, c = threadIdx.x & 1;
            const real *row = sm + j * S + c * L;
            real su = real(0.0);
            for (int k = 0; k < L; ++k) su = su + row[k];
            real *o = sc + kU3Sc * j;
            o[8 + c] = su * o[14];
        }
        __syncthreads();
        if (act) {
            const int z = cb.z;
            const real *o = sc + kU3Sc * cb.jl;
            const real U2p = o[8], V2p = o[9], uf = o[10], vf = o[11];
            const real4 w = make_real4(o[0], o[1], o[2], o[3]);
            const real4 an = make_real4(o[4], o[5], o[6], o[7]);
            const real jn = je_of(d, w, an, z);
            const real az = a_old / jn;
            d.U_n_filt[i] = az * ur + uf - U2p;
            d.V_n_filt[i] = az * vr + vf - V2p;
            d.U_n[i] = az * ur + o[12] - U2p;
            d.V_n[i] = az * vr + o[13] - V2p;
            d.Je[i] = jn;
            d.Ze[i] = wsum_z(d, w, an, z);
            d.ZBe[i] = wsum_zbar(d, w, an, z);
        }
        __syncthreads();
    }
}

// vert_vel_sigma (fv_3D_vel.F90:309-456): column block per node; the layer
// transport divergence of (node, level) gathered over the node's edges in
// edge order, then summed upward from the bottom per node.  The edge lists
// of a block's consecutive nodes are one contiguous range: its entries (side,
// elements, edge_cross, the elements' filtered 2D velocities; three dependent
// loads, the same for all levels) are staged in shared memory, kWvEdges per
// node on average; a block with more reads them where they are used.
// Blocks of 160 threads: 1.05 M nodes 0.82 -> 0.69 ms, 232 k FP32 0.167 ->
// 0.134, 40 k, 30 layers 0.070 -> 0.050.
constexpr int kWvEdges = 8;
struct WvEdge {
    real X[4], uf1, vf1, uf2, vf2;
    int code, e1, e2, pad;
};
__device__ __forceinline__ WvEdge wv_edge(const Dev &d, int p) {
    WvEdge w;
    w.code = d.node_eidx[p];
    const int ed = w.code >> 1;
    const int2 et = d.edge_tri[ed];
    const real4 X = d.edge_cross[ed];
    w.X[0] = X.x; w.X[1] = X.y; w.X[2] = X.z; w.X[3] = X.w;
    w.e1 = et.x;
    w.e2 = ed < d.Ed_in ? et.y : -1;
    w.uf1 = d.U_filt_2D[et.x];
    w.vf1 = d.V_filt_2D[et.x];
    w.uf2 = w.e2 >= 0 ? d.U_filt_2D[et.y] : real(0.0);
    w.vf2 = w.e2 >= 0 ? d.V_filt_2D[et.y] : real(0.0);
    return w;
}
__device__ __forceinline__ real wv_add(const Dev &d, real W, const WvEdge &w, int z) {
    const size_t i1 = (size_t)w.e1 * d.L + z;
    real c1 = d.Je[i1] * ((d.V_n_filt[i1] - w.vf1) * w.X[0] - (d.U_n_filt[i1] - w.uf1) * w.X[1]);
    if (w.e2 >= 0) {
        const size_t i2 = (size_t)w.e2 * d.L + z;
        c1 = c1 + d.Je[i2] * (-(d.V_n_filt[i2] - w.vf2) * w.X[2] + (d.U_n_filt[i2] - w.uf2) * w.X[3]);
    }
    return (w.code & 1) ? W - c1 : W + c1;
}
__global__ void k_wvel(Dev d) {
    pdl_enter();
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const int L = d.L, NS = d.NS;
    const ColBlock cb(d);
    const int S = L | 1, B = cb.B;
    WvEdge *const ed = reinterpret_cast<WvEdge *>(sm_raw);   // kWvEdges * B entries
    real *const sm = reinterpret_cast<real *>(ed + kWvEdges * B);
    real *const sc = sm + (size_t)B * S;  // per node: bottom Wvel, 1/area
    for (long long nb = (long long)blockIdx.x * B; nb < d.N; nb += (long long)gridDim.x * B) {
        const long long n_ = nb + cb.jl;
        const bool act = cb.jl < B && n_ < d.N;
        const int q0 = d.node_eptr[nb], q1 = d.node_eptr[nb + B < d.N ? nb + B : d.N];
        const bool staged = q1 - q0 <= kWvEdges * B;
        if (staged)
            for (int t = threadIdx.x; t < q1 - q0; t += blockDim.x) ed[t] = wv_edge(d, q0 + t);
        if (act && cb.z == 0) {
            sc[2 * cb.jl] = d.Wvel[(size_t)n_ * NS + NS - 1];
            sc[2 * cb.jl + 1] = real(1.0) / d.area[n_];
        }
        int p0 = 0, p1 = 0;
        if (act) {
            p0 = d.node_eptr[n_];
            p1 = d.node_eptr[n_ + 1];
        }
        __syncthreads();
        if (act) {
            real W = real(0.0);
            if (staged) {
#pragma unroll 4
                for (int p = p0; p < p1; ++p) W = wv_add(d, W, ed[p - q0], cb.z);
            } else {
                for (int p = p0; p < p1; ++p) W = wv_add(d, W, wv_edge(d, p), cb.z);
            }
            sm[cb.jl * S + cb.z] = W;
        }
        __syncthreads();
        const long long ns = nb + threadIdx.x;
        if ((int)threadIdx.x < B && ns < d.N) {
            real *row = sm + threadIdx.x * S;
            real below = sc[2 * threadIdx.x];
            for (int k = L - 1; k >= 0; --k) {
                below = row[k] + below;
                row[k] = below;
            }
        }
        __syncthreads();
        if (act) d.Wvel[(size_t)n_ * NS + cb.z] = sm[cb.jl * S + cb.z] * sc[2 * cb.jl + 1];
        __syncthreads();
    }
}

// ---- momentum_vert_impl_visc_tmp on tiles of element columns --------------
// (fv_viscosity.F90:1374-1486, no ice.)  A block takes kIvCols (32) consecutive
// elements, whose columns are one contiguous range of U_rhs, V_rhs, Je and
// Av.  All threads, one (element, layer) each: the staging, the coefficients a
// and c with their three divisions, and at the end the masked result.  The
// elimination (three quotients per layer by the same denominator) and the back
// substitution run from shared memory, [array][layer][column] with an odd
// column stride: free of bank conflicts both over the columns of a layer and
// over the layers of a column.  c, U and V are overwritten by xx1, yu and yv,
// then by the solution.
// Bound by latency: the chain of the elimination, whose FP64 divisions (114
// cycles each) one thread runs one after the other.  So in FP64 four lanes per
// column form the quotients of xx1, yu and yv at
// the same time; FP32, whose divisions are short, takes one thread per column.
// Staging (FP64): kIvBatch items per thread, the neighbour layers' Je and Av
// again from L1 instead of staged, so that four arrays remain and more blocks
// are resident; FP32 was slower with batches (0.060 -> 0.064 ms).
// FP64, against one thread per column reading global memory, and against
// tiles with one thread per column: 1.05 M nodes, 20 layers 0.68, 0.62 ->
// 0.43 ms, 232 k 0.185, 0.148 -> 0.107, 42 k 0.035, 0.040 -> 0.029, 40 k, 30
// layers 0.049, 0.064 -> 0.043, 16 k, 10 layers 0.017, 0.016 -> 0.013, 4.5 k,
// 39 layers 0.032, 0.025 -> 0.019.
// A column takes 32 B of shared memory per layer (FP64): where 32 of them
// leave an SM fewer than four blocks (55 layers on) a block takes 16, and 256
// threads, four times as many as its recurrences need, for the staging and its
// divisions; where 16 leave fewer than four (106 layers on) 8, and 128.  16 k
// nodes, 80 layers 0.091 -> 0.051 ms, 149 k nodes, 55 layers 0.328 -> 0.278, 69
// layers 0.404 -> 0.338, 100 k nodes, 80 layers 0.429 -> 0.260, 126 layers 1.235 ->
// 0.55 (one thread per column 0.416, 0.710; 16 columns with 64 threads 0.849, with
// 128 0.660, with 256 0.562); 8 columns with 128 threads at 74 layers 0.362 against
// 0.355.
#if !FESOMC_FP32
constexpr int kIvBatch = 3;
#endif

template <int kIvCols, int kIvThreads>
__global__ void __launch_bounds__(kIvThreads) k_implvisc_fic_tile(Dev d) {
    pdl_enter();
    extern __shared__ __align__(16) unsigned char iv_smem[];
    constexpr int CP = kIvCols + 1;
    const int L = d.L, NS = d.NS, E = d.E;
    const int A = L * CP;
    real *const sa = reinterpret_cast<real *>(iv_smem);   // layer z of column j at [z * CP + j]
    real *const sc = sa + A, *const sU = sa + 2 * A, *const sV = sa + 3 * A;
    const real dt = d.dt;
#if FESOMC_FP32
    // the warps of the recurrences alternate between the blocks of an SM
    constexpr int kChains = kIvCols / 32, kWarps = kIvThreads / 32;
    const int warp = (int)(threadIdx.x / 32 + kChains * (blockIdx.x / 148)) % kWarps;
    const bool mine = warp < kChains;
    const int lane = warp * 32 + (threadIdx.x & 31);   // column of a recurrence
#else
    static_assert(kIvThreads >= 4 * kIvCols && kIvCols % 8 == 0, "four lanes per column, all of a warp");
#endif
    for (int e0 = blockIdx.x * kIvCols; e0 < E; e0 += gridDim.x * kIvCols) {
        const int nt = E - e0 < kIvCols ? E - e0 : kIvCols;
#if FESOMC_FP32
        for (int i = threadIdx.x; i < nt * L; i += kIvThreads) {
            const int j = d.by_L.div(i), z = i - j * L, o = z * CP + j;
            const size_t g = (size_t)e0 * L + i, ga = g + e0 + j;
            const real jz = d.Je[g];
            const real d1 = (z == 0) ? real(0.5) * jz : real(0.5) * (jz + d.Je[g - 1]);
            const real d2 = (z == L - 1) ? real(0.5) * jz : real(0.5) * (jz + d.Je[g + 1]);
            const real zt = dt / jz;
            sa[o] = zt * d.Av[ga] / d1;
            sc[o] = zt * d.Av[ga + 1] / d2;
            sU[o] = d.U_rhs[g];
            sV[o] = d.V_rhs[g];
        }
#else
        // kIvBatch items per thread loaded before any is used
        for (int i0 = threadIdx.x; i0 < nt * L; i0 += kIvBatch * kIvThreads) {
            real ur[kIvBatch], vr[kIvBatch], j0[kIvBatch], jm[kIvBatch], jp[kIvBatch], a0[kIvBatch], a1[kIvBatch];
#pragma unroll
            for (int u = 0; u < kIvBatch; ++u) {
                const int i = i0 + u * kIvThreads < nt * L ? i0 + u * kIvThreads : i0;
                const int j = d.by_L.div(i), z = i - j * L;
                const size_t g = (size_t)e0 * L + i;
                ur[u] = d.U_rhs[g];
                vr[u] = d.V_rhs[g];
                j0[u] = d.Je[g];
                jm[u] = d.Je[z > 0 ? g - 1 : g];
                jp[u] = d.Je[z < L - 1 ? g + 1 : g];
                a0[u] = d.Av[g + e0 + j];
                a1[u] = d.Av[g + e0 + j + 1];
            }
#pragma unroll
            for (int u = 0; u < kIvBatch; ++u) {
                const int i = i0 + u * kIvThreads;
                if (i >= nt * L) break;
                const int j = d.by_L.div(i), z = i - j * L, o = z * CP + j;
                sU[o] = ur[u];
                sV[o] = vr[u];
                const real jz = j0[u];
                const real d1 = (z == 0) ? real(0.5) * jz : real(0.5) * (jz + jm[u]);
                const real d2 = (z == L - 1) ? real(0.5) * jz : real(0.5) * (jz + jp[u]);
                const real zt = dt / jz;
                sa[o] = zt * a0[u] / d1;
                sc[o] = zt * a1[u] / d2;
            }
        }
#endif
        __syncthreads();
#if FESOMC_FP32
        if (mine && lane < nt) {
            const int e = e0 + lane;
            const real mwd = d.mask_wd[e];
            real *a_ = sa + lane, *x_ = sc + lane, *u_ = sU + lane, *v_ = sV + lane;
            if (mwd != real(0.0)) {
                const real *J = d.Je + (size_t)e * L, *Av = d.Av + (size_t)e * NS;
                const real ub = d.U_n[(size_t)e * L + L - 1], vb = d.V_n[(size_t)e * L + L - 1];
                const real a_Cd = d.C_d * ((real(1.0) - d.elem_acc[e]) * d.Cd_bz + real(1.0));
                real de = J[0] / (Av[0] + Av[1]);
                const real rw = de / d.density_0;
                real xv = real(1.0), yuv = d.taux[e] * rw, yvv = d.tauy[e] * rw;
                const real jb = J[L - 1], av0 = Av[NS - 1], av1 = Av[L - 1];   // loaded ahead of the sweep
                real an = a_[0], cn = x_[0], un = u_[0], vn = v_[0];
                for (int z = 0; z < L; ++z) {
                    const real a = an, c = cn, Fx = un, Fy = vn;
                    const int zn = (z + 1 < L ? z + 1 : z) * CP;
                    an = a_[zn]; cn = x_[zn]; un = u_[zn]; vn = v_[zn];
                    const real b = a + c + real(1.0);
                    const real dd = b - a * xv;
                    xv = c / dd;
                    yuv = (a * yuv + Fx) / dd;
                    yvv = (a * yvv + Fy) / dd;
                    x_[z * CP] = xv;
                    u_[z * CP] = yuv;
                    v_[z * CP] = yvv;
                }
                de = jb / (av0 + av1);
                const real friction = de * a_Cd * sqrt(ub * ub + vb * vb);
                real Ut, Vt;
                if (d.fic_point == 0) { Ut = real(0.0); Vt = real(0.0); }
                else if (d.fic_point == 1) {
                    const real a = friction + real(1.0) - xv;
                    Ut = yuv / a; Vt = yvv / a;
                } else {
                    const real a = real(1.0) / (real(1.0) - friction) - xv;
                    Ut = yuv / a; Vt = yvv / a;
                }
                for (int z = L - 1; z >= 0; --z) {
                    const real x = x_[z * CP];
                    Ut = Ut * x + u_[z * CP];
                    Vt = Vt * x + v_[z * CP];
                    u_[z * CP] = Ut * mwd;
                    v_[z * CP] = Vt * mwd;
                }
            } else {
                for (int z = 0; z < L; ++z) { u_[z * CP] = real(0.0); v_[z * CP] = real(0.0); }
            }
        }
#else
        if (threadIdx.x < 4 * kIvCols) {
            // four lanes per column: xx1, yu and yv form their quotient each
            // at the same time and share xx1 (__shfl needs every lane: those
            // past the last column run along on column 0, the fourth lane on
            // yv; what they form is not used)
            const int role = threadIdx.x & 3, col = threadIdx.x >> 2;
            const bool in = col < nt;
            const int c0 = in ? col : 0, e = e0 + c0;
            const real mwd = d.mask_wd[e];
            const real *a_ = sa + c0, *J = d.Je + (size_t)e * L, *Av = d.Av + (size_t)e * NS;
            real *x_ = sc + c0, *const y_ = (role == 0 ? sc : role == 1 ? sU : sV) + c0;
            const bool out = in && role < 3;
            const real ub = d.U_n[(size_t)e * L + L - 1], vb = d.V_n[(size_t)e * L + L - 1];
            const real a_Cd = d.C_d * ((real(1.0) - d.elem_acc[e]) * d.Cd_bz + real(1.0));
            const real rw = J[0] / (Av[0] + Av[1]) / d.density_0;
            const real jb = J[L - 1], av0 = Av[NS - 1], av1 = Av[L - 1];
            real x = real(1.0), y = (role == 1 ? d.taux[e] : d.tauy[e]) * rw;
            real an = a_[0], cn = x_[0], fn = y_[0];
            for (int z = 0; z < L; ++z) {
                const real a = an, c = cn, F = fn;
                const int zn = (z + 1 < L ? z + 1 : z) * CP;
                an = a_[zn]; cn = x_[zn]; fn = y_[zn];
                const real b = a + c + real(1.0);
                const real q = (role == 0 ? c : a * y + F) / (b - a * x);
                x = __shfl_sync(kFull, q, threadIdx.x & 28);
                y = q;
                if (out) y_[z * CP] = q;
            }
            __syncwarp();
            if (out && role > 0) {
                const real de = jb / (av0 + av1);
                const real friction = de * a_Cd * sqrt(ub * ub + vb * vb);
                real W = real(0.0);
                if (d.fic_point == 1) W = y / (friction + real(1.0) - x);
                else if (d.fic_point != 0) W = y / (real(1.0) / (real(1.0) - friction) - x);
                if (mwd != real(0.0)) {
                    for (int z = L - 1; z >= 0; --z) {
                        W = W * x_[z * CP] + y_[z * CP];
                        y_[z * CP] = W * mwd;
                    }
                } else {
                    for (int z = 0; z < L; ++z) y_[z * CP] = real(0.0);
                }
            }
        }
#endif
        __syncthreads();
        for (int i = threadIdx.x; i < nt * L; i += kIvThreads) {
            const int j = d.by_L.div(i), z = i - j * L;
            const size_t g = (size_t)e0 * L + i;
            d.U_rhs[g] = sU[z * CP + j];
            d.V_rhs[g] = sV[z * CP + j];
        }
        __syncthreads();
    }
}
// The fic variant on tiles of 64 element columns with the layer count LC fixed
// at compile time (4 to 10): all threads stage U_rhs, V_rhs, Je and Av of the
// block's consecutive elements with batched loads, one thread per column
// solves with its recurrences in registers, from rows of odd stride.  The
// arithmetic and its order are k_implvisc_fic_tile's.
constexpr int kIrCols = 64;
template <int LC>
__global__ void __launch_bounds__(kIrCols) k_implvisc_fic_reg(Dev d) {
    pdl_enter();
    extern __shared__ __align__(16) unsigned char iv_smem[];
    constexpr int L = LC, LP = LC | 1, NS = LC + 1, KP = NS | 1, C = kIrCols, kB = 4;
    const int E = d.E;
    real *sU = reinterpret_cast<real *>(iv_smem);   // row j: element e0 + j
    real *sV = sU + C * LP, *sJ = sV + C * LP, *sA = sJ + C * LP;
    const real dt = d.dt;
    for (int e0 = blockIdx.x * C; e0 < E; e0 += gridDim.x * C) {
        const int nt = E - e0 < C ? E - e0 : C;
        for (int i0 = threadIdx.x; i0 < nt * NS; i0 += kB * C) {
            real av[kB];
#pragma unroll
            for (int u = 0; u < kB; ++u) {
                const int i = i0 + u * C;
                av[u] = i < nt * NS ? d.Av[(size_t)e0 * NS + i] : real(0.0);
            }
#pragma unroll
            for (int u = 0; u < kB; ++u) {
                const int i = i0 + u * C, j = i / NS;
                if (i < nt * NS) sA[j * KP + (i - j * NS)] = av[u];
            }
        }
        for (int i0 = threadIdx.x; i0 < nt * L; i0 += kB * C) {
            real ur[kB], vr[kB], jv[kB];
#pragma unroll
            for (int u = 0; u < kB; ++u) {
                const int i = i0 + u * C;
                const size_t g = (size_t)e0 * L + (i < nt * L ? i : 0);
                ur[u] = d.U_rhs[g];
                vr[u] = d.V_rhs[g];
                jv[u] = d.Je[g];
            }
#pragma unroll
            for (int u = 0; u < kB; ++u) {
                const int i = i0 + u * C;
                if (i >= nt * L) continue;
                const int j = i / L, z = i - j * L;
                sU[j * LP + z] = ur[u];
                sV[j * LP + z] = vr[u];
                sJ[j * LP + z] = jv[u];
            }
        }
        __syncthreads();
        if ((int)threadIdx.x < nt) {
            const int j = threadIdx.x, e = e0 + j;
            real *U = sU + j * LP, *V = sV + j * LP;
            const real *J = sJ + j * LP, *A = sA + j * KP;
            const real mwd = d.mask_wd[e];
            if (mwd != real(0.0)) {
                const real ub = d.U_n[(size_t)e * L + L - 1], vb = d.V_n[(size_t)e * L + L - 1];
                const real a_Cd = d.C_d * ((real(1.0) - d.elem_acc[e]) * d.Cd_bz + real(1.0));
                real xx1[LC + 1], yu[LC + 1], yv[LC + 1];
                real de = J[0] / (A[0] + A[1]);
                const real rw = de / d.density_0;
                real xv = real(1.0), yuv = d.taux[e] * rw, yvv = d.tauy[e] * rw;
                xx1[0] = xv;
                yu[0] = yuv;
                yv[0] = yvv;
#pragma unroll
                for (int z = 0; z < L; ++z) {
                    const real jz = J[z];
                    const real d1 = (z == 0) ? real(0.5) * jz : real(0.5) * (jz + J[z > 0 ? z - 1 : 0]);
                    const real d2 = (z == L - 1) ? real(0.5) * jz : real(0.5) * (jz + J[z + 1 < L ? z + 1 : z]);
                    const real zt = dt / jz;
                    const real a = zt * A[z] / d1;
                    const real c = zt * A[z + 1] / d2;
                    const real b = a + c + real(1.0);
                    const real dd = b - a * xv;
                    xv = c / dd;
                    yuv = (a * yuv + U[z]) / dd;
                    yvv = (a * yvv + V[z]) / dd;
                    xx1[z + 1] = xv;
                    yu[z + 1] = yuv;
                    yv[z + 1] = yvv;
                }
                de = J[L - 1] / (A[NS - 1] + A[L - 1]);
                const real friction = de * a_Cd * sqrt(ub * ub + vb * vb);
                real Ut, Vt;
                if (d.fic_point == 0) { Ut = real(0.0); Vt = real(0.0); }
                else if (d.fic_point == 1) {
                    const real a = friction + real(1.0) - xx1[L];
                    Ut = yu[L] / a; Vt = yv[L] / a;
                } else {
                    const real a = real(1.0) / (real(1.0) - friction) - xx1[L];
                    Ut = yu[L] / a; Vt = yv[L] / a;
                }
#pragma unroll
                for (int z = L - 1; z >= 0; --z) {
                    Ut = Ut * xx1[z + 1] + yu[z + 1];
                    Vt = Vt * xx1[z + 1] + yv[z + 1];
                    U[z] = Ut * mwd;
                    V[z] = Vt * mwd;
                }
            } else {
#pragma unroll
                for (int z = 0; z < L; ++z) { U[z] = real(0.0); V[z] = real(0.0); }
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < nt * L; i += C) {
            const int j = i / L, z = i - j * L;
            const size_t g = (size_t)e0 * L + i;
            d.U_rhs[g] = sU[j * LP + z];
            d.V_rhs[g] = sV[j * LP + z];
        }
        __syncthreads();
    }
}
static void (*implvisc_reg_kernel(const Dev &d))(Dev) {
    switch (d.L) {
        case 4: return k_implvisc_fic_reg<4>;
        case 5: return k_implvisc_fic_reg<5>;
        case 6: return k_implvisc_fic_reg<6>;
        case 7: return k_implvisc_fic_reg<7>;
        case 8: return k_implvisc_fic_reg<8>;
        case 9: return k_implvisc_fic_reg<9>;
        default: return k_implvisc_fic_reg<10>;
    }
}
static size_t implvisc_reg_smem(const Dev &d) { return (size_t)kIrCols * (3 * (d.L | 1) + (d.NS | 1)) * sizeof(real); }
// Few layers leave the level-parallel tiles little to share between their
// barriers: the register tiles from five of them per SM on, three in FP32
// (elements; ms at nodes, register / level-parallel tiles): 10 layers 40 k nodes 0.0183 /
// 0.0198, 1.0 M 0.229 / 0.251, FP32 40 k 0.0126 / 0.0138, 100 k 0.0164 / 0.0228,
// 1.0 M 0.095 / 0.127; 5 layers 1.0 M 0.101 / 0.176, FP32 0.054 / 0.088; 24 k
// nodes 0.0166 / 0.0149, FP32 6 layers 0.0085 / 0.0103.
static bool implvisc_reg(const Dev &d) { return d.L >= 4 && d.L <= 10 && d.E >= (FESOMC_FP32 ? 3 : 5) * 148 * kIrCols; }
static size_t implvisc_tile_smem(const Dev &d, int cols) { return (size_t)4 * d.L * (cols + 1) * sizeof(real); }
// columns of a tile
static int implvisc_cols(const Dev &d) {
    if (FESOMC_FP32 || implvisc_tile_smem(d, 32) <= 56 * 1024) return 32;
    return implvisc_tile_smem(d, 16) <= 56 * 1024 ? 16 : 8;
}
static void (*implvisc_tile_kernel(const Dev &d))(Dev) {
#if !FESOMC_FP32
    if (implvisc_cols(d) == 16) return k_implvisc_fic_tile<16, 256>;
    if (implvisc_cols(d) == 8) return k_implvisc_fic_tile<8, 128>;
#endif
    return k_implvisc_fic_tile<32, 128>;
}

// ---- launch wrappers --------------------------------------------------------
// Column blocks: B entities, B * L threads, about 160 of them (at most 16
// entities): the barriers between staging, levels and level sums then hold
// up 5 warps of an SM's 40, not 10 of 30 (blocks of 320 threads, 1.05 M nodes:
// update3d 0.63 against 0.60 ms, wvel 0.78 / 0.69).  The grid is the blocks
// resident at once; they stride over the entities.
static int col_b(const Dev &d) {
    return d.tune[TK_COLUMNS] > 0 ? d.tune[TK_COLUMNS] : default_columns(d.L);
}
// pressure_col's level sums take one lane per column, and its blocks do little
// else: four columns where the others take one or two.  100 k nodes, FP32: 54
// layers 0.064 -> 0.054 ms, 100 layers 0.144 -> 0.103, 126 layers 0.161 -> 0.126,
// FP64 0.100 -> 0.091, 0.222 -> 0.168, 0.251 -> 0.249.  Fewer layers: the count
// that fills its warps, 149 k nodes, 44 layers 0.113 -> 0.103 ms, FP32 0.073 ->
// 0.062, 27 layers 0.069 -> 0.064 (the others' barriers want small blocks).
static int pressure_b(const Dev &d) {
    if (d.tune[TK_COLUMNS] > 0) return col_b(d);
    return d.L > 53 ? 4 : filled_columns(d.L, default_columns(d.L));
}
static size_t pressure_smem(const Dev &d) { return (size_t)pressure_b(d) * (d.L | 1) * sizeof(real); }
static size_t bpg_smem(const Dev &d) {
    return (size_t)col_b(d) * (kEsReals + 12 + 2 * d.L + 1) * sizeof(real);
}
static size_t update3d_smem(const Dev &d) { return (size_t)col_b(d) * (2 * d.L + 1 + kU3Sc + 4) * sizeof(real); }
static size_t wvel_smem(const Dev &d) {
    return (size_t)col_b(d) * (kWvEdges * sizeof(WvEdge) + ((d.L | 1) + 2) * sizeof(real));
}
int config_columns(const Dev &d) {
    cudaError_t e = raise_smem_limit(implvisc_tile_kernel(d), implvisc_tile_smem(d, implvisc_cols(d)));
    if (e == cudaSuccess) e = raise_smem_limit(k_bpg_elem, bpg_smem(d));
    if (e == cudaSuccess) e = raise_smem_limit(k_update3d, update3d_smem(d));
    if (e == cudaSuccess) e = raise_smem_limit(k_pressure_col, pressure_smem(d));
    if (e == cudaSuccess) e = raise_smem_limit(k_wvel, wvel_smem(d));
    return e == cudaSuccess ? 0 : 1;
}
// first: nothing but copies, fills or graphs before it on the stream
void launch_pressure_col(const Dev &d, bool first, cudaStream_t s) {
    launch_resident_as(!first, k_pressure_col, d.N, pressure_b(d), pressure_b(d) * d.L, pressure_smem(d), s, d);
}
void launch_bpg_elem(const Dev &d, cudaStream_t s) {
    launch_resident(k_bpg_elem, d.E, col_b(d), col_b(d) * d.L, bpg_smem(d), s, d);
}
void launch_velgrad3d(const Dev &d, cudaStream_t s) {
    const int b = tuned(d, TK_VELGRAD3D, 256);
    launch_k(k_velgrad3d, grid_for((long long)d.E * d.L, b), b, 0, s, d);
}
void launch_adv3_edge(const Dev &d, cudaStream_t s) {
    const int b = tuned(d, TK_ADV3, 256);
    launch_k(k_adv3_edge, grid_for((long long)d.Ed_in * d.L, b), b, 0, s, d);
}
void launch_filt2x(const Dev &d, cudaStream_t s) {
    launch_k(k_filt2x_uc, grid_for((long long)d.E * d.L, 256), 256, 0, s, d);
}
void launch_bih_geom(const Dev &d, cudaStream_t s) { launch_k(k_bih_geom, grid_for(d.Ed, 256), 256, 0, s, d); }
void launch_bih(const Dev &d, cudaStream_t s) {
    const int ge = grid_for((long long)d.Ed * d.L, 256), gl = grid_for((long long)d.E * d.L, 256);
    launch_k(k_bih_edge, ge, 256, 0, s, d, d.U_n, d.V_n, 0);
    launch_k(k_bih_uc, gl, 256, 0, s, d, 0);
    launch_k(k_bih_grad<false>, gl, 256, 0, s, d, d.bihU, d.bihV);
    launch_k(k_bih_edge, ge, 256, 0, s, d, d.bihU, d.bihV, 1);
}
void launch_bih_puls(const Dev &d, cudaStream_t s) {
    const int ge = grid_for((long long)d.Ed * d.L, 256), gl = grid_for((long long)d.E * d.L, 256);
    launch_k(k_bih_grad<true>, gl, 256, 0, s, d, d.U_puls, d.V_puls);
    launch_k(k_bih_edge, ge, 256, 0, s, d, d.U_puls, d.V_puls, 0);
    launch_k(k_bih_uc, gl, 256, 0, s, d, 1);
    launch_k(k_bih_grad<false>, gl, 256, 0, s, d, d.bihU, d.bihV);
    launch_k(k_bih_edge, ge, 256, 0, s, d, d.bihU, d.bihV, 2);
}
void launch_velrhs(const Dev &d, real ff, cudaStream_t s) {
    const int b = tuned(d, TK_VELRHS, 256);
    launch_k(k_velrhs, grid_for((long long)d.E * d.L, b), b, 0, s, d, ff);
}
#define MAXL_DISPATCH(KERNEL, GRID, BLOCK, STREAM, ...)                                   \
    do {                                                                                   \
        if (d.L <= 24) launch_k(KERNEL<24>, GRID, BLOCK, 0, STREAM, __VA_ARGS__);                \
        else if (d.L <= 48) launch_k(KERNEL<48>, GRID, BLOCK, 0, STREAM, __VA_ARGS__);           \
        else launch_k(KERNEL<128>, GRID, BLOCK, 0, STREAM, __VA_ARGS__);                         \
    } while (0)
void launch_implvisc(const Dev &d, cudaStream_t s) {
    if (d.im_vert_visc) MAXL_DISPATCH(k_implvisc, grid_for(d.E, 128), 128, s, d);
    if (!d.im_vert_visc_fic) return;
    if (implvisc_reg(d)) launch_k(implvisc_reg_kernel(d), (d.E + kIrCols - 1) / kIrCols, kIrCols, implvisc_reg_smem(d), s, d);
    else {
        const int C = implvisc_cols(d);
        launch_k(implvisc_tile_kernel(d), (d.E + C - 1) / C, C == 16 ? 256 : 128, implvisc_tile_smem(d, C), s, d);
    }
}
void launch_jac_swap(const Dev &d, cudaStream_t s) {
    const int b = tuned(d, TK_ROT, 256);
    launch_k(k_jac_swap, grid_for(d.N, b), b, 0, s, d);
}
// after an upload or a copy of the elevation
void launch_je(const Dev &d, cudaStream_t s) { launch_plain(k_je_elem, grid_for((long long)d.E * d.L, 256), 256, 0, s, d); }
void launch_update3d(const Dev &d, real Mt_inv, cudaStream_t s) {
    launch_resident(k_update3d, d.E, col_b(d), col_b(d) * d.L, update3d_smem(d), s, d, Mt_inv);
}
void launch_wvel(const Dev &d, cudaStream_t s) { launch_resident(k_wvel, d.N, col_b(d), col_b(d) * d.L, wvel_smem(d), s, d); }


// Largest block (threads) each tunable kernel of this file can launch with
// (its registers and launch bounds): lim[knob] lowered to that.
static void tune_lower(int *lim, int knob, const void *k) {
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, k) == cudaSuccess && a.maxThreadsPerBlock < lim[knob]) lim[knob] = a.maxThreadsPerBlock;
}
void tune_limits_baroclinic(int *lim) {
    tune_lower(lim, TK_VELRHS, (const void *)k_velrhs);
    tune_lower(lim, TK_VELGRAD3D, (const void *)k_velgrad3d);
    tune_lower(lim, TK_ADV3, (const void *)k_adv3_edge);
}

FESOMC_PREC_END
