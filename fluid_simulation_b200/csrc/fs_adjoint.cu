// Adjoint (reverse-mode derivative) of one WCSPH substep (fs_wcsph.cu;
// reference SolverWCSPH.step, solver_wcsph.py:431-535), with the neighbour
// set of the step held fixed (the grid is a piecewise-constant function of
// the positions: it contributes no derivative).
//
// Forward, per dynamic particle i (j over active neighbours within h):
//   rho_i = sum_j mv_j W(r_ij)                              (self included)
//   p_i   = B_i ((rho_i / rho0_i)^gamma_i - 1)   [max(p, 0) when clamped;
//           its derivative is taken as 1 where p > 0 and 0 elsewhere]
//   P_i   = p_i / max(rho_i^2, 1e-6),  R_i = 1 / max(rho_i, 1e-6)
//   a_i   = g + sum_{j != i} c_ij d_ij,          d_ij = x_i - x_j,
//   c_ij  = (visc_ij + pres_ij) gs(r) - coh_i m_j W(max(r, r_p))
//   visc_ij = 10 nu_i m_j R_j (u_ij . d_ij) / (r^2 + 0.01 h^2),  u_ij = v_i - v_j
//   pres_ij = -m_j (P_i + P_j),                   grad W(d) = gs(r) d
//   u' = v + dt a;  x' = x + dt u';  walls(x', u')
// Given the adjoints of the outputs (xb', vb') the three passes compute:
//   gather     (in the grid build) cell-order copies of the step's data, and
//              walls^T and the integrator -> ab_i
//   force      per particle k, both sides of every pair (k, j): its own term
//              of a_k (weights ab_k) and its term in a_j (weights ab_j), so
//              each thread sums into its own slot (a gather, no atomics):
//                xb_k += dc/dd-terms,  vb_k += visc terms,
//                Pb_k, Rb_k, nub_k;  then the EOS chain rule per particle:
//                rhob_k, Bb_k (stiffness), rho0b_k (rest density).
//   density    xb_k += sum_j (rhob_k mv_j + rhob_j mv_k) gs(r) d_kj
// The force pass records the neighbour lists of the step's positions; the
// density pass reuses them.
#include "fs_build.cuh"

namespace fs {

namespace {

// Backward of apply_walls (mode 0/1), one axis: forward p, v before the walls;
// in: pb, vb adjoints after the walls; out: adjoints before the walls.
FS_DEV void wall_axis_adjoint(float p0, float v0, float lo, float hi, float damping, bool cond, float& pb, float& vb) {
  const bool c1 = p0 < lo;
  const bool d1 = c1 && (!cond || v0 < 0.f);
  const float p1 = c1 ? lo : p0;
  const float v1 = d1 ? v0 * damping : v0;
  const bool c2 = p1 > hi;
  const bool d2 = c2 && (!cond || v1 > 0.f);
  if (d2) vb *= damping;
  if (c2) pb = 0.f;
  if (d1) vb *= damping;
  if (c1) pb = 0.f;
}

// Adjoint of integrate_velocity / integrate_positions / apply_bounds for one
// dynamic particle: returns ab (= dt * ub) and the direct xb, vb.
FS_DEV void integrate_adjoint(const Walls& w, float3 x, float3 v, float3 a, float dt, float3 xbo, float3 vbo,
                              float3& xb, float3& vb, float3& ab) {
  const float3 u = make_float3(v.x + dt * a.x, v.y + dt * a.y, v.z + dt * a.z);
  const float3 p = make_float3(x.x + u.x * dt, x.y + u.y * dt, x.z + u.z * dt);
  const bool cond = w.mode != 1;
  float3 pb = xbo, ub = vbo;
  wall_axis_adjoint(p.x, u.x, w.xmin, w.xmax, w.damping, cond, pb.x, ub.x);
  wall_axis_adjoint(p.y, u.y, w.ymin, w.ymax, w.damping, cond, pb.y, ub.y);
  wall_axis_adjoint(p.z, u.z, w.zmin, w.zmax, w.damping, cond, pb.z, ub.z);
  // p = x + u dt;  u = v + dt a
  ub = make_float3(ub.x + dt * pb.x, ub.y + dt * pb.y, ub.z + dt * pb.z);
  xb = pb;
  vb = ub;
  ab = make_float3(dt * ub.x, dt * ub.y, dt * ub.z);
}

struct AdjArgs {
  GridDev g;
  NbrList L;
  ScanXyz q;
  int64_t n;
  fs_model m;
  const float4* xs;    // (x, flags)
  const float4* vs;    // (v, mass)
  const float* mv;     // rest_density * volume
  const float2* sc2;   // (P, R)
  const float* nu;     // viscosity, cell order (0: does not move)
  const float* coh;    // surface_tension / mass, cell order (0: does not move)
  float4* ab;          // (ab, 0), cell order
  float4* xr;          // (xb partial, rhob), cell order
  const float* xin;    // step input positions, original order
  const float* vin;    // step input velocities
  const float* accel;  // forward accel, original order
  const float* rho;    // forward rho, original order
  const float* pressure;
  const float* xbo;    // adjoint of particle_q out, original order
  const float* vbo;    // adjoint of particle_qd out
  float* xbi;          // adjoint of particle_q in
  float* vbi;          // adjoint of particle_qd in
  float* gb_stiffness; // += (may be null)
  float* gb_viscosity;
  float* gb_rest_density;
  float h, particle_radius, dt;
  int clamp;
  Walls walls;
};

// Cell-order copies of what the adjoint passes read (gathered by the grid
// build's last kernel): positions
// + flags, velocities + mass, mv, (P, R) from the step's rho and pressure,
// viscosity, cohesion / mass, and ab from the walls / integrator adjoint.
struct AdjGather {
  AdjArgs a;
  float *nu, *coh;
  float4* xs;
  ScanOut q;
  float4* vs;
  float* mv;
  float2* sc2;
  FS_DEV void operator()(int64_t s, int32_t i) const {
    const fs_model& m = a.m;
    const float3 x = ld3(a.xin, i), v = ld3(a.vin, i);
    const int pf = particle_pf(m.particle_flags, m.particle_mask, i);
    const int w = (a.g.nworlds > 0 && m.particle_world) ? world_index(m.particle_world[i], a.g.nworlds) : 0;
    const float mass = m.particle_mass[i];
    xs[s] = make_float4(x.x, x.y, x.z, pack_pf(pf, w));
    scan_put(q, s, x, (pf & PF_ACTIVE) != 0);
    vs[s] = make_float4(v.x, v.y, v.z, mass);
    const float rd = m.rest_density[i];
    mv[s] = rd * (mass / fmaxf(rd, 1.0e-6f));
    const float r = a.rho[i];
    sc2[s] = make_float2(a.pressure[i] / fmaxf(r * r, 1.0e-6f), 1.0f / fmaxf(r, 1.0e-6f));
    // A particle that does not move has no terms of its own.  Its coefficients
    // are 0 as its ab is, so that the products of the two are 0: without mass,
    // surface_tension / mass is not finite.
    const bool dyn = pf & PF_DYNAMIC;
    nu[s] = dyn ? m.viscosity[i] : 0.f;
    coh[s] = dyn ? m.surface_tension[i] / mass : 0.f;
    float3 ab = make_float3(0.f, 0.f, 0.f);
    if (dyn) {
      float3 xb, vb;
      integrate_adjoint(walls_of(a.walls, a.g, w), x, v, ld3(a.accel, i), a.dt, ld3(a.xbo, i), ld3(a.vbo, i), xb, vb,
                        ab);
    }
    a.ab[s] = make_float4(ab.x, ab.y, ab.z, 0.f);
  }
};

// What both sides of a pair share: gs(r) and its derivative (Cubic.grad_scale),
// 1 / (r^2 + 0.01 h^2), the cohesion weight W(max(r, r_p)) and its derivative
// in r (0 unless needed).
struct PairGeometry {
  float rinv, gs, dgs, den, w, dw;
  FS_DEV PairGeometry(const Cubic& K, float h, float particle_radius, float r2, bool cohesion) {
    float r;
    r_and_inv(r2, r, rinv);
    const float q = r * K.inv_h;
    gs = dgs = w = dw = 0.f;
    if (r > 1.0e-5f && q <= 1.f) {
      if (q <= 0.5f) {
        gs = K.g_in * fmaf(3.f, q, -2.f);
        dgs = K.g_in * 3.f * K.inv_h;
      } else {
        const float t = 1.f - q;
        gs = K.g_out * t * t * rinv;
        dgs = K.g_out * (-2.f * t * K.inv_h * rinv - t * t * rinv * rinv);
      }
    }
    den = 1.0f / (r2 + 0.01f * (h * h));
    if (cohesion) {
      const float s = fmaxf(r, particle_radius);
      w = K.w(s);
      if (r > particle_radius && s > 1.0e-5f) dw = K.grad_scale(s, 1.0f / s) * s;
    }
  }
};

// G lanes per particle add up their own pairs' terms, then the lanes' sums
// (the adjoint's sums have no order to keep).
template <int G>
__global__ void FS_NB_BOUNDS k_adj_force(AdjArgs a) {
  extern __shared__ uint2 smem[];
  grid_begin();
  lists_recorded(a.L);
  struct Neighbour {
    float4 v, ab;
    float2 PR;
    float nu, coh;
  };
  auto fetch = [&](int t) {
    return Neighbour{__ldg(a.vs + t), __ldg(a.ab + t), __ldg(a.sc2 + t), __ldg(a.nu + t), __ldg(a.coh + t)};
  };
  // with one thread per particle four neighbours are in flight: their records
  // would not fit the registers, and load when their terms need them
  auto load = [&](int t) {
    if constexpr (G > 1)
      return fetch(t);
    else
      return 0;
  };
  for_groups<G>(a.n, [&](int64_t s, bool live, bool lead) {
    const float4 xk = a.xs[s];
    const int32_t i = a.g.perm[s];
    const int pfk = pf_of(xk);
    const bool on = live && (pfk & PF_ACTIVE);
    const float4 vk = a.vs[s];
    const float m_k = vk.w;
    const float2 PRk = a.sc2[s];
    const float nu_k = a.nu[s], coh_k = a.coh[s];
    float3 xb = make_float3(0.f, 0.f, 0.f), vb = make_float3(0.f, 0.f, 0.f), abk = make_float3(0.f, 0.f, 0.f);
    if (pfk & PF_DYNAMIC)
      integrate_adjoint(walls_of(a.walls, a.g, world_of(xk)), xyz(xk), xyz(vk), ld3(a.accel, i), a.dt, ld3(a.xbo, i),
                        ld3(a.vbo, i), xb, vb, abk);
    else
      xb = ld3(a.xbo, i), vb = ld3(a.vbo, i);
    if (!lead) xb = vb = make_float3(0.f, 0.f, 0.f);  // the lead lane's sums start at the direct terms
    const Cubic K(a.h);
    const float h2m = a.h * a.h * kSupportMargin;
    float Pb = 0.f, Rb = 0.f, nub = 0.f;
    scan_sum<G, false, false, false, kExact, 0>(
        a.g, a.q, a.xs, (int)s, xk, a.h, h2m, h2m, a.L, smem, on, -1, load,
        [&](int t, float4 xj, const auto& p) {
          const float3 d = make_float3(xk.x - xj.x, xk.y - xj.y, xk.z - xj.z);
          const float r2 = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z));
          if (r2 == 0.f) return Terms<0>{};  // the forward skips coincident pairs
          Neighbour nb;
          if constexpr (G > 1)
            nb = p;
          else
            nb = fetch(t);
          // The two terms of the pair, of a_k (weights ab_k) and of a_j (weights
          // ab_j, d_jk = -d, u_jk = -u), share their geometry and directions:
          //   c = A gs - coh m W with A = kv ud den - m Psum, kv = 10 nu m R
          //   d(c d)/dd . ab = c ab + (ab . d) (tang u + radial d)
          // (evaluated side by side, they took twice the operations; ab, nu and
          // coh are 0 for a particle that is not dynamic)
          const float3 u = make_float3(vk.x - nb.v.x, vk.y - nb.v.y, vk.z - nb.v.z);
          const float m_j = nb.v.w;
          const PairGeometry P(K, a.h, a.particle_radius, r2, coh_k != 0.f || nb.coh != 0.f);
          const float ud = fmaf(u.x, d.x, fmaf(u.y, d.y, u.z * d.z)), udd = ud * P.den;
          const float abk_d = fmaf(abk.x, d.x, fmaf(abk.y, d.y, abk.z * d.z));
          const float abj_d = fmaf(nb.ab.x, d.x, fmaf(nb.ab.y, d.y, nb.ab.z * d.z));
          const float Psum = PRk.x + nb.PR.x;
          const float visc_k = 10.f * m_j * nb.PR.y, visc_j = 10.f * m_k * PRk.y;  // kv / nu
          const float kv_k = nu_k * visc_k, kv_j = nb.nu * visc_j;
          const float A_k = fmaf(kv_k, udd, -m_j * Psum), A_j = fmaf(kv_j, udd, -m_k * Psum);
          const float g_k = coh_k * m_j, g_j = nb.coh * m_k;
          const float c_k = fmaf(A_k, P.gs, -g_k * P.w), c_j = fmaf(A_j, P.gs, -g_j * P.w);
          const float curl = 2.f * udd * P.den * P.gs;
          const float radial_k = fmaf(fmaf(A_k, P.dgs, -g_k * P.dw), P.rinv, -kv_k * curl);
          const float radial_j = fmaf(fmaf(A_j, P.dgs, -g_j * P.dw), P.rinv, -kv_j * curl);
          const float S = P.den * P.gs * fmaf(abk_d, kv_k, -abj_d * kv_j);
          const float T = fmaf(abk_d, radial_k, -abj_d * radial_j);
          xb.x += fmaf(c_k, abk.x, fmaf(-c_j, nb.ab.x, fmaf(S, u.x, T * d.x)));
          xb.y += fmaf(c_k, abk.y, fmaf(-c_j, nb.ab.y, fmaf(S, u.y, T * d.y)));
          xb.z += fmaf(c_k, abk.z, fmaf(-c_j, nb.ab.z, fmaf(S, u.z, T * d.z)));
          vb = make_float3(fmaf(S, d.x, vb.x), fmaf(S, d.y, vb.y), fmaf(S, d.z, vb.z));
          Pb = fmaf(P.gs, fmaf(m_k, abj_d, -m_j * abk_d), Pb);
          const float gu = P.gs * udd;
          nub = fmaf(abk_d * visc_k, gu, nub);
          Rb = fmaf(-abj_d * (10.f * nb.nu * m_k), gu, Rb);
          return Terms<0>{};
        },
        [](const Terms<0>&) {});
    if constexpr (G > 1) {
      xb = make_float3(group_sum<G>(xb.x), group_sum<G>(xb.y), group_sum<G>(xb.z));
      vb = make_float3(group_sum<G>(vb.x), group_sum<G>(vb.y), group_sum<G>(vb.z));
      Pb = group_sum<G>(Pb), Rb = group_sum<G>(Rb), nub = group_sum<G>(nub);
    }
    if (!lead) return;
    if (!on) {  // untouched by the step: identity
      a.L.cnt[s] = 0;
      a.xr[s] = make_float4(0.f, 0.f, 0.f, 0.f);
      st3(a.xbi, i, xb);
      st3(a.vbi, i, vb);
      return;
    }
    // P = p / max(rho^2, 1e-6), R = 1 / max(rho, 1e-6), then the EOS
    const float rho = a.rho[i], p = a.pressure[i];
    const float rr = rho * rho;
    const float inv_rr = 1.0f / fmaxf(rr, 1.0e-6f);
    float rhob = 0.f;
    if (rr > 1.0e-6f) rhob -= 2.f * Pb * p * inv_rr / rho;
    if (rho > 1.0e-6f) rhob -= Rb / rr;
    const float pb = Pb * inv_rr;
    const float B = a.m.stiffness[i], gam = a.m.exponent[i], rd = a.m.rest_density[i];
    const float rho0 = fmaxf(rd, 1.0e-6f);
    const float ratio = rho / rho0;
    const float pw = powf(ratio, gam);
    const float p_raw = B * (pw - 1.0f);
    // max(p, 0) has no derivative at p = 0; there the clamped side is taken
    // (d/dp = 0), as for a ReLU: the pressure responds only where p > 0
    if (!(a.clamp && !(p_raw > 0.f)) && pb != 0.f) {
      const float dp_dratio = B * gam * (ratio > 0.f ? pw / ratio : 0.f);
      rhob += pb * dp_dratio / rho0;
      if (a.gb_stiffness) a.gb_stiffness[i] += pb * (pw - 1.0f);
      if (a.gb_rest_density && rd > 1.0e-6f) a.gb_rest_density[i] += -pb * dp_dratio * ratio / rho0;
    }
    if (a.gb_viscosity) a.gb_viscosity[i] += nub;
    a.xr[s] = make_float4(xb.x, xb.y, xb.z, rhob);
    st3(a.vbi, i, vb);
  });
}

// The compiler takes 64 registers (40 and 12 bytes of spills with several
// lanes); no other budget was measured.
template <int G>
__global__ void FS_NB_BOUNDS k_adj_density(AdjArgs a) {
  grid_begin();
  for_groups<G>(a.n, [&](int64_t s, bool live, bool lead) {
    const float4 xk = a.xs[s];
    const bool on = live && (pf_of(xk) & PF_ACTIVE);
    const int32_t i = a.g.perm[s];
    const float4 xr = a.xr[s];
    const float mv_k = a.mv[s];
    const Cubic K(a.h);
    float3 xb = lead ? make_float3(xr.x, xr.y, xr.z) : make_float3(0.f, 0.f, 0.f);
    list_sum<G, false, false, true, true, 0, kAhead>(
        a.g, a.xs, a.xs, (int)s, xk, a.h, a.h * a.h * kSupportMargin, a.L, lists_usable(a.L), on,
        [&](int t) { return make_float2(__ldg(a.mv + t), __ldg(&a.xr[t].w)); },
        [&](int t, float4 xj, const float2& j) {
          const float dx = xk.x - xj.x, dy = xk.y - xj.y, dz = xk.z - xj.z;
          float r, rinv;
          r_and_inv(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), r, rinv);
          const float w = (xr.w * j.x + j.y * mv_k) * K.grad_scale(r, rinv);
          xb = make_float3(fmaf(w, dx, xb.x), fmaf(w, dy, xb.y), fmaf(w, dz, xb.z));
          return Terms<0>{};
        },
        [](const Terms<0>&) {});
    if constexpr (G > 1) xb = make_float3(group_sum<G>(xb.x), group_sum<G>(xb.y), group_sum<G>(xb.z));
    if (lead && on) st3(a.xbi, i, xb);  // inactive: written by the force pass
  });
}

}  // namespace
}  // namespace fs

using namespace fs;

extern "C" {

int fs_wcsph_substep_adjoint(fs_context* c, const fs_model* m, const fs_state* si, const float* rho,
                             const float* pressure, const float* accel, const float* adj_x_out, const float* adj_v_out,
                             float* adj_x_in, float* adj_v_in, float* adj_stiffness, float* adj_viscosity,
                             float* adj_rest_density, const fs_wcsph_params* p, fs_stream_t stream) {
  if (!c || !m || !si || !p) return set_error(FS_ERR_INVALID, "fs_wcsph_substep_adjoint: null argument");
  if (m->n < 0) return set_error(FS_ERR_INVALID, "fs_wcsph_substep_adjoint: negative n");
  if (m->n == 0) return FS_OK;
  if (!m->particle_flags || !m->particle_mask || !m->particle_mass || !m->gravity || m->n_worlds < 1 ||
      !m->rest_density || !m->viscosity || !m->surface_tension || !m->stiffness || !m->exponent ||
      !si->particle_q || !si->particle_qd || !rho || !pressure || !accel || !adj_x_out || !adj_v_out || !adj_x_in ||
      !adj_v_in)
    return set_error(FS_ERR_INVALID, "fs_wcsph_substep_adjoint: missing array");
  if (m->n > c->capacity) return set_error(FS_ERR_CAPACITY, "fs_wcsph_substep_adjoint: n > capacity");
  DeviceGuard dg(c->device);
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t n = m->n;
  const float h = p->smoothing_length;
  int rc;
  AdjArgs a;
  a.g = grid_view(c);
  a.L = nbr_list(c);
  a.q = scan_xyz(c);
  a.n = n;
  a.m = *m;
  a.xs = c->xs;
  a.vs = c->vs;
  a.mv = c->mv;
  a.sc2 = c->sc2;
  a.nu = c->sc1;
  a.coh = c->sc1b;
  a.ab = c->xs2;
  a.xr = c->vs2;
  a.xin = si->particle_q;
  a.vin = si->particle_qd;
  a.accel = accel;
  a.rho = rho;
  a.pressure = pressure;
  a.xbo = adj_x_out;
  a.vbo = adj_v_out;
  a.xbi = adj_x_in;
  a.vbi = adj_v_in;
  a.gb_stiffness = adj_stiffness;
  a.gb_viscosity = adj_viscosity;
  a.gb_rest_density = adj_rest_density;
  a.h = h;
  a.particle_radius = p->particle_radius;
  a.dt = p->dt;
  a.clamp = p->clamp_negative_pressure;
  a.walls = make_walls(p->bound_width, p->bound_height, p->bound_length, p->boundary_damping, 0, 0.f, 0.f);
  if ((rc = grid_build(c, n, h * c->cell_ratio, st, m->particle_world, nullptr, KeyPositions{si->particle_q},
                       AdjGather{a, c->sc1, c->sc1b, c->xs, scan_out(c), c->vs, c->mv, c->sc2})))
    return rc;
  a.g = grid_view(c);
  {
    PassScope ps_(c, P_ADJ_FORCE, st);
    FS_NB_LAUNCH(k_adj_force, c, n, nb_group(n), st, true, a);
  }
  {
    PassScope ps_(c, P_ADJ_DENSITY, st);
    FS_NB_LAUNCH(k_adj_density, c, n, nb_group(n), st, false, a);
  }
  c->last_stream = st;
  return launch_check("fs_wcsph_substep_adjoint");
}

}  // extern "C"
