// Hand-written adjoint of the fixed-iteration VBD step (one substep: membrane, bending, tetrahedra and springs
// with their damping, particle-shape contacts on static shapes).
//
// Forward map of one substep (vbd_kernels.cuh, CSR path, one lane per vertex):
//   y   = q + (qd + (g + f_ext / m) dt) dt                    inertial target, also the first iterate
//   for it < I, for color c, for v in c (Jacobi within the color, positions x of the color's start):
//       g_v = (m / dt^2)(y_v - x_v) + sum_e f_e,v(x),   H_v = (m / dt^2) I + sum_e H_e,v(x)
//       x_v <- x_v + H_v^-1 g_v          (skipped when |det H_v| <= 1e-8)
//   q_out = x,   qd_out = (x - q) / dt
//
// Reverse of one color update x' = x + D(x), D_v = H_v^-1 g_v, given the adjoint a = dL/dx':
//   w = H_v^-1 a_v        (H_v is symmetric)
//   dL/dg_v = w,   dL/dH_v = -w D_v^T   (only its symmetric part meets the symmetric dH)
//   dL/dx = a + [dg_v/dx]^T w + [dH_v/dx] : (-w D_v^T),   likewise for y and the element parameters.
// The positions x of a color's start need no recomputation: within an iteration a vertex moves once, in its own
// color, so they are the iteration's end positions where the vertex's color comes earlier and its start positions
// elsewhere (ColorState over two consecutive checkpoints).
// The element terms f_e,v and H_e,v are differentiated with forward-mode dual numbers over the element's vertex
// coordinates (and the triangle's mu, lambda), running the same element routines as the forward pass. A warp works on
// one vertex and four lanes on one of its elements, each with the derivative slots of one of the element's vertices
// (3, or 6 with damping). Vertices of one color are never neighbours, so the vertices written through atomics (the
// neighbours, the triangle parameters) are never read by the same launch.
// A contact term and a damped element depend on positions x and, through friction and damping, on the
// positions at the start of the substep, q; the derivatives in q are accumulated per vertex (adj_xp) and
// join dL/dq_in at the end. The contact set, the contact points and normals and the penalty
// stiffness are held fixed (the derivative of the step for its contacts; the AVBD ramp is off).
#pragma once
#include "vbd_dual.cuh"
#include "vbd_kernels.cuh"

namespace vbd {

// Positions at the start of a color: `after` holds the vertices of the colors before it, `before` the others.
template <typename R>
struct ColorState {
  const R* before;  // [V*3] positions at the iteration's start
  const R* after;   // [V*3] positions at its end
  const int* color_of;
  int color;
  __device__ __forceinline__ vec3<R> ld(int i) const {
    const R* a = __ldg(color_of + i) < color ? after : before;
    return {a[3 * size_t(i)], a[3 * size_t(i) + 1], a[3 * size_t(i) + 2]};
  }
};

template <typename R>
struct AdjCtx {
  StepCtx<R> c;           // model arrays (CSR) and dt
  ColorState<R> x;        // positions at the start of the color (the forward state)
  const R* y;             // [V*3] inertial targets
  R* adj_x;               // [V*3] in: dL/dx', out: dL/dx (in place)
  R* adj_y;               // [V*3] accumulated dL/dy
  R* adj_mu;              // [T] accumulated dL/dmu (triangle), may be NULL
  R* adj_lambda;          // [T] accumulated dL/dlambda, may be NULL
  R* adj_xp;              // [V*3] accumulated dL/dq through the contact terms (contacts only)
};

// mass used by the solve (0 for a fixed particle), as forward_particle stores it
template <typename R>
__device__ __forceinline__ R solve_mass(const StepCtx<R>& c, int v) {
  const float m = c.mass[v];
  return ((c.flags[v] & 1) && m != 0.f) ? R(m) : R(0);
}

template <typename R>
__device__ __forceinline__ vec3<R> ldx(const R* a, int i) {
  return {a[3 * i], a[3 * i + 1], a[3 * i + 2]};
}

template <typename R>
__device__ __forceinline__ void atomic_add3(R* a, int i, vec3<R> v) {
  atomicAdd(a + 3 * i, v.x);
  atomicAdd(a + 3 * i + 1, v.y);
  atomicAdd(a + 3 * i + 2, v.z);
}

// <g_bar, df> + <H_bar, dH> for one derivative slot k (H_bar symmetric, stored as 6 with the
// off-diagonal entries counted twice)
template <typename R, int N>
__device__ __forceinline__ R contract(const vec3<Dual<R, N>>& f, const sym3<Dual<R, N>>& H, vec3<R> gb,
                                      const sym3<R>& Hb, int k) {
  return gb.x * f.x.d[k] + gb.y * f.y.d[k] + gb.z * f.z.d[k] + Hb.xx * H.xx.d[k] + Hb.yy * H.yy.d[k] +
         Hb.zz * H.zz.d[k] + R(2) * (Hb.xy * H.xy.d[k] + Hb.xz * H.xz.d[k] + Hb.yz * H.yz.d[k]);
}

// This lane's share (of L lanes) of the element and contact terms of vertex v at the positions X: each kind of
// element starts at lane 0, the contacts are lane 0's.
template <typename R, int L>
__device__ __forceinline__ void assemble(const StepCtx<R>& c, const ColorState<R>& X, int v, int lane, vec3<R>& f,
                                         sym3<R>& H) {
  for (int a = c.face_off[v] + lane; a < c.face_off[v + 1]; a += L) {
    const int t = c.face_adj[a] >> 2, ord = c.face_adj[a] & 3;
    const float4 mat = c.tri_mat[t];
    if (!(mat.x > 0.f || mat.y > 0.f)) continue;
    const int4 ti = c.tri_idx[t];
    const float4 dm = c.tri_pose[t];
    const R pose[4] = {R(dm.x), R(dm.y), R(dm.z), R(dm.w)};
    vec3<R> xp[3];
    if (mat.z > 0.f) xp[0] = ld3<R>(c.qprev[ti.x]), xp[1] = ld3<R>(c.qprev[ti.y]), xp[2] = ld3<R>(c.qprev[ti.z]);
    membrane_add<R>(ord, X.ld(ti.x), X.ld(ti.y), X.ld(ti.z), pose, R(mat.x), R(mat.y), R(mat.z), R(mat.w), c.dt, xp, f,
                    H);
  }
  for (int a = c.edge_off[v] + lane; a < c.edge_off[v + 1]; a += L) {
    const int e = c.edge_adj[a] >> 2, ord = c.edge_adj[a] & 3;
    const float4 pr = c.edge_prop[e];
    if (!(pr.z > 0.f)) continue;
    const int4 ei = c.edge_idx[e];
    const vec3<R> xs[4] = {X.ld(ei.x), X.ld(ei.y), X.ld(ei.z), X.ld(ei.w)};
    vec3<R> xp[4];
    if (pr.w > 0.f)
      xp[0] = ld3<R>(c.qprev[ei.x]), xp[1] = ld3<R>(c.qprev[ei.y]), xp[2] = ld3<R>(c.qprev[ei.z]),
      xp[3] = ld3<R>(c.qprev[ei.w]);
    bending_add<R>(ord, xs, R(pr.x), R(pr.y), R(pr.z), R(pr.w), c.dt, xp, f, H);
  }
  if (c.tet_off) {  // tetrahedra (solve_elasticity adds them after the hinges)
    for (int a = c.tet_off[v] + lane; a < c.tet_off[v + 1]; a += L) {
      const int t = c.tet_adj[a] >> 2, ord = c.tet_adj[a] & 3;
      const float4 r0 = c.tet_pose[3 * t], r1 = c.tet_pose[3 * t + 1], r2 = c.tet_pose[3 * t + 2];
      if (!(r0.w > 0.f || r1.w > 0.f)) continue;
      const int4 ti = c.tet_idx[t];
      const R dm[9] = {R(r0.x), R(r0.y), R(r0.z), R(r1.x), R(r1.y), R(r1.z), R(r2.x), R(r2.y), R(r2.z)};
      const vec3<R> xs[4] = {X.ld(ti.x), X.ld(ti.y), X.ld(ti.z), X.ld(ti.w)};
      vec3<R> xp[4];
      if (r2.w > 0.f)
        xp[0] = ld3<R>(c.qprev[ti.x]), xp[1] = ld3<R>(c.qprev[ti.y]), xp[2] = ld3<R>(c.qprev[ti.z]),
        xp[3] = ld3<R>(c.qprev[ti.w]);
      tet_add<R>(ord, xs, xp, dm, R(r0.w), R(r1.w), R(r2.w), c.dt, f, H);
    }
  }
  if (c.spr_off) {  // springs to other colors, then springs within the color: all at the color's start state
    for (int pass = 0; pass < 2; ++pass) {
      const int* off = pass == 0 ? c.spr_off : c.sspr_off;
      const int* adj = pass == 0 ? c.spr_adj : c.sspr_adj;
      for (int a = off[v] + lane; a < off[v + 1]; a += L) {
        const int sp = adj[a] >> 1, end = adj[a] & 1;
        const int2 ij = c.spr_idx[sp];
        const float4 pr = c.spr_prop[sp];
        const vec3<R> xa = pr.z != 0.f ? ld3<R>(c.qprev[v]) : zero3<R>();
        spring_add<R>(end, X.ld(v), X.ld(end == 0 ? ij.y : ij.x), xa, R(pr.x), R(pr.y), R(pr.z), c.dt, f, H);
      }
    }
  }
  if (c.has_contacts && lane == 0) contacts_add<R>(c, v, X.ld(v), f, H);
}

template <int L, typename R>
__device__ __forceinline__ void sum_lanes(vec3<R>& f, sym3<R>& H) {
  f = {group_sum<L>(f.x), group_sum<L>(f.y), group_sum<L>(f.z)};
  H = {group_sum<L>(H.xx), group_sum<L>(H.yy), group_sum<L>(H.zz),
       group_sum<L>(H.xy), group_sum<L>(H.xz), group_sum<L>(H.yz)};
}

// Contact terms of vertex v with dual numbers over its position x (slots 0-2) and its position at the start of the
// substep (slots 3-5, c.qprev), as contacts_add_n evaluates them for static shapes; their derivatives contracted
// with (w, H_bar) add to ax and to adj_xp.
template <typename R>
__device__ __forceinline__ void contacts_adjoint(const StepCtx<R>& c, int v, vec3<R> x, vec3<R> w, const sym3<R>& Hb,
                                                 vec3<R>& ax, R* adj_xp) {
  int n = c.slot_cnt[v];
  if (n > c.K) n = c.K;
  if (n <= 0) return;
  using D6 = Dual<R, 6>;
  const vec3<R> xp = ld3<R>(c.qprev[v]);
  const vec3<D6> xd = {D6::seed(x.x, 0), D6::seed(x.y, 1), D6::seed(x.z, 2)};
  const vec3<D6> xpd = {D6::seed(xp.x, 3), D6::seed(xp.y, 4), D6::seed(xp.z, 5)};
  const D6 r = D6(R(c.radius[v]));
  const D6 dt = D6(c.dt);
  vec3<R> gxp = zero3<R>();
  for (int j = 0; j < n; ++j) {
    const int t = c.slots[v * c.K + j];
    const vec3<D6> bx = {D6(R(c.c_body_pos[3 * t])), D6(R(c.c_body_pos[3 * t + 1])), D6(R(c.c_body_pos[3 * t + 2]))};
    const vec3<D6> nn = {D6(R(c.c_normal[3 * t])), D6(R(c.c_normal[3 * t + 1])), D6(R(c.c_normal[3 * t + 2]))};
    const D6 pen = -(dot(nn, xd - bx) - r);
    if (!(pen > D6(R(0)))) continue;
    const vec3<D6> bv = {D6(R(c.c_body_vel[3 * t])), D6(R(c.c_body_vel[3 * t + 1])), D6(R(c.c_body_vel[3 * t + 2]))};
    const vec3<D6> rel = (xd - xpd) - bv * dt;
    vec3<D6> fd = {D6(R(0)), D6(R(0)), D6(R(0))};
    sym3<D6> Hd = szero<D6>();
    contact_add<D6>(pen, nn, rel, D6(R(c.c_k[t])), D6(R(c.c_kd[t])), D6(R(c.c_mu[t])), D6(c.fric_eps), dt, fd, Hd);
    ax = ax + vec3<R>{contract(fd, Hd, w, Hb, 0), contract(fd, Hd, w, Hb, 1), contract(fd, Hd, w, Hb, 2)};
    gxp = gxp + vec3<R>{contract(fd, Hd, w, Hb, 3), contract(fd, Hd, w, Hb, 4), contract(fd, Hd, w, Hb, 5)};
  }
  atomic_add3(adj_xp, v, gxp);  // neighbours' damped elements add to the same entry in this launch
}

// The gradient of one element with respect to vertex u (slots 0-2 of this lane's dual numbers): the solved vertex's
// part goes to ax, the others' through atomics; slots 3-5, with damping, are u's start position.
template <typename R, int N>
__device__ __forceinline__ void scatter_vertex(const AdjCtx<R>& A, int v, int u, const vec3<Dual<R, N>>& fd,
                                               const sym3<Dual<R, N>>& Hd, vec3<R> w, const sym3<R>& Hb, vec3<R>& ax) {
  const vec3<R> g = {contract(fd, Hd, w, Hb, 0), contract(fd, Hd, w, Hb, 1), contract(fd, Hd, w, Hb, 2)};
  if (u == v)
    ax = ax + g;
  else
    atomic_add3(A.adj_x, u, g);
  if constexpr (N > 3)
    atomic_add3(A.adj_xp, u,
                vec3<R>{contract(fd, Hd, w, Hb, 3), contract(fd, Hd, w, Hb, 4), contract(fd, Hd, w, Hb, 5)});
}

// Position p (and, with N = 6, start position) of one vertex as dual numbers: seeded when it is this lane's vertex.
template <typename R, int N>
__device__ __forceinline__ vec3<Dual<R, N>> dual_point(vec3<R> p, bool seeded, int slot) {
  using D = Dual<R, N>;
  vec3<D> x = {D(p.x), D(p.y), D(p.z)};
  x.x.d[slot] = R(seeded), x.y.d[slot + 1] = R(seeded), x.z.d[slot + 2] = R(seeded);
  return x;
}

// Membrane term of face t for the solved vertex v: this lane's derivatives are those of vertex k of the face, or of
// (mu, lambda) for k = 3.
template <typename R, int N>
__device__ __forceinline__ void membrane_adjoint(const AdjCtx<R>& A, int v, int t, int ord, int k, vec3<R> w,
                                                 const sym3<R>& Hb, vec3<R>& ax) {
  const StepCtx<R>& c = A.c;
  using D = Dual<R, N>;
  const float4 mat = c.tri_mat[t];
  const int4 ti = c.tri_idx[t];
  const int vid[3] = {ti.x, ti.y, ti.z};
  const float4 dm = c.tri_pose[t];
  vec3<D> xs[3], xp[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    xs[j] = dual_point<R, N>(A.x.ld(vid[j]), j == k, 0);
    if constexpr (N > 3) xp[j] = dual_point<R, N>(ld3<R>(c.qprev[vid[j]]), j == k, 3);
  }
  const D pose[4] = {D(R(dm.x)), D(R(dm.y)), D(R(dm.z)), D(R(dm.w))};
  D mu = D(R(mat.x)), lm = D(R(mat.y));
  mu.d[0] = R(k == 3), lm.d[1] = R(k == 3);
  vec3<D> fd = {D(R(0)), D(R(0)), D(R(0))};
  sym3<D> Hd = szero<D>();
  membrane_add<D>(ord, xs[0], xs[1], xs[2], pose, mu, lm, D(R(N > 3 ? mat.z : 0.f)), D(R(mat.w)), D(c.dt), xp, fd, Hd);
  if (k == 3) {
    if (A.adj_mu) atomicAdd(A.adj_mu + t, contract(fd, Hd, w, Hb, 0));
    if (A.adj_lambda) atomicAdd(A.adj_lambda + t, contract(fd, Hd, w, Hb, 1));
    return;
  }
  scatter_vertex<R, N>(A, v, k == 0 ? ti.x : (k == 1 ? ti.y : ti.z), fd, Hd, w, Hb, ax);
}

// Bending term of hinge e: this lane's derivatives are those of vertex k of the hinge.
template <typename R, int N>
__device__ __forceinline__ void bending_adjoint(const AdjCtx<R>& A, int v, int e, int ord, int k, vec3<R> w,
                                                const sym3<R>& Hb, vec3<R>& ax) {
  const StepCtx<R>& c = A.c;
  using D = Dual<R, N>;
  const float4 pr = c.edge_prop[e];
  const int4 ei = c.edge_idx[e];
  const int vid[4] = {ei.x, ei.y, ei.z, ei.w};
  vec3<D> xs[4], xp[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    xs[j] = dual_point<R, N>(A.x.ld(vid[j]), j == k, 0);
    if constexpr (N > 3) xp[j] = dual_point<R, N>(ld3<R>(c.qprev[vid[j]]), j == k, 3);
  }
  vec3<D> fd = {D(R(0)), D(R(0)), D(R(0))};
  sym3<D> Hd = szero<D>();
  bending_add<D>(ord, xs, D(R(pr.x)), D(R(pr.y)), D(R(pr.z)), D(R(N > 3 ? pr.w : 0.f)), D(c.dt), xp, fd, Hd);
  scatter_vertex<R, N>(A, v, k == 0 ? ei.x : (k == 1 ? ei.y : (k == 2 ? ei.z : ei.w)), fd, Hd, w, Hb, ax);
}

// Tetrahedron term: this lane's derivatives are those of vertex k of the tet.
template <typename R, int N>
__device__ __forceinline__ void tet_adjoint(const AdjCtx<R>& A, int v, int t, int ord, int k, vec3<R> w,
                                            const sym3<R>& Hb, vec3<R>& ax) {
  const StepCtx<R>& c = A.c;
  using D = Dual<R, N>;
  const float4 r0 = c.tet_pose[3 * t], r1 = c.tet_pose[3 * t + 1], r2 = c.tet_pose[3 * t + 2];
  const int4 ti = c.tet_idx[t];
  const int vid[4] = {ti.x, ti.y, ti.z, ti.w};
  const D dm[9] = {D(R(r0.x)), D(R(r0.y)), D(R(r0.z)), D(R(r1.x)), D(R(r1.y)), D(R(r1.z)),
                   D(R(r2.x)), D(R(r2.y)), D(R(r2.z))};
  vec3<D> xs[4], xp[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    xs[j] = dual_point<R, N>(A.x.ld(vid[j]), j == k, 0);
    if constexpr (N > 3) xp[j] = dual_point<R, N>(ld3<R>(c.qprev[vid[j]]), j == k, 3);
  }
  vec3<D> fd = {D(R(0)), D(R(0)), D(R(0))};
  sym3<D> Hd = szero<D>();
  tet_add<D>(ord, xs, xp, dm, D(R(r0.w)), D(R(r1.w)), D(R(N > 3 ? r2.w : 0.f)), D(c.dt), fd, Hd);
  scatter_vertex<R, N>(A, v, k == 0 ? ti.x : (k == 1 ? ti.y : (k == 2 ? ti.z : ti.w)), fd, Hd, w, Hb, ax);
}

// Spring term of entry (spring << 1) | end of vertex v: this lane's derivatives are those of x_v (k = 0), the other
// end (1) and v's start position (2, read by the damping).
template <typename R>
__device__ __forceinline__ void spring_adjoint(const AdjCtx<R>& A, int v, int a, int k, vec3<R> w, const sym3<R>& Hb,
                                               vec3<R>& ax) {
  if (k == 3) return;
  const StepCtx<R>& c = A.c;
  using D = Dual<R, 3>;
  const int sp = a >> 1, end = a & 1;
  const int2 ij = c.spr_idx[sp];
  const float4 pr = c.spr_prop[sp];
  const int o = end == 0 ? ij.y : ij.x;
  const vec3<D> xv = dual_point<R, 3>(A.x.ld(v), k == 0, 0), xo = dual_point<R, 3>(A.x.ld(o), k == 1, 0),
                xa = dual_point<R, 3>(ld3<R>(c.qprev[v]), k == 2, 0);
  vec3<D> fd = {D(R(0)), D(R(0)), D(R(0))};
  sym3<D> Hd = szero<D>();
  spring_add<D>(end, xv, xo, xa, D(R(pr.x)), D(R(pr.y)), D(R(pr.z)), D(c.dt), fd, Hd);
  const vec3<R> g = {contract(fd, Hd, w, Hb, 0), contract(fd, Hd, w, Hb, 1), contract(fd, Hd, w, Hb, 2)};
  if (k == 0)
    ax = ax + g;
  else
    atomic_add3(k == 1 ? A.adj_x : A.adj_xp, k == 1 ? o : v, g);
}

// A warp per vertex: with one thread per vertex a color was a serial chain of 18 elements whose dual numbers over all
// of an element's coordinates (11 or 12 slots, 24 with damping) spilled. The gradient of two substeps of a 64 x 64
// cloth (10 iterations, forward and backward) went from 6.71 to 1.57 ms, with the recorded forward on 16 lanes per
// vertex, the per-color states read from the checkpoints instead of recomputed, and the copies between them gone.
// Bound by the latency of the chain that is left: assembly, block solve, one face and two hinge rounds per color.
template <typename R>
__global__ void __launch_bounds__(128) k_adjoint_color(AdjCtx<R> A, const int* __restrict__ verts, int n) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= n) return;  // the whole warp
  const StepCtx<R>& c = A.c;
  const int v = verts[i];
  const R m = solve_mass(c, v);
  if (m == R(0)) return;  // fixed particle: no update, the adjoint passes through unchanged
  const R md = m * c.dt2r;
  const vec3<R> x = A.x.ld(v);
  // forward quantities at this color's start
  vec3<R> f = zero3<R>();
  sym3<R> H = szero<R>();
  assemble<R, 32>(c, A.x, v, lane, f, H);
  sum_lanes<32>(f, H);
  f = f + md * (ldx(A.y, v) - x);
  H = H + sdiag(md);
  const R det = sdet(H);
  if (!(fabs(double(det)) > 1e-8) || !isfinite(double(det))) return;  // update skipped: D = 0
  const R idet = R(1) / det;
  const vec3<R> D = sadj_mul(H, f) * idet;
  const vec3<R> a = ldx(A.adj_x, v);
  const vec3<R> w = sadj_mul(H, a) * idet;
  // H_bar = -sym(w D^T)
  const sym3<R> Hb = {-w.x * D.x, -w.y * D.y, -w.z * D.z, R(-0.5) * (w.x * D.y + w.y * D.x),
                      R(-0.5) * (w.x * D.z + w.z * D.x), R(-0.5) * (w.y * D.z + w.z * D.y)};
  vec3<R> ax = zero3<R>();
  const int e8 = lane >> 2, k = lane & 3;  // eight elements at a time, four lanes each
  // membranes: three vertices and (mu, lambda)
  for (int q = c.face_off[v] + e8; q < c.face_off[v + 1]; q += 8) {
    const int t = c.face_adj[q] >> 2, ord = c.face_adj[q] & 3;
    const float4 mat = c.tri_mat[t];
    if (!(mat.x > 0.f || mat.y > 0.f)) continue;
    if (mat.z > 0.f)
      membrane_adjoint<R, 6>(A, v, t, ord, k, w, Hb, ax);
    else
      membrane_adjoint<R, 3>(A, v, t, ord, k, w, Hb, ax);
  }
  for (int q = c.edge_off[v] + e8; q < c.edge_off[v + 1]; q += 8) {
    const int e = c.edge_adj[q] >> 2, ord = c.edge_adj[q] & 3;
    const float4 pr = c.edge_prop[e];
    if (!(pr.z > 0.f)) continue;
    if (pr.w > 0.f)
      bending_adjoint<R, 6>(A, v, e, ord, k, w, Hb, ax);
    else
      bending_adjoint<R, 3>(A, v, e, ord, k, w, Hb, ax);
  }
  if (c.tet_off) {
    for (int q = c.tet_off[v] + e8; q < c.tet_off[v + 1]; q += 8) {
      const int t = c.tet_adj[q] >> 2, ord = c.tet_adj[q] & 3;
      const float4 r0 = c.tet_pose[3 * t], r1 = c.tet_pose[3 * t + 1], r2 = c.tet_pose[3 * t + 2];
      if (!(r0.w > 0.f || r1.w > 0.f)) continue;
      if (r2.w > 0.f)
        tet_adjoint<R, 6>(A, v, t, ord, k, w, Hb, ax);
      else
        tet_adjoint<R, 3>(A, v, t, ord, k, w, Hb, ax);
    }
  }
  if (c.spr_off) {
    for (int q = c.spr_off[v] + e8; q < c.spr_off[v + 1]; q += 8) spring_adjoint(A, v, c.spr_adj[q], k, w, Hb, ax);
    for (int q = c.sspr_off[v] + e8; q < c.sspr_off[v + 1]; q += 8) spring_adjoint(A, v, c.sspr_adj[q], k, w, Hb, ax);
  }
  if (c.has_contacts && lane == 0) contacts_adjoint(c, v, x, w, Hb, ax, A.adj_xp);
  __syncwarp();
  ax = {group_sum<32>(ax.x), group_sum<32>(ax.y), group_sum<32>(ax.z)};
  if (lane != 0) return;
  // inertia term: g = md (y - x)
  ax = ax + a - md * w;
  atomic_add3(A.adj_y, v, md * w);
  A.adj_x[3 * v] = ax.x;
  A.adj_x[3 * v + 1] = ax.y;
  A.adj_x[3 * v + 2] = ax.z;
}

// One color of the forward sweep on checkpoints: reads the iteration's start (X.before) and the colors it has already
// moved (X.after), writes all of its own particles into `out` (X.after's array, which needs no copy of the start).
// L lanes per vertex, so that a vertex of a cloth takes one round of faces and one of hinges.
template <typename R, int L>
__global__ void __launch_bounds__(128) k_record_color(StepCtx<R> c, ColorState<R> X, const R* __restrict__ y, R* out,
                                                      const int* __restrict__ verts, int n) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) / L, lane = threadIdx.x % L;
  const bool valid = i < n;
  const int v = valid ? verts[i] : 0;
  const R m = valid ? solve_mass(c, v) : R(0);
  vec3<R> f = zero3<R>();
  sym3<R> H = szero<R>();
  if (m != R(0)) assemble<R, L>(c, X, v, lane, f, H);
  __syncwarp();
  sum_lanes<L>(f, H);
  if (!valid || lane != 0) return;
  vec3<R> x = X.ld(v);
  if (m != R(0)) {
    const R md = m * c.dt2r;
    f = f + md * (ldx(y, v) - x);
    H = H + sdiag(md);
    const R det = sdet(H);
    if (fabs(double(det)) > 1e-8 && isfinite(double(det))) x = x + sadj_mul(H, f) * (R(1) / det);
  }
  out[3 * v] = x.x;
  out[3 * v + 1] = x.y;
  out[3 * v + 2] = x.z;
}

// y (inertial target) and the mass flag of every particle, as forward_particle computes them; y is also the first
// checkpoint
template <typename R>
__global__ void k_record_forward(StepCtx<R> c, R* y, R* ck) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.V) return;
  forward_particle(c, GlobalPos<R>{c.pos}, i);
  const vec3<R> p = ld3<R>(c.inertia[i]);
  y[3 * i] = p.x;
  y[3 * i + 1] = p.y;
  y[3 * i + 2] = p.z;
  ck[3 * i] = p.x;
  ck[3 * i + 1] = p.y;
  ck[3 * i + 2] = p.z;
}

// dL/dx of the last iterate from dL/dq_out and dL/dqd_out (q_out = x, qd_out = (x - q) / dt), the accumulators' zeros,
// and the substep's start positions where the damping and contact terms read them (c.qprev)
template <typename R>
__global__ void k_adjoint_begin(StepCtx<R> c, const R* aq, const R* aqd, R* ax, R* ay, R* axp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.V) return;
  const R inv_dt = R(1) / c.dt;
  for (int j = 3 * i; j < 3 * i + 3; ++j) {
    ax[j] = (aq ? aq[j] : R(0)) + (aqd ? aqd[j] * inv_dt : R(0));
    ay[j] = R(0);
    axp[j] = R(0);
  }
  c.qprev[i] = pk4(vec3<R>{c.q_in[3 * i], c.q_in[3 * i + 1], c.q_in[3 * i + 2]}, R(0));
}

// dL/dq_in, dL/dqd_in from dL/dy (the first iterate is y), the direct qd_out term and the contact terms' dL/dq
// (axp, or NULL)
template <typename R>
__global__ void k_adjoint_end(StepCtx<R> c, const R* ax, const R* ay, const R* axp, const R* aqd, R* aq_in,
                              R* aqd_in) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.V) return;
  const bool moves = (c.flags[i] & 1) && c.inv_mass[i] != 0.f;
  for (int j = 0; j < 3; ++j) {
    const R gy = ay[3 * i + j] + ax[3 * i + j];
    aq_in[3 * i + j] = gy - (aqd ? aqd[3 * i + j] / c.dt : R(0)) + (axp ? axp[3 * i + j] : R(0));
    if (aqd_in) aqd_in[3 * i + j] = moves ? gy * c.dt : R(0);
  }
}

// q_out = x, qd_out = (x - q) / dt
template <typename R>
__global__ void k_record_finish(StepCtx<R> c, const R* x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 3 * c.V) return;
  c.q_out[i] = x[i];
  c.qd_out[i] = (x[i] - c.q_in[i]) / c.dt;
}

}  // namespace vbd
