// Cloths swept by several CTAs each: the persistent schedule for instances that are too few, or too large, to fill the
// GPU with one CTA per instance.
//
// Why. A Gauss-Seidel sweep has a barrier after every color, so its time is (colors x iterations) times the latency
// of one color. With one CTA per instance that latency is a whole color's work on one SM, and with one launch per
// color and one lane per vertex it is a launch plus a chain of 18 element evaluations (13 us per color for a
// 161 x 97 cloth as for a 256 x 256 one).
//
// How. The particles of a job are cut into parts, one per CTA. A CTA keeps its own particles' positions, inertial
// targets and its ghosts' positions in shared memory for the whole substep (16-byte loads without bank conflicts, as
// the vertices of a color sit next to each other), and L lanes of a warp share a vertex's elements. After a color,
// vertices that are ghosts elsewhere are written to global memory and fetched from L2 by the parts that read them.
// Ghosts' first positions need no exchange: every CTA predicts them itself.
//   grid = false: the only job on one cluster, barrier.cluster between colors (up to 1,024 particles: 16 CTAs).
//   grid = true:  the jobs in turn over the whole (cooperative) grid. A part waits only for the parts whose particles
//                 it reads: each publishes the colors it has finished, and the thread that fetches a ghost polls its
//                 owner's flag (bounded). Two parts that share an element read each other's particles, in two colors
//                 of an iteration at least (the plan takes no coloring with two vertices of an element in one color), so
//                 none overwrites a position that a neighbour has yet to fetch. A barrier over the grid instead (an
//                 atomic counter) cost about 3 us per color.
//
// Measured, us per substep (collide + step), before and after, 10 iterations unless said:
//   32 x 32 FP32          1,557 -> 145   (one CTA, 8 lanes per vertex, before)
//   161 x 97 FP32           517 -> 173   (40 launches of one lane per vertex)
//   256 x 256 FP32, 20 it 1,025 -> 426
//   512 x 512 mixed, 30 it 2,605 -> 1,772
//   96 x 96 FP64            791 -> 251
//   60 worlds of 16..40 squared, damped 1,126 -> 342 (one CTA per world before)
//   512 worlds of 16..128 squared (3.3 M particles) 10,101 -> 5,296: seven jobs; issue and the records' stream from
//   HBM bound it, 6.2e9 vertex-iterations/s
// What bounds the small ones now is the serial chain of a color: about 4 us of dependent instructions and loads (161 x 97:
// 19 % of issue slots used, 2.7 barrier and 2.0 long-scoreboard stalls per issue).
#include "vbd_parts.h"

#include <cooperative_groups.h>

namespace vbd {

namespace {

// A barrier wait ends after this many polls (seconds), sets VBD_DEVERR_BARRIER and the kernel returns.
constexpr unsigned kBarrierPolls = 1u << 22;
constexpr int kErrBarrier = 16;

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// waits until *flag >= target; false when the wait ran out
__device__ __forceinline__ bool wait_done(const unsigned* flag, unsigned target) {
  for (unsigned polls = 0; polls < kBarrierPolls; ++polls)
    if (ld_acquire(flag) >= target) return true;
  return false;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile(
      "barrier.cluster.arrive.release.aligned;\n\t"
      "barrier.cluster.wait.acquire.aligned;" ::
          : "memory");
}

// positions another CTA of this launch wrote: from L2, not from this SM's L1
__device__ __forceinline__ float4 ld_l2(const float4* p) { return __ldcg(p); }
__device__ __forceinline__ double4 ld_l2(const double4* p) {
  const double2 a = __ldcg(reinterpret_cast<const double2*>(p)), b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}

template <typename R>
struct PartPos {
  const pos4_t<R>* s;
  __device__ __forceinline__ vec3<R> ld(int i) const { return ld3<R>(s[i]); }
};

// Start positions of part-local places, for the damping terms: state_in's positions, which nobody writes before the
// last barrier.
template <typename R>
struct PartStart {
  const R* q;
  const int* vert;   // own places
  const int* ghost;  // ghost places, from place nown
  int nown;
  __device__ __forceinline__ vec3<R> ld(int i) const {
    const int v = i < nown ? (__ldg(vert + i) & 0x7fffffff) : __ldg(ghost + (i - nown));
    return {q[3 * size_t(v)], q[3 * size_t(v) + 1], q[3 * size_t(v) + 2]};
  }
};

// Inertial target (also the first position) and solve mass of particle v, as forward_particle has them.
template <typename R>
__device__ __forceinline__ vec3<R> predict(const StepCtx<R>& c, int v, vec3<R>& q, R& msolve) {
  q = {c.q_in[3 * size_t(v)], c.q_in[3 * size_t(v) + 1], c.q_in[3 * size_t(v) + 2]};
  const int fl = c.flags[v];
  const float im = c.inv_mass[v], m = c.mass[v];
  msolve = ((fl & 1) && m != 0.f) ? R(m) : R(0);
  if (!(fl & 1) || im == 0.f) return q;
  const vec3<R> g = {R(c.gravity[0]), R(c.gravity[1]), R(c.gravity[2])};
  vec3<R> fe = zero3<R>();
  if (c.f_ext) fe = {c.f_ext[3 * size_t(v)], c.f_ext[3 * size_t(v) + 1], c.f_ext[3 * size_t(v) + 2]};
  const vec3<R> u = vec3<R>{c.qd_in[3 * size_t(v)], c.qd_in[3 * size_t(v) + 1], c.qd_in[3 * size_t(v) + 2]} +
                    (g + fe * R(im)) * c.dt;
  return q + u * c.dt;
}

// The only contact of a particle with a static shape, laid out by place once per substep: (point, k), (normal, kd),
// (velocity, mu). contacts_add_n reaches the same values through five dependent loads per color.
template <typename A>
__device__ __forceinline__ void part_contact_add(float4 a, float4 b, float4 d, A radius, vec3<A> x0, A fric_eps, A dt,
                                                 vec3<A> x, vec3<A>& f, sym3<A>& H) {
  const vec3<A> bx = {A(a.x), A(a.y), A(a.z)}, nn = {A(b.x), A(b.y), A(b.z)}, bv = {A(d.x), A(d.y), A(d.z)};
  const A pen = -(dot(nn, x - bx) - radius);
  if (pen > A(0)) contact_add<A>(pen, nn, (x - x0) - bv * dt, A(a.w), A(b.w), A(d.w), fric_eps, dt, f, H);
}

// Places of one vertex's contacts: none, one laid out (kOneContact), or as many as its count says (contacts_add_n).
constexpr int kOneContact = 1 << 30;

// Reads the vertex's contacts at the substep's start; returns their kind for the inertia entry.
template <typename R>
__device__ __forceinline__ int lay_contact(const StepCtx<R>& c, const PartsView& p, int v, int place) {
  if (!c.has_contacts) return 0;
  const int n = c.slot_cnt[v];
  if (n != 1 || c.beta != R(0)) return n;
  const int t = c.slots[size_t(v) * c.K], s = c.c_shape[t];
  if (c.shape_body && s >= 0 && c.shape_body[s] >= 0 && c.body_q) return n;  // on a body: its motion enters
  p.contact[3 * size_t(place)] =
      make_float4(c.c_body_pos[3 * t], c.c_body_pos[3 * t + 1], c.c_body_pos[3 * t + 2], c.c_k[t]);
  p.contact[3 * size_t(place) + 1] =
      make_float4(c.c_normal[3 * t], c.c_normal[3 * t + 1], c.c_normal[3 * t + 2], c.c_kd[t]);
  p.contact[3 * size_t(place) + 2] =
      make_float4(c.c_body_vel[3 * t], c.c_body_vel[3 * t + 1], c.c_body_vel[3 * t + 2], c.c_mu[t]);
  return kOneContact;
}

// One vertex by L lanes (all lanes of the warp call this). fb, eb: this lane's first records; stride: records per
// round.
template <typename R, int MODE, int L, bool GENERAL, bool EARLY>
__device__ __forceinline__ void solve_part(const StepCtx<R>& c, const PartsView& p, pos4_t<R>* s_pos,
                                           const pos4_t<R>* s_y, const int* s_kind, const int v0,
                                           const PartStart<R>& start, int slot, bool valid, int lane, int nf, int ne,
                                           long long fb, long long eb, int stride, int iteration) {
  const PartPos<R> pos{s_pos};
  vec3<R> f = zero3<R>();
  sym3<R> H = szero<R>();
  pos4_t<R> in4 = pk4(zero3<R>(), R(0));
  if (valid) in4 = s_y[slot];
  const R m = R(in4.w);
  const bool active = valid && m != R(0);
  int code = 0, kind = 0;
  float4 ca = make_float4(0.f, 0.f, 0.f, 0.f), cn = ca, cv = ca;
  float radius = 0.f;
  vec3<R> x0 = zero3<R>();
  const auto read_contact = [&]() {
    code = __ldg(p.vert + v0 + slot);
    kind = s_kind[slot];
    if (kind == kOneContact) {
      const float4* q = p.contact + 3 * size_t(v0 + slot);
      ca = q[0], cn = q[1], cv = q[2];
      radius = c.radius[code & 0x7fffffff];
      x0 = ld3<R>(c.qprev[code & 0x7fffffff]);
    }
  };
  if (active) {
    if (EARLY && lane == 0) read_contact();  // in flight during the element loops
    const vec3<R> x = pos.ld(slot);
    const uint4* pa = p.faceA + fb;
    const uint4* pb = p.faceB + fb;
    const uint4* ph = p.hinge + eb;
    const float* pk = GENERAL ? p.hinge_kd + eb : nullptr;
    uint4 A_n = make_uint4(0u, 0u, 0u, 0u), B_n = A_n, h_n = A_n;
    if (nf > 0) A_n = __ldg(pa), B_n = __ldg(pb);
    if (ne > 0) h_n = __ldg(ph);  // the first hinge record loads under the faces
    for (int s = 0; s < nf; ++s) {
      const uint4 A = A_n, B = B_n;
      if (s + 1 < nf) {
        pa += stride;
        pb += stride;
        A_n = __ldg(pa);
        B_n = __ldg(pb);
      }
      if (!(A.x & kRecordLive)) continue;
      const float muA = __uint_as_float(A.y), lmA = __uint_as_float(A.z);
      const R pose[4] = {R(__uint_as_float(A.w)), R(__uint_as_float(B.x)), R(__uint_as_float(B.y)),
                         R(__uint_as_float(B.z))};
      const float kd = __uint_as_float(B.w);
      const int ia = int(A.x & (kMostPlaces - 1)), ib = int((A.x >> 16) & (kMostPlaces - 1));
      vec3<R> xp[3];
      if constexpr (sizeof(R) == 8) {
        const int ord = int((A.x >> 14) & 3u);  // the triangle's vertices in its own order: (slot, a, b) from vertex `ord` on
        const int i0 = ord == 0 ? slot : (ord == 1 ? ib : ia), i1 = ord == 0 ? ia : (ord == 1 ? slot : ib);
        const int i2 = ord == 0 ? ib : (ord == 1 ? ia : slot);
        if (kd > 0.f) xp[0] = start.ld(i0), xp[1] = start.ld(i1), xp[2] = start.ld(i2);
        const R area = R(__ldg(p.face_area + fb + (long long)s * stride));
        membrane_add<R>(ord, pos.ld(i0), pos.ld(i1), pos.ld(i2), pose, R(muA), R(lmA), R(kd), area, c.dt, xp, f, H);
        continue;
      }
      if (kd > 0.f) xp[0] = start.ld(slot), xp[1] = start.ld(ia), xp[2] = start.ld(ib);
      if constexpr (GENERAL) {
        if (A.x & kRecordFloor) {
          const R lnh_floor = R(1.0e-6) * R(__ldg(p.face_area + fb + (long long)s * stride));
          membrane_add<R>(0, x, pos.ld(ia), pos.ld(ib), pose, R(muA), R(lmA), R(kd), R(1), c.dt, xp, f, H, lnh_floor);
          continue;
        }
      }
      membrane_add<R>(0, x, pos.ld(ia), pos.ld(ib), pose, R(muA), R(lmA), R(kd), R(1), c.dt, xp, f, H, R(0));
    }
    for (int s = 0; s < ne; ++s) {
      const uint4 hh = h_n;
      float kd = 0.f;
      if constexpr (GENERAL) {
        kd = __ldg(pk);
        pk += stride;
      }
      if (s + 1 < ne) {
        ph += stride;
        h_n = __ldg(ph);
      }
      if (!(hh.y & kRecordLive)) continue;
      const float k = __uint_as_float(hh.w);
      R length = R(1);
      if constexpr (sizeof(R) == 8) length = R(__ldg(p.hinge_length + eb + (long long)s * stride));
      const int i0 = int(hh.x & 0xffffu), i1 = int(hh.x >> 16);
      const int i2 = int(hh.y & 0xffffu), i3 = int((hh.y >> 16) & (kMostPlaces - 1));
      // the solved vertex's role is where its place appears (bending_add_coef's constants)
      const bool r0 = i0 == slot, r1 = i1 == slot, r2 = i2 == slot, r3 = !(r0 || r1 || r2);
      const R ca = r0 ? R(-1) : (r2 ? R(1) : R(0));
      const R cb = r1 ? R(-1) : (r3 ? R(1) : R(0));
      const R dd = r2 ? R(1) : (r3 ? R(-1) : R(0));
      const vec3<R> xs[4] = {pos.ld(i0), pos.ld(i1), pos.ld(i2), pos.ld(i3)};
      const R rest = R(__uint_as_float(hh.z));
      if constexpr (GENERAL) {
        if (kd > 0.f) {
          const vec3<R> xp[4] = {start.ld(i0), start.ld(i1), start.ld(i2), start.ld(i3)};
          bending_add_coef<R>(ca, cb, dd, xs, rest, length, R(k), R(kd), c.dt, xp, f, H);
          continue;
        }
      }
      bending_add_coef<R>(ca, cb, dd, xs, rest, length, R(k), R(0), c.dt, nullptr, f, H);
    }
  }
  if (L > 1) {
    f.x = group_sum<L>(f.x);
    f.y = group_sum<L>(f.y);
    f.z = group_sum<L>(f.z);
    H.xx = group_sum<L>(H.xx);
    H.yy = group_sum<L>(H.yy);
    H.zz = group_sum<L>(H.zz);
    H.xy = group_sum<L>(H.xy);
    H.xz = group_sum<L>(H.xz);
    H.yz = group_sum<L>(H.yz);
  }
  if (!active || lane != 0) return;
  if (!EARLY) read_contact();
  const vec3<R> x = pos.ld(slot);
  const R md = m * c.dt2r;
  f = f + md * (ld3<R>(in4) - x);
  H.xx += md;
  H.yy += md;
  H.zz += md;
  vec3<R> dlt;
  double r2;
  const int v = code & 0x7fffffff;
  const auto contacts = [&](auto xa, auto& fa, auto& Ha) {
    using A = decltype(xa.x);
    if (kind == kOneContact)
      part_contact_add<A>(ca, cn, cv, A(radius), vec3<A>{A(x0.x), A(x0.y), A(x0.z)}, A(c.fric_eps), A(c.dt), xa, fa, Ha);
    else
      contacts_add_n<R, A>(c, v, kind, xa, fa, Ha);
  };
  const double det_used = solve_with_contacts<R, MODE>(c, kind > 0, contacts, x, f, H, nullptr, dlt, r2);
  if (MODE == MODE_MIXED && c.residual) residual_add(c.residual, iteration, r2);
  if (MODE == MODE_FP32) {  // the same tests on the FP32 determinant, without FP64 conversions on the critical path
    const float d = float(det_used);
    if (!isfinite(d)) {
      set_err(c.err, 1);
      return;
    }
    if (!(fabsf(d) > 1e-8f)) {
      set_err(c.err, 4);
      return;
    }
  } else {
    if (!isfinite(det_used)) {
      set_err(c.err, 1);
      return;
    }
    if (!(fabs(det_used) > 1e-8)) {
      set_err(c.err, 4);
      return;
    }
  }
  const vec3<R> xn = x + dlt;
  if (!(isfinite(xn.x) && isfinite(xn.y) && isfinite(xn.z))) {
    set_err(c.err, 1);
    return;
  }
  s_pos[slot] = pk4(xn, R(0));
  if (code < 0) c.pos[v] = pk4(xn, R(0));
}

// The job's plan entries of this part in shared memory.
struct PartShared {
  int abort;
  int start[kPartColors + 1], go[kPartColors + 1], nf[kPartColors], ne[kPartColors];
  long long fb[kPartColors], eb[kPartColors];
};

// The iterations of one job. False: a wait ran out.
template <typename R, int MODE, int L, bool GENERAL, bool EARLY>
__device__ __forceinline__ bool sweep_part(const StepCtx<R>& c, const PartsView& p, PartShared& s, pos4_t<R>* s_pos,
                                           const pos4_t<R>* s_y, const int* s_kind, int v0, int nown, int g0,
                                           const PartStart<R>& start, int rank, int grid_mode, int iterations,
                                           unsigned& phase) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int group = tid / L, lane = tid % L, per_round = nt / L;
  for (int it = 0; it < iterations; ++it)
    for (int col = 0; col < p.C; ++col) {
      const int a = s.start[col], n = s.start[col + 1] - a;
      const int nf = s.nf[col], ne = s.ne[col];
      const long long fb = s.fb[col], eb = s.eb[col];
      const int gb = s.go[col], ge = s.go[col + 1];
      int mine = 0, owner = 0;  // this thread's ghost, known before the wait
      if (gb + tid < ge) mine = __ldg(p.ghost + gb + tid), owner = __ldg(p.ghost_part + gb + tid);
      for (int base = 0; base < n; base += per_round) {
        const int j = base + group;
        const long long o = (long long)j * L + lane;
        solve_part<R, MODE, L, GENERAL, EARLY>(c, p, s_pos, s_y, s_kind, v0, start, a + j, j < n, lane, nf, ne,
                                                     fb + o, eb + o, n * L, it);
      }
      if (p.P > 1) {
        if (grid_mode) {
          __syncthreads();
          ++phase;
          if (tid == 0) st_release(p.done + rank * kDoneStride, phase);
          if (gb + tid < ge && !wait_done(p.done + owner * kDoneStride, phase)) s.abort = 1;
        } else {
          cluster_barrier();
        }
        if (gb + tid < ge) s_pos[nown + gb + tid - g0] = ld_l2(c.pos + mine);
        for (int g = gb + tid + nt; g < ge; g += nt) {
          if (grid_mode && !wait_done(p.done + __ldg(p.ghost_part + g) * kDoneStride, phase)) s.abort = 1;
          s_pos[nown + g - g0] = ld_l2(c.pos + __ldg(p.ghost + g));
        }
      }
      __syncthreads();
      if (grid_mode && s.abort) {  // a wait ran out: report and leave
        if (tid == 0) set_err(c.err, kErrBarrier);
        return false;
      }
    }
  return true;
}

// T: threads that the register budget allows, 512 (128 registers) for the latency of few vertices, 896 (72 registers)
// where a part's colors have enough work to fill them, 384 in FP64.
template <typename R, int MODE, int L, int T>
__global__ void __launch_bounds__(T, 1)
    k_parts(const __grid_constant__ StepCtx<R> c, const __grid_constant__ PartsView p, int grid_mode, int iterations) {
  extern __shared__ __align__(32) unsigned char s_raw[];
  pos4_t<R>* s_pos = reinterpret_cast<pos4_t<R>*>(s_raw);
  __shared__ PartShared s;
  namespace cg = cooperative_groups;
  const int rank = grid_mode ? int(blockIdx.x) : int(cg::this_cluster().block_rank());
  const int tid = threadIdx.x, nt = blockDim.x;
  const int flags = *p.flags;
  unsigned phase = 0;
  if (tid == 0) s.abort = 0;
  for (int job = 0; job < p.njobs; ++job) {
    __syncthreads();
    const int part = job * p.P + rank;
    const int v0 = __ldg(p.part_base + part), nown = __ldg(p.part_base + part + 1) - v0;
    const int* go = p.ghost_off + size_t(part) * (p.C + 1);
    const int g0 = __ldg(go), g1 = __ldg(go + p.C);
    const PartStart<R> start{c.q_in, p.vert + v0, p.ghost + g0, nown};
    pos4_t<R>* s_y = s_pos + p.places;
    int* s_kind = reinterpret_cast<int*>(s_y + p.most_own);
    if (tid <= p.C) {
      s.go[tid] = __ldg(go + tid);
      s.start[tid] = __ldg(p.start + part * (p.C + 1) + tid);
      if (tid < p.C) {
        s.nf[tid] = __ldg(p.nf + part * p.C + tid);
        s.ne[tid] = __ldg(p.ne + part * p.C + tid);
        s.fb[tid] = __ldg(p.fbase + part * p.C + tid);
        s.eb[tid] = __ldg(p.ebase + part * p.C + tid);
      }
    }
    for (int slot = tid; slot < nown; slot += nt) {
      const int code = __ldg(p.vert + v0 + slot), v = code & 0x7fffffff;
      vec3<R> q;
      R ms;
      const vec3<R> y = predict(c, v, q, ms);
      c.qprev[v] = pk4(q, R(0));
      s_y[slot] = pk4(y, ms);
      s_pos[slot] = pk4(y, R(0));
      s_kind[slot] = lay_contact(c, p, v, v0 + slot);
      if (code < 0) c.pos[v] = pk4(y, R(0));  // a ghost's position also where no solve moves it
    }
    if (iterations > 0)
      for (int g = g0 + tid; g < g1; g += nt) {
        vec3<R> q;
        R ms;
        s_pos[nown + g - g0] = pk4(predict(c, __ldg(p.ghost + g), q, ms), R(0));
      }
    __syncthreads();
    // A sweep of its own for models without damped hinges and triangles under the floor: deciding per element took 5 %
    // (32 x 32, 256 x 256) to 13 % (512 worlds) of their steps for the hinges and 3 to 8 % for the floor. Both in one
    // kernel take 1 (512 x 512) to 3 % (32 x 32: 4 us) against two kernels, between which a captured step could not
    // change.
    const bool done = flags & (kHingeDamping | kFloor)
                          ? sweep_part<R, MODE, L, true, (T <= 512)>(c, p, s, s_pos, s_y, s_kind, v0, nown, g0, start,
                                                                     rank, grid_mode, iterations, phase)
                          : sweep_part<R, MODE, L, false, (T <= 512)>(c, p, s, s_pos, s_y, s_kind, v0, nown, g0, start,
                                                                      rank, grid_mode, iterations, phase);
    if (!done) return;
    // the damping terms read ghosts' start positions from state_in: their owners write it back when all have finished
    if (grid_mode && (flags & (kFaceDamping | kHingeDamping))) {
      for (int g = g0 + tid; g < g1; g += nt)
        if (!wait_done(p.done + __ldg(p.ghost_part + g) * kDoneStride, phase)) s.abort = 1;
      __syncthreads();
      if (s.abort) {
        if (tid == 0) set_err(c.err, kErrBarrier);
        return;
      }
    }
    __syncthreads();
    for (int slot = tid; slot < nown; slot += nt) {
      const int v = __ldg(p.vert + v0 + slot) & 0x7fffffff;
      const vec3<R> x = ld3<R>(s_pos[slot]);
      const vec3<R> u = (x - ld3<R>(c.qprev[v])) * (R(1) / c.dt);
      c.q_in[3 * size_t(v)] = x.x, c.q_in[3 * size_t(v) + 1] = x.y, c.q_in[3 * size_t(v) + 2] = x.z;
      c.q_out[3 * size_t(v)] = x.x, c.q_out[3 * size_t(v) + 1] = x.y, c.q_out[3 * size_t(v) + 2] = x.z;
      c.qd_out[3 * size_t(v)] = u.x, c.qd_out[3 * size_t(v) + 1] = u.y, c.qd_out[3 * size_t(v) + 2] = u.z;
    }
  }
}

}  // namespace

template <typename R, int MODE>
const void* parts_fn(int L, bool wide) {
  if constexpr (sizeof(R) == 4) {
    if (wide) return L == 1 ? (const void*)k_parts<R, MODE, 1, 896> : (const void*)k_parts<R, MODE, 2, 896>;
  }
  constexpr int T = sizeof(R) == 4 ? 512 : 384;
  switch (L) {
    case 1: return (const void*)k_parts<R, MODE, 1, T>;
    case 2: return (const void*)k_parts<R, MODE, 2, T>;
    case 4: return (const void*)k_parts<R, MODE, 4, T>;
    default: return (const void*)k_parts<R, MODE, 8, T>;
  }
}

template <typename R, int MODE>
cudaError_t launch_parts(const PartsConfig& g, const StepCtx<R>& c, const PartsView& p, int iterations, cudaStream_t st) {
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g.P);
  cfg.blockDim = dim3(g.block);
  cfg.dynamicSmemBytes = g.smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (g.grid) {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  } else {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = g.P;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  }
  int grid_mode = g.grid ? 1 : 0;
  void* args[] = {(void*)&c, (void*)&p, (void*)&grid_mode, (void*)&iterations};
  return cudaLaunchKernelExC(&cfg, parts_fn<R, MODE>(g.L, g.wide), args);
}

#define VBD_PARTS(R, MODE)                                                                                       \
  template const void* parts_fn<R, MODE>(int, bool);                                                            \
  template cudaError_t launch_parts<R, MODE>(const PartsConfig&, const StepCtx<R>&, const PartsView&, int, cudaStream_t);
VBD_PARTS(float, MODE_FP32)
VBD_PARTS(float, MODE_MIXED)
VBD_PARTS(double, MODE_FP64)

}  // namespace vbd
