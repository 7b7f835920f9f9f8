// The split-instance plan (vbd_parts.cu): on the host the cut into parts, places and ghosts, once; on the device the
// element records, at creation and at every refresh of the model.
#include <algorithm>
#include <atomic>
#include <thread>

#include "vbd_parts.h"

namespace vbd {

namespace {

// f(part, scratch) for every part; scratch: an int per particle, its contents left from other parts
template <typename F>
void for_parts(int parts, int V, F f) {
  // a thread per 4,096 particles: below that its start costs more than it saves
  const int threads = std::max(1, std::min({int(std::thread::hardware_concurrency()), 8, parts, V >> 12}));
  std::atomic<int> next{0};
  auto work = [&]() {
    std::vector<int> scratch(V, -1);
    for (int k = next++; k < parts; k = next++) f(k, scratch);
  };
  std::vector<std::thread> pool;
  for (int t = 1; t < threads; ++t) pool.emplace_back(work);
  work();
  for (auto& t : pool) t.join();
}

// the other vertices of v's elements
template <typename F>
void neighbours(const PartsInput& in, int v, F f) {
  for (int q = in.foff[v]; q < in.foff[v + 1]; ++q) {
    const int* t = in.tri + 3 * size_t(in.fadj[q] >> 2);
    f(t[0]), f(t[1]), f(t[2]);
  }
  for (int q = in.eoff[v]; q < in.eoff[v + 1]; ++q) {
    const int* e = in.edges + 4 * size_t(in.eadj[q] >> 2);
    for (int k = 0; k < 4; ++k) f(e[k]);
  }
}

}  // namespace

bool parts_plan(const PartsInput& in, const std::vector<int>& job_v0, int P, int L, PartsPlan& plan) {
  const int V = in.V, C = in.C;
  // Vertices of an element in one color (a coloring without the hinges leaves opposite vertices so) would break the flags'
  // argument in vbd_parts.cu; whatever the element's stiffness, which a refresh can switch on. Also rules out an element
  // that names a vertex twice.
  const auto apart = [&](const int* x, int n) {
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < i; ++j)
        if (in.color_of[x[i]] == in.color_of[x[j]]) return false;
    return true;
  };
  for (int t = 0; t < in.T; ++t)
    if (!apart(in.tri + 3 * size_t(t), 3)) return false;
  for (int e = 0; e < in.E; ++e) {
    const int* x = in.edges + 4 * size_t(e);
    if (x[0] < 0 || x[1] < 0) continue;  // a boundary hinge: no record
    if (!apart(x, 4)) return false;
  }
  plan = PartsPlan();
  plan.P = P, plan.L = L, plan.C = C;
  plan.njobs = int(job_v0.size()) - 1;
  const int parts = plan.njobs * P;
  plan.part_of.assign(V, 0);
  plan.slot_of.assign(V, 0);
  plan.vert.assign(V, 0);
  plan.part_base.assign(size_t(parts) + 1, 0);
  plan.start.assign(size_t(parts) * (C + 1), 0);
  for (int job = 0; job < plan.njobs; ++job) {
    std::vector<int> count(C, 0), rank(C, 0);
    for (int v = job_v0[job]; v < job_v0[job + 1]; ++v) ++count[in.color_of[v]];
    for (int v = job_v0[job]; v < job_v0[job + 1]; ++v) {
      const int c = in.color_of[v];
      plan.part_of[v] = job * P + int((long long)rank[c]++ * P / count[c]);
      ++plan.start[size_t(plan.part_of[v]) * (C + 1) + c + 1];
    }
  }
  for (int part = 0; part < parts; ++part) {
    int* start = &plan.start[size_t(part) * (C + 1)];
    for (int c = 0; c < C; ++c) start[c + 1] += start[c];
    plan.part_base[part + 1] = plan.part_base[part] + start[C];
    plan.most_own = std::max(plan.most_own, start[C]);
  }
  {
    std::vector<int> at(size_t(parts) * C);
    for (int part = 0; part < parts; ++part)
      for (int c = 0; c < C; ++c) at[size_t(part) * C + c] = plan.start[size_t(part) * (C + 1) + c];
    for (int v = 0; v < V; ++v) {
      const int part = plan.part_of[v];
      plan.slot_of[v] = at[size_t(part) * C + in.color_of[v]]++;
      plan.vert[plan.part_base[part] + plan.slot_of[v]] = v;
    }
  }
  plan.nf.assign(size_t(parts) * C, 0);
  plan.ne.assign(size_t(parts) * C, 0);
  std::vector<std::vector<int>> ghosts(parts);
  for_parts(parts, V, [&](int part, std::vector<int>& seen) {
    std::vector<int>& g = ghosts[part];
    for (int k = plan.part_base[part]; k < plan.part_base[part + 1]; ++k) {
      const int v = plan.vert[k], c = in.color_of[v];
      int &nf = plan.nf[size_t(part) * C + c], &ne = plan.ne[size_t(part) * C + c];
      nf = std::max(nf, (in.foff[v + 1] - in.foff[v] + L - 1) / L);
      ne = std::max(ne, (in.eoff[v + 1] - in.eoff[v] + L - 1) / L);
      neighbours(in, v, [&](int u) {
        if (plan.part_of[u] != part && seen[u] != part) {
          seen[u] = part;
          g.push_back(u);
        }
      });
    }
    std::sort(g.begin(), g.end(), [&](int a, int b) {
      return in.color_of[a] != in.color_of[b] ? in.color_of[a] < in.color_of[b] : a < b;
    });
  });
  plan.ghost_off.assign(size_t(parts) * (C + 1), 0);
  plan.fbase.assign(size_t(parts) * C, 0);
  plan.ebase.assign(size_t(parts) * C, 0);
  for (int part = 0; part < parts; ++part) {
    int* off = &plan.ghost_off[size_t(part) * (C + 1)];
    const int g0 = int(plan.ghost.size());
    for (int u : ghosts[part]) {
      ++off[in.color_of[u] + 1];
      plan.ghost.push_back(u);
      plan.ghost_part.push_back(plan.part_of[u] % P);
    }
    off[0] = g0;
    for (int c = 0; c < C; ++c) {
      off[c + 1] += off[c];
      const size_t r = size_t(part) * C + c;
      const int* start = &plan.start[size_t(part) * (C + 1)];
      const long long n = start[c + 1] - start[c];
      plan.fbase[r] = plan.faces, plan.ebase[r] = plan.hinges;
      plan.faces += n * L * plan.nf[r], plan.hinges += n * L * plan.ne[r];
    }
    const int places = plan.part_base[part + 1] - plan.part_base[part] + int(ghosts[part].size());
    plan.most_places = std::max(plan.most_places, places);
  }
  std::vector<char> shared(V, 0);
  for (int u : plan.ghost) shared[u] = 1;
  for (int& v : plan.vert)
    if (shared[v]) v = int(unsigned(v) | 0x80000000u);
  return plan.most_places < kMostPlaces;
}

namespace {

__global__ void k_parts_places(const PartsView p, int2* place_of) {
  const int part = blockIdx.x, k0 = p.part_base[part], k1 = p.part_base[part + 1];
  for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) place_of[p.vert[k] & 0x7fffffff] = make_int2(part, k - k0);
}

// A block per part and slice of its particles, a thread per particle. Bound by the scattered reads of elements and places;
// a refresh of a 256 x 256 sheet takes 0.7 ms with it (12 ms with the records built on the host and uploaded), of 512
// worlds of side U{16..128} (3.3 M particles, 1.3 GB of records) 68 ms, most of it the check of the materials (901 ms).
constexpr int kPackSlices = 4;
template <bool F64>
__global__ void __launch_bounds__(256) k_parts_pack(const PartsModel m, const PartsView p, int L, const PartsRecords r) {
  const int part = blockIdx.x, C = p.C;
  const int k0 = p.part_base[part], k1 = p.part_base[part + 1], nown = k1 - k0;
  const int* go = p.ghost_off + size_t(part) * (C + 1);
  const int* start = p.start + size_t(part) * (C + 1);
  const int g0 = go[0];
  // a neighbour's place: its own, or by its id among the part's ghosts of its color
  const auto place = [&](int u) -> unsigned {
    const int2 q = m.place_of[u];
    if (q.x == part) return unsigned(q.y);
    const int c = m.color_of[u];
    int lo = go[c], hi = go[c + 1];
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (p.ghost[mid] < u)
        lo = mid + 1;
      else
        hi = mid;
    }
    return unsigned(nown + lo - g0);
  };
  int flags = 0;
  for (int k = k0 + blockIdx.y * blockDim.x + threadIdx.x; k < k1; k += kPackSlices * blockDim.x) {
    const int v = p.vert[k] & 0x7fffffff, c = m.color_of[v];
    const size_t range = size_t(part) * C + c;
    const long long n = start[c + 1] - start[c], j = k - k0 - start[c];
    int s = 0;
    for (int q = m.face_off[v]; q < m.face_off[v + 1]; ++q, ++s) {
      const int t = m.face_adj[q] >> 2, ord = m.face_adj[q] & 3;
      const int4 ti = m.tri_idx[t];
      const float4 D = m.tri_pose[t], mat = m.tri_mat[t];  // mat: mu, lambda, damping, area
      const size_t i = size_t(p.fbase[range] + ((s / L) * n + j) * L + s % L);
      const double area = mat.w;
      const float mu = mat.x * mat.w, lambda = mat.y * mat.w;
      if (!(F64 ? mat.x * area > 0.0 || mat.y * area > 0.0 : mu > 0.f || lambda > 0.f)) {
        r.faceA[i] = r.faceB[i] = make_uint4(0u, 0u, 0u, 0u);
        continue;
      }
      if (mat.z > 0.f) flags |= kFaceDamping;
      const unsigned a = place(ord == 0 ? ti.y : (ord == 1 ? ti.z : ti.x));
      const unsigned b = place(ord == 0 ? ti.z : (ord == 1 ? ti.x : ti.y));
      r.face_area[i] = mat.w;
      if constexpr (F64) {  // products and a re-expressed rest inverse rounded to FP32 would cost 1e-12 m per substep
        r.faceA[i] = make_uint4(a | (unsigned(ord) << 14) | (b << 16) | kRecordLive, __float_as_uint(mat.x),
                                __float_as_uint(mat.y), __float_as_uint(D.x));
        r.faceB[i] = make_uint4(__float_as_uint(D.y), __float_as_uint(D.z), __float_as_uint(D.w), __float_as_uint(mat.z));
        continue;
      }
      // the solved vertex as vertex 0 of the triangle: the rest inverse re-expressed for that (vbd_ell.cuh)
      double P00 = D.x, P01 = D.y, P10 = D.z, P11 = D.w;
      if (ord == 1)
        P00 = D.z, P01 = D.w, P10 = -double(D.x) - D.z, P11 = -double(D.y) - D.w;
      else if (ord == 2)
        P00 = -double(D.x) - D.z, P01 = -double(D.y) - D.w, P10 = D.x, P11 = D.y;
      const unsigned floor = fabsf(mat.y + mat.x) >= 1.0e-6f ? 0u : kRecordFloor;
      if (floor) flags |= kFloor;
      r.faceA[i] = make_uint4(a | (b << 16) | kRecordLive | floor, __float_as_uint(mu),
                              __float_as_uint(lambda), __float_as_uint(float(P00)));
      r.faceB[i] = make_uint4(__float_as_uint(float(P01)), __float_as_uint(float(P10)), __float_as_uint(float(P11)),
                              __float_as_uint(mat.z));
    }
    s = 0;
    for (int q = m.edge_off[v]; q < m.edge_off[v + 1]; ++q, ++s) {
      const int e = m.edge_adj[q] >> 2;
      const int4 ei = m.edge_idx[e];
      const float4 pr = m.edge_prop[e];  // rest angle, rest length, ke, kd
      const size_t i = size_t(p.ebase[range] + ((s / L) * n + j) * L + s % L);
      if (!(pr.z > 0.f)) {
        r.hinge[i] = make_uint4(0u, 0u, 0u, 0u);
        r.hinge_kd[i] = 0.f;
        continue;
      }
      if (pr.w > 0.f) flags |= kHingeDamping;
      r.hinge[i] = make_uint4(place(ei.x) | (place(ei.y) << 16), place(ei.z) | (place(ei.w) << 16) | kRecordLive,
                              __float_as_uint(pr.x), __float_as_uint(F64 ? pr.z : pr.z * pr.y));
      if constexpr (F64) r.hinge_length[i] = pr.y;
      r.hinge_kd[i] = pr.w;
    }
  }
  if (flags) atomicOr(r.flags, flags);
}

}  // namespace

cudaError_t parts_places(const PartsModel& m, const PartsView& p, cudaStream_t st) {
  k_parts_places<<<p.njobs * p.P, 256, 0, st>>>(p, m.place_of);
  return cudaGetLastError();
}

cudaError_t parts_pack(const PartsModel& m, const PartsView& p, int L, bool f64, const PartsRecords& r,
                       cudaStream_t st) {
  const cudaError_t rc = cudaMemsetAsync(r.flags, 0, sizeof(int), st);
  if (rc != cudaSuccess) return rc;
  const dim3 grid(p.njobs * p.P, kPackSlices);
  if (f64)
    k_parts_pack<true><<<grid, 256, 0, st>>>(m, p, L, r);
  else
    k_parts_pack<false><<<grid, 256, 0, st>>>(m, p, L, r);
  return cudaGetLastError();
}

}  // namespace vbd
