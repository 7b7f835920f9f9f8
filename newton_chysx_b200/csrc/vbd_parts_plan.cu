// Host side of the split-instance plan (vbd_parts.cu): the cut into parts, places, ghosts and element records. The
// loops over parts run on a few threads: a large batch has millions of records.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>

#include "vbd_parts.h"

namespace vbd {

namespace {

unsigned bits(float f) {
  unsigned u;
  std::memcpy(&u, &f, 4);
  return u;
}

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
  plan.job_order.resize(plan.njobs);
  for (int j = 0; j < plan.njobs; ++j) plan.job_order[j] = j;
  std::stable_sort(plan.job_order.begin(), plan.job_order.end(), [&](int a, int b) {
    return job_v0[a + 1] - job_v0[a] > job_v0[b + 1] - job_v0[b];
  });
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
  return plan.most_places < 65536;
}

void parts_records(const PartsInput& in, const PartsPlan& plan, std::vector<uint4>& faceA,
                   std::vector<uint4>& faceB, std::vector<uint4>& hinge, std::vector<float>& kd) {
  const uint4 none = make_uint4(0u, 0u, 0u, 0u);
  faceA.assign(size_t(std::max(plan.faces, 1LL)), none);
  faceB.assign(faceA.size(), none);
  hinge.assign(size_t(std::max(plan.hinges, 1LL)), none);
  kd.assign(hinge.size(), 0.f);
  const int C = plan.C, L = plan.L;
  for_parts(plan.njobs * plan.P, in.V, [&](int part, std::vector<int>& place) {
    const int k0 = plan.part_base[part], k1 = plan.part_base[part + 1];
    for (int k = k0; k < k1; ++k) place[plan.vert[k] & 0x7fffffff] = k - k0;
    const int g0 = plan.ghost_off[size_t(part) * (C + 1)], g1 = plan.ghost_off[size_t(part) * (C + 1) + C];
    for (int g = g0; g < g1; ++g) place[plan.ghost[g]] = k1 - k0 + g - g0;
    for (int k = k0; k < k1; ++k) {
      const int v = plan.vert[k] & 0x7fffffff, c = in.color_of[v];
      const size_t r = size_t(part) * C + c;
      const int* start = &plan.start[size_t(part) * (C + 1)];
      const long long n = start[c + 1] - start[c], j = plan.slot_of[v] - start[c];
      int s = 0;
      for (int q = in.foff[v]; q < in.foff[v + 1]; ++q, ++s) {
        const int t = in.fadj[q] >> 2, ord = in.fadj[q] & 3;
        const int* ti = in.tri + 3 * size_t(t);
        const float* D = in.pose + 4 * size_t(t);
        const float* m = in.mat + 5 * size_t(t);
        // the solved vertex as vertex 0 of the triangle: the rest inverse re-expressed as in build_ell
        const double D00 = D[0], D01 = D[1], D10 = D[2], D11 = D[3];
        double P00 = D00, P01 = D01, P10 = D10, P11 = D11;
        if (ord == 1)
          P00 = D10, P01 = D11, P10 = -D00 - D10, P11 = -D01 - D11;
        else if (ord == 2)
          P00 = -D00 - D10, P01 = -D01 - D11, P10 = D00, P11 = D01;
        const float mu = m[0] * in.area[t], lm = m[1] * in.area[t];
        if (!(mu > 0.f || lm > 0.f)) continue;
        const size_t i = size_t(plan.fbase[r] + ((s / L) * n + j) * L + s % L);
        const unsigned a = unsigned(place[ti[(ord + 1) % 3]]), b = unsigned(place[ti[(ord + 2) % 3]]);
        faceA[i] = make_uint4(a | (b << 16), bits(mu), bits(lm), bits(float(P00)));
        faceB[i] = make_uint4(bits(float(P01)), bits(float(P10)), bits(float(P11)), bits(m[2]));
      }
      s = 0;
      for (int q = in.eoff[v]; q < in.eoff[v + 1]; ++q, ++s) {
        const int e = in.eadj[q] >> 2;
        const int* ei = in.edges + 4 * size_t(e);
        const float ke = in.bending[2 * size_t(e)], kl = ke > 0.f ? ke * in.rest_length[e] : 0.f;
        if (!(kl > 0.f)) continue;
        const size_t i = size_t(plan.ebase[r] + ((s / L) * n + j) * L + s % L);
        hinge[i] = make_uint4(unsigned(place[ei[0]]) | (unsigned(place[ei[1]]) << 16),
                              unsigned(place[ei[2]]) | (unsigned(place[ei[3]]) << 16), bits(in.rest_angle[e]), bits(kl));
        kd[i] = in.bending[2 * size_t(e) + 1];
      }
    }
  });
}

}  // namespace vbd
