// Split instances: the sweep of one cloth (or of a few, merged) by several CTAs at once, see vbd_parts.cu.
#pragma once
#include <vector>

#include "vbd_ell.cuh"

namespace vbd {

// The device side of a plan. A job is a run of consecutive worlds; its particles are cut into P parts, one per CTA:
// each color's particles, in index order, into P runs of equal length, so that every part has the same work in every
// color (cuts by index alone give strips of a grid up to twice the average in some colors). A part keeps the positions of its own particles (by color, then by index) and of
// the ghosts (other parts' particles that its elements touch, by color) in shared memory.
struct PartsView {
  int C;                      // colors
  int P;                      // parts per job
  int njobs;
  const int* flags;           // kFaceDamping, kHingeDamping, kFloor (a refresh rewrites it)
  int places, most_own;       // most places and most own particles of a part: the shared-memory layout
  const int* part_base;       // [parts + 1] own particles of all parts before
  const int* vert;            // [V] particle of part-local place s at part_base + s; bit 31: ghost of another part
  const int* start;           // [parts, C + 1] own places by color
  const int* ghost_off;       // [parts, C + 1] into ghost; a ghost's place is nown + (index - ghost_off[part, 0])
  const int* ghost;           // particles
  const int* ghost_part;      // the rank in the job of the part that owns each
  const int* nf;              // [parts, C] face rounds of L lanes
  const int* ne;              // [parts, C] hinge rounds
  const long long* fbase;     // [parts, C] first face record
  const long long* ebase;
  const uint4* faceA;         // the records of vbd_ell.cuh's compact layout with part-local 14-bit places (at bits 0 and
  const uint4* faceB;         //   16 of a word) and kRecordLive, round major: base + (round * n + vertex) * L + lane
  const uint4* hinge;         // places in words 0 and 1, kRecordLive in word 1
                              // FP64: as the csr layout reads its elements, the rest inverse of the triangle's own order
                              //   (the solved vertex's at bit 14 of faceA's places), mu, lambda and ke unscaled
  const float* face_area;     // read in FP64 and for records with kRecordFloor
  const float* hinge_length;  // read in FP64
  const float* hinge_kd;      // read with kHingeDamping or kFloor
  float4* contact;            // [3 V] by place: a particle's only contact with a static shape, as part_contact_add reads it
  unsigned* done;             // [P * kDoneStride] colors finished by each CTA over its jobs, zero before launch (grid)
};

constexpr int kMostPlaces = 1 << 14;  // the shared memory of an SM holds fewer
// Flags of a record's word beside its places. Live: the element has stiffness. Floor: |lambda + mu| is under the reference's
// floor of 1e-6, which the kernel applies to the coefficients times the area.
constexpr unsigned kRecordLive = 1u << 31, kRecordFloor = 1u << 30;

// Bits of PartsView::flags: some triangle, some hinge is damped, some record has kRecordFloor. In device memory, as the
// records are: a captured step follows a refresh that brings one of them or takes it away.
constexpr int kFaceDamping = 1, kHingeDamping = 2, kFloor = 4;

constexpr int kDoneStride = 32;  // one flag per 128-byte line

constexpr int kPartColors = 32;  // most colors of a plan

struct PartsConfig {
  int P = 0;           // parts per job
  bool grid = false;   // jobs in turn over the whole grid (cooperative launch); else one job on one cluster
  int L = 1;           // lanes per vertex
  bool wide = false;   // the variant for up to 896 threads (72 registers) instead of 512 (128 registers)
  int block = 0;
  size_t smem = 0;
};

template <typename R, int MODE>
const void* parts_fn(int L, bool wide);

template <typename R, int MODE>
cudaError_t launch_parts(const PartsConfig& g, const StepCtx<R>& c, const PartsView& p, int iterations, cudaStream_t st);

}  // namespace vbd

namespace vbd {

// The host side of a plan: the cut, the places, the ghosts and the layout of the records (topology only).
struct PartsInput {
  int V = 0, T = 0, E = 0, C = 0;
  const int *tri = nullptr, *edges = nullptr;                                    // topology
  const int *foff = nullptr, *fadj = nullptr, *eoff = nullptr, *eadj = nullptr;  // packed adjacency
  const int* color_of = nullptr;                                                 // [V]
};
struct PartsPlan {
  int P = 0, L = 1, njobs = 0, C = 0, most_places = 0, most_own = 0;
  std::vector<int> part_base, part_of, slot_of, vert, start, ghost_off, ghost, ghost_part, nf, ne;
  std::vector<long long> fbase, ebase;
  long long faces = 0, hinges = 0;
};

// Cuts the jobs (job_v0: first particle of each job, then V) into P parts each. False: the plan does not exist
// (a part with kMostPlaces places or more, or an element with two vertices of one color).
bool parts_plan(const PartsInput& in, const std::vector<int>& job_v0, int P, int L, PartsPlan& plan);

// The records from the packed model (device arrays of StepCtx), written by kernels on `st` where they stand, so that a
// refresh needs no synchronisation and captured steps read the new ones.
struct PartsModel {
  const int4* tri_idx;
  const float4 *tri_pose, *tri_mat;
  const int4* edge_idx;
  const float4* edge_prop;
  const int *face_off, *face_adj, *edge_off, *edge_adj;
  const int* color_of;
  int2* place_of;  // [V] part and own place of each particle
};
struct PartsRecords {
  uint4 *faceA, *faceB, *hinge;
  float *face_area, *hinge_length, *hinge_kd;
  int* flags;
};
cudaError_t parts_places(const PartsModel& m, const PartsView& p, cudaStream_t st);  // place_of, once per plan
cudaError_t parts_pack(const PartsModel& m, const PartsView& p, int L, bool f64, const PartsRecords& r,
                       cudaStream_t st);

}  // namespace vbd
