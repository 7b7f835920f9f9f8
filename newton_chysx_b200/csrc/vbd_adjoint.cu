// Launch sequences of the recorded substep and its reverse, see vbd_adjoint.cuh.
#include "vbd_adjoint.h"

#include "vbd_adjoint.cuh"

namespace vbd {

namespace {

constexpr int kRecordLanes = 16;

template <typename R>
void prepare_contacts(const StepCtx<R>& c, cudaStream_t st) {
  cudaMemsetAsync(c.slot_cnt, 0, sizeof(int) * c.V, st);
  k_contact_prepare<R><<<(c.c_max + 255) / 256, 256, 0, st>>>(c);
}

}  // namespace

template <typename R>
cudaError_t record_substep(const StepCtx<R>& c, const ColorLists& l, int iterations, R* y, R* ck, cudaStream_t st) {
  const int V = c.V;
  const size_t n3 = size_t(3) * V;
  k_record_forward<R><<<(V + 255) / 256, 256, 0, st>>>(c, y, ck);
  if (c.has_contacts) prepare_contacts(c, st);
  for (int it = 0; it < iterations; ++it) {
    R* out = ck + size_t(it + 1) * n3;
    for (size_t col = 0; col + 1 < l.offsets->size(); ++col) {
      const int a = (*l.offsets)[col], n = (*l.offsets)[col + 1] - a;
      const ColorState<R> X{ck + size_t(it) * n3, out, l.color_of, int(col)};
      const long threads = long(n) * kRecordLanes;
      if (n > 0)
        k_record_color<R, kRecordLanes>
            <<<unsigned((threads + 127) / 128), 128, 0, st>>>(c, X, y, out, l.particles + a, n);
    }
  }
  k_record_finish<R><<<int((n3 + 255) / 256), 256, 0, st>>>(c, ck + size_t(iterations) * n3);
  return cudaGetLastError();
}

template <typename R>
cudaError_t adjoint_substep(const StepCtx<R>& c, const ColorLists& l, int iterations, const R* y, const R* ck, R* work,
                            const R* aq_out, const R* aqd_out, R* aq_in, R* aqd_in, R* adj_mu, R* adj_lambda,
                            cudaStream_t st) {
  const int V = c.V;
  const size_t n3 = size_t(3) * V;
  R *ax = work, *ay = work + n3, *axp = work + 2 * n3;
  // the adjoints' start, and this substep's start positions (damping and contact terms) as its forward pass had them
  k_adjoint_begin<R><<<(V + 255) / 256, 256, 0, st>>>(c, aq_out, aqd_out, ax, ay, axp);
  if (c.has_contacts) prepare_contacts(c, st);
  for (int it = iterations - 1; it >= 0; --it)
    for (int col = int(l.offsets->size()) - 2; col >= 0; --col) {
      const int a = (*l.offsets)[col], n = (*l.offsets)[col + 1] - a;
      const ColorState<R> X{ck + size_t(it) * n3, ck + size_t(it + 1) * n3, l.color_of, col};
      const AdjCtx<R> A{c, X, y, ax, ay, adj_mu, adj_lambda, axp};
      if (n > 0) k_adjoint_color<R><<<(n + 3) / 4, 128, 0, st>>>(A, l.particles + a, n);
    }
  k_adjoint_end<R><<<(V + 255) / 256, 256, 0, st>>>(c, ax, ay, axp, aqd_out, aq_in, aqd_in);
  return cudaGetLastError();
}

#define VBD_ADJOINT(R)                                                                                             \
  template cudaError_t record_substep<R>(const StepCtx<R>&, const ColorLists&, int, R*, R*, cudaStream_t);        \
  template cudaError_t adjoint_substep<R>(const StepCtx<R>&, const ColorLists&, int, const R*, const R*, R*,      \
                                          const R*, const R*, R*, R*, R*, R*, cudaStream_t);
VBD_ADJOINT(float)
VBD_ADJOINT(double)

}  // namespace vbd
