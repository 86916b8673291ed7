// APIC particle separation on B200 (replaces the neighbour pass of
// SolverAPIC._apply_particle_separation, solver_apic.py:1003-1064, with its
// kernels accumulate_particle_separation, 193-248, and
// apply_particle_separation_delta, 251-266).
//
// Per iteration: the hash grid of the context (dims chosen by the caller as
// the reference does: the bounds' extent over the query radius, at least 4)
// is built over the current positions with cell width query_radius, the
// positions are gathered into cell order, and one thread per cell-sorted slot
// averages the pushes of its active neighbours closer than rest_dist in the
// reference's visiting order, adds the push and clamps to the bounds inset by
// wall_margin.  The pair arithmetic uses
// individually rounded operations (no contraction into FMAs), as the
// reference's float32 expression does, so the result equals the reference's
// bit for bit.
#include "fs_build.cuh"

namespace fs {
namespace {

// positions (original order) into cell order, with the active bit in .w
struct SepGather {
  const float* x;
  const int32_t* flags;
  float4* xs;
  FS_DEV void operator()(int64_t s, int32_t i) const {
    const float3 p = ld3(x, i);
    xs[s] = make_float4(p.x, p.y, p.z, pack_pf((flags[i] & 1) ? PF_ACTIVE : 0));
  }
};

struct SepArgs {
  GridDev g;
  int64_t n;
  const float4* xs;
  float rest, qr, strength, band;
  float lo[3], hi[3];    // bounds
  float clo[3], chi[3];  // bounds inset by the wall margin
  float* delta;          // original order [n][3]
  float* x;              // original order [n][3], moved in place
};

FS_DEV float clamp_ref(float v, float lo, float hi) {  // min(max(v, lo), hi) with the reference's comparisons
  const float t = v > lo ? v : lo;
  return t < hi ? t : hi;
}

// The slot ranges of a usual query in visiting order: up to 3 x 3 rows of one
// range each (no wrap modulo dim_x), all offsets loaded at once, empty where a
// row is not there; false where the query is another one.
FS_DEV bool usual_rows(const GridDev& g, const QueryBox& b, int (&a)[9], int (&e)[9]) {
  const int nx = b.x1 - b.x0 + 1, ny = b.y1 - b.y0 + 1, nz = b.z1 - b.z0 + 1, xa = b.x0 + (1 << 20);
  const int c0 = g.mask_x >= 0 ? (xa & g.mask_x) : xa % g.dim_x;
  if (nx <= 0 || ny > 3 || nz > 3 || xa < 0 || c0 + nx > g.dim_x) return false;
  const int32_t* const o = g.off + c0;
  int wy[3], wz[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    wy[k] = wrap_axis(b.y0 + k, g.dim_y, g.mask_y) * g.dim_x;
    wz[k] = wrap_axis(b.z0 + k, g.dim_z, g.mask_z) * g.dim_x * g.dim_y;
  }
#pragma unroll
  for (int z = 0; z < 3; ++z)
#pragma unroll
    for (int y = 0; y < 3; ++y) {
      const bool in = z < nz && y < ny;
      a[z * 3 + y] = in ? __ldg(o + wz[z] + wy[y]) : 0;
      e[z * 3 + y] = in ? __ldg(o + wz[z] + wy[y] + nx) : 0;
    }
  return true;
}

// accumulate_particle_separation and apply_particle_separation_delta of one
// particle (the neighbours' positions are the gathered copies, so that the
// move needs no pass of its own).  A few of the ~27 candidates push, and a
// push costs a rounded square root and three rounded divisions: the scan notes
// the candidates within reach (a column of shared memory) and the pushes are
// evaluated afterwards, all lanes of a warp at once, in the same order.  A
// particle with more than kSepHits in reach evaluates them as it meets them.
// At 401,856 particles, two iterations with their builds: 199 us when each
// candidate was tested and pushed where it was met and the move was a pass of
// its own, 145 now (the kernel 40 of its 72 before, held by the latency of the
// table and of the candidates, a row of three at a time).
constexpr int kSepThreads = 128;
constexpr int kSepHits = 24;

__global__ void __launch_bounds__(kSepThreads, 8) k_sep_accumulate(SepArgs a) {
  __shared__ int32_t hits[kSepHits][kSepThreads];
  grid_begin();
  const int64_t s = thread_id();
  if (s >= a.n) return;
  const float4 xi = a.xs[s];
  const int32_t i = a.g.perm[s];
  if (!(pf_of(xi) & PF_ACTIVE)) {
    st3(a.delta, i, make_float3(0.f, 0.f, 0.f));
    return;
  }
  float dx_ = 0.f, dy_ = 0.f, dz_ = 0.f, count = 0.f;
  // d2 above rest^2 (1 + 1e-6) gives a rounded sqrt(d2) >= rest (at least
  // ~3 ulps above it), which the test d < rest rejects; the scan's fused d2 is
  // within a few ulps of the rounded one
  const float r2lim = __fmul_rn(__fmul_rn(a.rest, a.rest), 1.000001f), near = r2lim * 1.000002f;
  auto push = [&](int t) {
    const float4 xj = __ldg(a.xs + t);
    const float rx = __fsub_rn(xi.x, xj.x), ry = __fsub_rn(xi.y, xj.y), rz = __fsub_rn(xi.z, xj.z);
    const float d2 = dist2_rn(rx, ry, rz);
    if (!(d2 <= r2lim) || t == (int)s || !(pf_of(xj) & PF_ACTIVE)) return;
    const float d = __fsqrt_rn(d2);
    if (d > 1.0e-8f && d < a.rest) {
      const float w = __fmul_rn(a.strength, __fsub_rn(a.rest, d));
      dx_ = __fadd_rn(dx_, __fmul_rn(__fdiv_rn(rx, d), w));
      dy_ = __fadd_rn(dy_, __fmul_rn(__fdiv_rn(ry, d), w));
      dz_ = __fadd_rn(dz_, __fmul_rn(__fdiv_rn(rz, d), w));
      count = __fadd_rn(count, 1.0f);
    }
  };
  int b[9], e[9], n = kSepHits + 1;
  if (usual_rows(a.g, query_box_hash(a.g, xi.x, xi.y, xi.z, a.qr), b, e)) {
    n = 0;
#pragma unroll
    for (int k = 0; k < 9; ++k)
      for (int t = b[k]; t < e[k]; t += 2) {  // two loads in flight (one at a time: +3 %, four: the same)
        float4 xj[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) xj[j] = __ldg(a.xs + min(t + j, e[k] - 1));
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float dx = xi.x - xj[j].x, dy = xi.y - xj[j].y, dz = xi.z - xj[j].z;
          if (fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, xj[j].w))) <= near && t + j < e[k]) {  // +inf for inactive
            if (n < kSepHits) hits[n][threadIdx.x] = t + j;
            ++n;
          }
        }
      }
  }
  if (n <= kSepHits)
    for (int k = 0; k < n; ++k) push(hits[k][threadIdx.x]);
  else
    for_each_range(a.g, 0, xi.x, xi.y, xi.z, a.qr, [&](int first, int end) {
      for (int t = first; t < end; ++t) push(t);
    });
  if (count > 0.f) {
    dx_ = __fdiv_rn(dx_, count);
    dy_ = __fdiv_rn(dy_, count);
    dz_ = __fdiv_rn(dz_, count);
  } else {
    dx_ = dy_ = dz_ = 0.f;
  }
  // components that push into a wall within the band are removed
  if (xi.x <= __fadd_rn(a.lo[0], a.band) && dx_ < 0.f) dx_ = 0.f;
  if (xi.x >= __fsub_rn(a.hi[0], a.band) && dx_ > 0.f) dx_ = 0.f;
  if (xi.y <= __fadd_rn(a.lo[1], a.band) && dy_ < 0.f) dy_ = 0.f;
  if (xi.y >= __fsub_rn(a.hi[1], a.band) && dy_ > 0.f) dy_ = 0.f;
  if (xi.z <= __fadd_rn(a.lo[2], a.band) && dz_ < 0.f) dz_ = 0.f;
  if (xi.z >= __fsub_rn(a.hi[2], a.band) && dz_ > 0.f) dz_ = 0.f;
  st3(a.delta, i, make_float3(dx_, dy_, dz_));
  st3(a.x, i, make_float3(clamp_ref(__fadd_rn(xi.x, dx_), a.clo[0], a.chi[0]),
                          clamp_ref(__fadd_rn(xi.y, dy_), a.clo[1], a.chi[1]),
                          clamp_ref(__fadd_rn(xi.z, dz_), a.clo[2], a.chi[2])));
}

}  // namespace
}  // namespace fs

using namespace fs;

extern "C" {

int fs_apic_separation(fs_context* c, float* x, const int32_t* flags, int64_t n, const fs_separation_params* p,
                       float* delta, fs_stream_t stream) {
  if (!c || !p) return set_error(FS_ERR_INVALID, "fs_apic_separation: null argument");
  if (n < 0) return set_error(FS_ERR_INVALID, "fs_apic_separation: negative n");
  if (n == 0) return FS_OK;
  if (!x || !flags || !delta) return set_error(FS_ERR_INVALID, "fs_apic_separation: missing array");
  if (c->worlds) return set_error(FS_ERR_INVALID, "fs_apic_separation: needs a hash-grid context");
  if (n > c->capacity) return set_error(FS_ERR_CAPACITY, "fs_apic_separation: n > capacity");
  if (!(p->query_radius > 0.f)) return set_error(FS_ERR_INVALID, "fs_apic_separation: query_radius must be > 0");
  DeviceGuard dg(c->device);
  cudaStream_t st = (cudaStream_t)stream;
  const int iters = p->iterations > 1 ? p->iterations : 1;
  int rc;
  for (int it = 0; it < iters; ++it) {
    if ((rc = grid_build(c, n, p->query_radius, st, nullptr, nullptr, KeyPositions{x}, SepGather{x, flags, c->xs})))
      return rc;
    SepArgs a;
    a.g = grid_view(c);
    a.n = n;
    a.xs = c->xs;
    a.rest = p->rest_dist;
    a.qr = p->query_radius;
    a.strength = p->strength;
    a.band = p->wall_band;
    for (int k = 0; k < 3; ++k) {
      a.lo[k] = p->bound_lo[k];
      a.hi[k] = p->bound_hi[k];
      // (apply_particle_separation_delta, 263-264)
      a.clo[k] = p->bound_lo[k] + p->wall_margin;
      a.chi[k] = p->bound_hi[k] - p->wall_margin;
    }
    a.delta = delta;
    a.x = x;
    {
      PassScope ps_(c, P_APIC_SEPARATION, st);
      launch(k_sep_accumulate, blocks_for(n, kSepThreads), kSepThreads, 0, st, a);
    }
    if ((rc = launch_check("fs_apic_separation"))) return rc;
  }
  c->last_stream = st;
  return FS_OK;
}

}  // extern "C"
