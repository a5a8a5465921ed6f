// gi_inputs.cu -- the passes that feed the GI path (SSVGIRenderer.h:61-205):
// G-buffer, shadow map and direct light.  The reference rasterises meshes; here
// the scene is ray cast through the pixel centres, two pixels a thread: those of the
// procedural primitives (boxes and spheres inside a room) that the bounds of a warp's
// rays meet; with the triangle meshes of a loaded scene one pixel a thread, those after
// the primitives, object by object behind a bounds test.
#include <type_traits>

#include "gi_device.cuh"
#include "gi_internal.h"
#include "gi_kernels.h"

namespace gi {
namespace {

using namespace dev;

constexpr int kTx = 32, kTy = 4;          // direct light: one row of 32 pixels a warp
// Ray casts: a CTA's pixels, in warps of 8 x (4 kPixels).  Without meshes a thread takes
// two pixels, 4 rows apart, which share the bounds of their warp's primitives.  The triangle
// loops share nothing and would run one after the other, so with meshes it takes one, and a
// CTA fewer threads, for more CTAs of small images.  G-buffer of 64 objects of 512 triangles
// at 200 x 120, 640 x 360 and 1920 x 1080: 845, 1126 and 3368 us with two pixels, 585, 732
// and 2661 with one; of one object of 20000 triangles at 200 x 120 10.7 and 5.2 ms.
template <bool MESH> struct Cast {
  static constexpr int kPixels = MESH ? 1 : 2, kThreads = MESH ? 128 : 256;
  static constexpr int kX = 32, kY = kPixels * kThreads / kX;  // pixels of a CTA
};
constexpr int kPrimStage = 256;  // primitives staged per shared-memory batch
constexpr int kOwnPrims = 4;     // of them that a lane bounds at a time

struct ViewArgs {
  Mat4 inv_view_proj, inv_view, view_proj, view;
  int width, height;
};

ViewArgs view_args(const gi_view& v) {
  ViewArgs a;
  for (int k = 0; k < 16; k++) {
    a.inv_view_proj.m[k] = v.inv_view_proj[k];
    a.inv_view.m[k] = v.inv_view[k];
    a.view_proj.m[k] = v.view_proj[k];
    a.view.m[k] = v.view[k];
  }
  a.width = v.width;
  a.height = v.height;
  return a;
}

struct Hit {
  float t;
  int prim;  // analytic primitive hit, or -1
  int tri;   // triangle hit (when prim == -1), or -1
  int obj;   // the triangle's object
  float u, v;
};

// Triangle meshes of a loaded scene (num_objects == 0: none).
struct MeshSet {
  const gi_mesh_object* objects;
  const gi_triangle* tris;
  int num_objects;
  int cull;  // GI_CULL_BACK: only triangles whose right-hand winding faces the ray (det > 0)
};

__device__ __forceinline__ f3 ld3(const float (&p)[3]) { return mk3(__ldg(p + 0), __ldg(p + 1), __ldg(p + 2)); }

// The mesh part of the ray cast: each object's bounds (slab test), then its
// triangles (Moller-Trumbore, t > 0, nearer than the hit so far).
__device__ void cast_mesh(const MeshSet& m, f3 o, f3 d, const float (&iv)[3], Hit& h) {
  const float ov[3] = {o.x, o.y, o.z};
  for (int k = 0; k < m.num_objects; k++) {
    const gi_mesh_object& ob = m.objects[k];
    float tn = 0.0f, tf = h.t;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float a = (__ldg(ob.lo + c) - ov[c]) * iv[c];
      const float b = (__ldg(ob.hi + c) - ov[c]) * iv[c];
      tn = gmax(tn, gmin(a, b));
      tf = gmin(tf, gmax(a, b));
    }
    if (!(tn <= tf)) continue;
    const int first = __ldg(&ob.first), count = __ldg(&ob.count);
    for (int i = first; i < first + count; i++) {
      const gi_triangle& tr = m.tris[i];
      const f3 p0 = ld3(tr.p[0]);
      const f3 e1 = sub3(ld3(tr.p[1]), p0), e2 = sub3(ld3(tr.p[2]), p0);
      const f3 pv = cross3(d, e2);
      const float det = dot3(e1, pv);  // -d . (e1 x e2): > 0 when the ray meets the front face
      if (m.cull ? !(det > 0.0f) : det == 0.0f) continue;
      const float inv = rcp_(det);
      const f3 tv = sub3(o, p0);
      const float u = dot3(tv, pv) * inv;
      if (u < 0.0f || u > 1.0f) continue;
      const f3 qv = cross3(tv, e1);
      const float v = dot3(d, qv) * inv;
      if (v < 0.0f || u + v > 1.0f) continue;
      const float t = dot3(e2, qv) * inv;
      if (t > 0.0f && t < h.t) {
        h.t = t;
        h.prim = -1;
        h.tri = i;
        h.obj = k;
        h.u = u;
        h.v = v;
      }
    }
  }
}

// A staged primitive: what its ray tests read that is the same for every ray of the
// camera.  Room, box: its corners minus the origin.  Sphere: origin - centre, and
// |origin - centre|^2 - r^2.  Two 16-byte reads.
struct __align__(16) PrimTest {
  float a[3];
  int kind;  // gi_prim_kind, | kFinite; -1: no kind that a ray meets
  float b[3];
  float pad;
};
constexpr int kFinite = 0x100;  // every value is finite

__device__ __forceinline__ bool finite(float v) { return v - v == 0.0f; }

__device__ __forceinline__ PrimTest prim_test(const gi_prim& p, f3 o) {
  PrimTest r;
  const float ov[3] = {o.x, o.y, o.z};
  r.kind = p.kind == GI_PRIM_ROOM || p.kind == GI_PRIM_BOX || p.kind == GI_PRIM_SPHERE ? p.kind : -1;
  if (p.kind == GI_PRIM_SPHERE) {
    const f3 oc = sub3(o, mk3(p.a[0], p.a[1], p.a[2]));
    r.a[0] = oc.x;
    r.a[1] = oc.y;
    r.a[2] = oc.z;
    r.b[0] = dot3(oc, oc) - p.b[0] * p.b[0];
    r.b[1] = r.b[2] = 0.0f;
  } else {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      r.a[k] = p.a[k] - ov[k];
      r.b[k] = p.b[k] - ov[k];
    }
  }
  bool all = true;
#pragma unroll
  for (int k = 0; k < 3; k++) all = all && finite(r.a[k]) && finite(r.b[k]);
  if (all) r.kind |= kFinite;
  r.pad = 0.0f;
  return r;
}

// Componentwise bounds of the warp's ray directions; NaN if a lane's is NaN.
struct RayBounds {
  float dlo[3], dhi[3];
  float ilo[3], ihi[3];  // bounds of their reciprocals
  bool open[3];          // an axis whose directions lie about zero: no bounds
  bool closed;           // no axis is open, no direction NaN
};

__device__ __forceinline__ float warp_min(float v) {
  float r;
  asm("redux.sync.min.NaN.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_max(float v) {
  float r;
  asm("redux.sync.max.NaN.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

__device__ __forceinline__ float min_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

template <int PIX> __device__ __forceinline__ RayBounds ray_bounds(const float (&d)[PIX][3]) {
  RayBounds r;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    float lo = d[0][k], hi = d[0][k];
#pragma unroll
    for (int q = 1; q < PIX; q++) {
      lo = min_nan(lo, d[q][k]);
      hi = max_nan(hi, d[q][k]);
    }
    r.dlo[k] = warp_min(lo);
    r.dhi[k] = warp_max(hi);
    r.open[k] = !(r.dlo[k] >= 1e-37f || r.dhi[k] <= -1e-37f);
    // The rounded reciprocal decreases with d on each side of zero.
    r.ilo[k] = rcp_(r.dhi[k]);
    r.ihi[k] = rcp_(r.dlo[k]);
  }
  r.closed = !(r.open[0] || r.open[1] || r.open[2]);
  return r;
}

// A lower bound of the distance at which the warp's rays can hit the primitive, +inf
// if none can.  Rounding is monotone, so the bounds of a ray test's intermediate
// values are the same operations on the bounds of its operands, without a margin.
__device__ __forceinline__ float nearest_entry(const PrimTest& p, const RayBounds& r) {
  if (p.kind == (GI_PRIM_BOX | kFinite)) {
    float tn = -kInf, tf = kInf;  // lower bound of the entry, upper bound of the exit
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const float a0 = p.a[k] * r.ilo[k], a1 = p.a[k] * r.ihi[k], b0 = p.b[k] * r.ilo[k], b1 = p.b[k] * r.ihi[k];
      tn = r.open[k] ? tn : fmaxf(tn, fminf(fminf(a0, a1), fminf(b0, b1)));
      tf = r.open[k] ? tf : fminf(tf, fmaxf(fmaxf(a0, a1), fmaxf(b0, b1)));
    }
    // An entry needs tn <= tf and tn > 0.
    return tn > tf || tf <= 0.0f ? kInf : tn;
  }
  if (p.kind == (GI_PRIM_SPHERE | kFinite)) {
    float lo[3], hi[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const float u = p.a[k] * r.dlo[k], v = p.a[k] * r.dhi[k];
      lo[k] = fminf(u, v);
      hi[k] = fmaxf(u, v);
    }
    const float blo = lo[0] + lo[1] + lo[2], bhi = hi[0] + hi[1] + hi[2];
    // A hit needs disc = b^2 - cc >= 0 and t = -b - sqrt(disc) > 0.
    const float disc = fmaxf(blo * blo, bhi * bhi) - p.b[0];
    return disc < 0.0f || -blo <= 0.0f ? kInf : fmaxf(-bhi - sqrtf(disc), -kInf);  // NaN: no bound
  }
  return -kInf;
}

// Slab distances of a staged room or box.  NUMBERS: no product is NaN, and the minimum
// and maximum are one instruction (they differ from GLSL's in the sign of a zero, which
// no hit has).
template <bool NUMBERS>
__device__ __forceinline__ void slabs(const PrimTest& p, const float (&iv)[3], float (&t1)[3], float (&t2)[3]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float a = p.a[k] * iv[k], b = p.b[k] * iv[k];
    t1[k] = NUMBERS ? fminf(a, b) : gmin(a, b);
    t2[k] = NUMBERS ? fmaxf(a, b) : gmax(a, b);
  }
}
__device__ __forceinline__ float room_exit(const float (&t2)[3], int& ax) {
  ax = 0;
  float tf = t2[0];
  if (t2[1] < tf) { ax = 1; tf = t2[1]; }
  if (t2[2] < tf) { ax = 2; tf = t2[2]; }
  return tf;
}
__device__ __forceinline__ float box_entry(const float (&t1)[3], int& ax) {
  ax = 0;
  float tn = t1[0];
  if (t1[1] > tn) { ax = 1; tn = t1[1]; }
  if (t1[2] > tn) { ax = 2; tn = t1[2]; }
  return tn;
}

// Distance of a ray's hit on a staged primitive; not > 0 if there is none.
template <bool NUMBERS>
__device__ __forceinline__ float prim_hit(const PrimTest& p, f3 d, const float (&iv)[3]) {
  const int kind = p.kind & ~kFinite;
  if (kind == GI_PRIM_SPHERE) {
    const float b = p.a[0] * d.x + p.a[1] * d.y + p.a[2] * d.z;
    const float disc = b * b - p.b[0];
    return disc >= 0.0f ? -b - sqrtf(disc) : -1.0f;
  }
  if (kind != GI_PRIM_ROOM && kind != GI_PRIM_BOX) return -1.0f;
  float t1[3], t2[3];
  int ax;
  slabs<NUMBERS>(p, iv, t1, t2);
  if (NUMBERS) {
    const float tf = fminf(fminf(t2[0], t2[1]), t2[2]);
    if (kind == GI_PRIM_ROOM) return tf;
    const float tn = fmaxf(fmaxf(t1[0], t1[1]), t1[2]);
    return tn <= tf ? tn : -1.0f;
  }
  if (kind == GI_PRIM_ROOM) return room_exit(t2, ax);
  const float tn = box_entry(t1, ax);
  return tn <= gmin(gmin(t2[0], t2[1]), t2[2]) ? tn : -1.0f;
}

// Nearest hit: room interior (exit face), box exterior (entry face), sphere
// (near root), ties kept by the earlier primitive.
//
// The cast was bound by its arithmetic, every ray testing every primitive.  Now each
// lane of a warp bounds one primitive's distance to the warp's 8 x 8 pixels of rays
// (32 primitives in the time of one test), and the rays test the primitives in order
// of that bound until it passes their farthest hit: the same nearest hit, bit for
// bit.  Measured with 64 boxes and 16 spheres: the G-buffer at 1920 x 1080 319 -> 53 us, a
// shadow map of 1024 x 1024 171 -> 20 us (in index order 87 and 35; one pixel a thread and
// one primitive a lane at a time 67 and 27).
template <bool MESH, int PIX>
__device__ __forceinline__ void cast_rays(const gi_prim* __restrict__ prims, int np, const MeshSet& mesh, f3 o,
                                          const f3 (&d)[PIX], Hit (&h)[PIX], PrimTest* s_prims) {
  float iv[PIX][3], dv[PIX][3];
#pragma unroll
  for (int q = 0; q < PIX; q++) {
    h[q].t = kInf;
    h[q].prim = -1;
    h[q].tri = -1;
    h[q].obj = -1;
    h[q].u = h[q].v = 0.0f;
    dv[q][0] = d[q].x;
    dv[q][1] = d[q].y;
    dv[q][2] = d[q].z;
#pragma unroll
    for (int k = 0; k < 3; k++) iv[q][k] = rcp_(dv[q][k]);
  }
  const RayBounds bounds = ray_bounds<PIX>(dv);
  const int lane = threadIdx.x & 31;
  float farthest = kInf;  // of the warp's hits so far
  for (int base = 0; base < np; base += kPrimStage) {
    const int cnt = min(kPrimStage, np - base);
    __syncthreads();
    for (int i = threadIdx.x; i < cnt; i += Cast<MESH>::kThreads) s_prims[i] = prim_test(prims[base + i], o);
    __syncthreads();
    for (int first = 0; first < cnt; first += 32 * kOwnPrims) {
      // Each lane's primitives, 32 apart; the nearest of them and its place.
      float entry[kOwnPrims];
#pragma unroll
      for (int k = 0; k < kOwnPrims; k++) {
        const int own = first + 32 * k + lane;
        entry[k] = own < cnt ? nearest_entry(s_prims[own], bounds) : kInf;
      }
      for (;;) {
        float mine = entry[0];
        int place = 0;
#pragma unroll
        for (int k = 1; k < kOwnPrims; k++) {
          place = entry[k] < mine ? k : place;
          mine = fminf(mine, entry[k]);
        }
        const float next = warp_min(mine);
        if (next == kInf || next > farthest) break;
        const int from = __ffs((int)__ballot_sync(0xffffffffu, mine == next)) - 1;
        const int at = first + 32 * __shfl_sync(0xffffffffu, place, from) + from;
#pragma unroll
        for (int k = 0; k < kOwnPrims; k++)
          if (first + 32 * k + lane == at) entry[k] = kInf;
        const PrimTest p = s_prims[at];
        const int prim = base + at;
        const bool numbers = bounds.closed && (p.kind & kFinite);
        float far = 0.0f;
#pragma unroll
        for (int q = 0; q < PIX; q++) {
          const float t = numbers ? prim_hit<true>(p, d[q], iv[q]) : prim_hit<false>(p, d[q], iv[q]);
          if (t > 0.0f && (t < h[q].t || (t == h[q].t && prim < h[q].prim))) {
            h[q].t = t;
            h[q].prim = prim;
          }
          far = fmaxf(far, h[q].t);
        }
        farthest = warp_max(far);
      }
    }
  }
  if (MESH)
    for (int q = 0; q < PIX; q++) cast_mesh(mesh, o, d[q], iv[q], h[q]);
}

// The surface normal at the hit of an analytic primitive.
__device__ __forceinline__ f3 prim_normal(const gi_prim& g, f3 o, f3 d, float t) {
  if (g.kind == GI_PRIM_SPHERE) return normalize3(sub3(add3(o, mul3s(d, t)), mk3(g.a[0], g.a[1], g.a[2])));
  const PrimTest p = prim_test(g, o);
  const float iv[3] = {rcp_(d.x), rcp_(d.y), rcp_(d.z)}, dv[3] = {d.x, d.y, d.z};
  float t1[3], t2[3];
  slabs<false>(p, iv, t1, t2);
  int ax;
  if (g.kind == GI_PRIM_ROOM) room_exit(t2, ax);
  else box_entry(t1, ax);
  float nv[3];
#pragma unroll
  for (int k = 0; k < 3; k++) nv[k] = k == ax ? (dv[k] > 0.0f ? -1.0f : 1.0f) : 0.0f;
  return mk3(nv[0], nv[1], nv[2]);
}

// A thread's pixels and rays.  Pixels past the image take its last row or column (they
// join the warp's votes) and store nothing.
template <int PIX> struct CastPixels {
  int x, y[PIX];
  bool live[PIX];
  f3 org, dir[PIX];
};
template <bool MESH, int PIX> __device__ __forceinline__ CastPixels<PIX> cast_pixels(const ViewArgs& v) {
  CastPixels<PIX> c;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int x = blockIdx.x * Cast<MESH>::kX + (w & 3) * 8 + (l & 7);
  c.x = min(x, v.width - 1);
  const float sx = div_((float)c.x + 0.5f, (float)v.width);
  const float4 o4 = mat_vec(v.inv_view, 0.0f, 0.0f, 0.0f, 1.0f);
  c.org = mk3(o4.x, o4.y, o4.z);
#pragma unroll
  for (int q = 0; q < PIX; q++) {
    const int y = blockIdx.y * Cast<MESH>::kY + ((w >> 2) * PIX + q) * 4 + (l >> 3);
    c.live[q] = x < v.width && y < v.height;
    c.y[q] = min(y, v.height - 1);
    const float sy = div_((float)c.y[q] + 0.5f, (float)v.height);
    c.dir[q] = normalize3(sub3(unproject(v.inv_view_proj, sx, sy, 1.0f), c.org));
  }
  return c;
}

// gBufferBuilder.frag:28-38 at the primary hit.  The eight powers of a surface's
// colours are the same for every pixel that shows it: a warp evaluates them once for
// each of the surfaces it hits, four surfaces at a time, a lane per channel.
__device__ __forceinline__ void shade(const ViewArgs& v, const gi_prim* __restrict__ prims, int np, const MeshSet& mesh,
                                      int x, int y, bool live, f3 org, f3 dir, const Hit& h, float (&colour)[32][8],
                                      float* __restrict__ albedo, float* __restrict__ emissive,
                                      float* __restrict__ normal, float* __restrict__ moments,
                                      float* __restrict__ ndc) {
  const int lane = threadIdx.x & 31;
  const int surface = h.prim >= 0 ? h.prim : (h.tri >= 0 ? np + h.obj : -1);
  int slot = 0;
  {
    __syncwarp();  // the last pixel's colours have been read
    unsigned todo = __ballot_sync(0xffffffffu, surface >= 0);
    for (int n = 0; todo; n += 4) {  // four surfaces a round: lanes 8 k .. 8 k + 7 take the k-th
      int mine = -1;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if (!todo) break;
        const int id = __shfl_sync(0xffffffffu, surface, __ffs((int)todo) - 1);
        todo &= ~__ballot_sync(0xffffffffu, surface == id);
        if (surface == id) slot = n + k;
        if ((lane >> 3) == k) mine = id;
      }
      if (mine >= 0) {
        const int ch = lane & 3;
        const float* al = mine < np ? prims[mine].albedo : mesh.objects[mine - np].albedo;
        const float* em = mine < np ? prims[mine].emissive : mesh.objects[mine - np].emissive;
        colour[n + (lane >> 3)][lane & 7] = powf_((lane & 4) ? em[ch] : al[ch], 2.2f);
      }
    }
    __syncwarp();
  }
  if (!live) return;
  const size_t i = (size_t)y * v.width + x;
  if (surface < 0) {
    reinterpret_cast<float4*>(albedo)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    reinterpret_cast<float4*>(emissive)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    reinterpret_cast<float4*>(normal)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    reinterpret_cast<float2*>(moments)[i] = make_float2(0.0f, 0.0f);
    ndc[i] = 1.0f;
    return;
  }
  const f3 hit = add3(org, mul3s(dir, h.t));
  const f3 dl = sub3(hit, org);
  const float delta_len = sqrtf(dot3(dl, dl));
  f3 n;
  if (h.prim >= 0) {
    n = prim_normal(prims[h.prim], org, dir, h.t);
  } else {
    // Barycentric blend of the vertex normals, (1 - u - v) n0 + u n1 + v n2.
    const gi_triangle& tr = mesh.tris[h.tri];
    const float w0 = 1.0f - h.u - h.v;
    const f3 n0 = ld3(tr.n[0]), n1 = ld3(tr.n[1]), n2 = ld3(tr.n[2]);
    n = add3(add3(mul3s(n0, w0), mul3s(n1, h.u)), mul3s(n2, h.v));
  }
  reinterpret_cast<float4*>(albedo)[i] = *reinterpret_cast<const float4*>(&colour[slot][0]);
  reinterpret_cast<float4*>(emissive)[i] = *reinterpret_cast<const float4*>(&colour[slot][4]);
  reinterpret_cast<float4*>(normal)[i] = make_float4(n.x, n.y, n.z, 1.0f);
  reinterpret_cast<float2*>(moments)[i] = make_float2(delta_len, delta_len * delta_len);
  ndc[i] = project(v.view_proj, hit).z;
}

template <bool MESH>
__global__ void __launch_bounds__(Cast<MESH>::kThreads) gbuffer_kernel(const __grid_constant__ ViewArgs v,
                                                               const gi_prim* __restrict__ prims, int np, MeshSet mesh,
                                                               float* __restrict__ albedo,
                                                               float* __restrict__ emissive,
                                                               float* __restrict__ normal,
                                                               float* __restrict__ moments, float* __restrict__ ndc) {
  __shared__ PrimTest s_prims[kPrimStage];
  __shared__ __align__(16) float s_colour[Cast<MESH>::kThreads / 32][32][8];  // a warp's surfaces: albedo, emissive
  constexpr int PIX = Cast<MESH>::kPixels;
  const CastPixels<PIX> c = cast_pixels<MESH, PIX>(v);
  Hit h[PIX];
  cast_rays<MESH, PIX>(prims, np, mesh, c.org, c.dir, h, s_prims);
#pragma unroll
  for (int q = 0; q < PIX; q++)
    shade(v, prims, np, mesh, c.x, c.y[q], c.live[q], c.org, c.dir[q], h[q], s_colour[threadIdx.x >> 5], albedo, emissive,
          normal, moments, ndc);
}

template <bool MESH>
__global__ void __launch_bounds__(Cast<MESH>::kThreads) shadow_kernel(const __grid_constant__ ViewArgs v,
                                                              const gi_prim* __restrict__ prims, int np, MeshSet mesh,
                                                              float* __restrict__ out) {
  __shared__ PrimTest s_prims[kPrimStage];
  constexpr int PIX = Cast<MESH>::kPixels;
  const CastPixels<PIX> c = cast_pixels<MESH, PIX>(v);
  Hit h[PIX];
  cast_rays<MESH, PIX>(prims, np, mesh, c.org, c.dir, h, s_prims);
#pragma unroll
  for (int q = 0; q < PIX; q++) {
    if (!c.live[q]) continue;
    float z = 1.0f;
    if (h[q].prim >= 0 || h[q].tri >= 0) z = project(v.view_proj, add3(c.org, mul3s(c.dir[q], h[q].t))).z;
    out[(size_t)c.y[q] * v.width + c.x] = z;
  }
}

// directLighting.frag:45-79.
__global__ void __launch_bounds__(kTx* kTy) direct_kernel(const __grid_constant__ ViewArgs v,
                                                          const __grid_constant__ ViewArgs lv,
                                                          const float* __restrict__ albedo,
                                                          const float* __restrict__ emissive,
                                                          const float* __restrict__ normal,
                                                          const float* __restrict__ ndc,
                                                          const float* __restrict__ shadow, int ssize,
                                                          float* __restrict__ out) {
  const int x = blockIdx.x * kTx + threadIdx.x, y = blockIdx.y * kTy + threadIdx.y;
  if (x >= v.width || y >= v.height) return;
  const int W = v.width, H = v.height;
  const float fx = div_((float)x + 0.5f, (float)W), fy = div_((float)y + 0.5f, (float)H);
  const float depth = sample1(ndc, W, H, fx, fy);
  const float4 n4 = sample4(normal, W, H, fx, fy);
  const f3 wn = mk3(n4.x, n4.y, n4.z);
  const float4 lp4 = mat_vec(lv.inv_view, 0.0f, 0.0f, 0.0f, 1.0f);
  const f3 light_pos = mk3(lp4.x, lp4.y, lp4.z);
  const f3 wp = unproject(v.inv_view_proj, fx, fy, depth);
  const f3 lvec = sub3(wp, light_pos);
  const float diffuse = gmax(0.0f, -dot3(normalize3(lvec), wn));
  f3 sc = project(lv.view_proj, wp);
  const float4 lvp = mat_vec(lv.view, wp.x, wp.y, wp.z, 1.0f);
  f3 li = mk3(5.0f, 5.0f, 5.0f);
  const float rx = sc.x - 0.5f, ry = sc.y - 0.5f;
  const float radius = sqrtf(rx * rx + ry * ry) * 2.0f;
  float t = div_(1.0f - saturate(div_(radius - 0.6f, 1.0f - 0.6f)) - 0.0f, 1.0f - 0.0f);
  t = gmin(gmax(t, 0.0f), 1.0f);
  const float penumbra = t * t * (3.0f - 2.0f * t) * (lvp.z > 0.0f ? 1.0f : 0.0f);
  li = mul3s(li, penumbra);
  const float bias = 2e-4f;
  sc.z = sc.z - bias;
  // sampler2DShadow, linear, compare LESS_OR_EQUAL.
  float pcf;
  {
    const Bilin B = bilin(sc.x, sc.y, ssize, ssize);
    const float r = sc.z;
    const float p00 = r <= __ldg(shadow + B.o00) ? 1.0f : 0.0f;
    const float p10 = r <= __ldg(shadow + B.o10) ? 1.0f : 0.0f;
    const float p01 = r <= __ldg(shadow + B.o01) ? 1.0f : 0.0f;
    const float p11 = r <= __ldg(shadow + B.o11) ? 1.0f : 0.0f;
    pcf = blend1(B, p00, p10, p01, p11);
  }
  li = mul3s(li, powf_(pcf, 2.2f));
  const float4 al = sample4(albedo, W, H, fx, fy);
  const float4 em = sample4(emissive, W, H, fx, fy);
  float4 o;
  o.x = diffuse * al.x * li.x + em.x;
  o.y = diffuse * al.y * li.y + em.y;
  o.z = diffuse * al.z * li.z + em.z;
  o.w = 1.0f;
  reinterpret_cast<float4*>(out)[(size_t)y * W + x] = o;
}

dim3 grid2d(int w, int h) { return dim3((w + kTx - 1) / kTx, (h + kTy - 1) / kTy); }
// go(mesh, grid, threads) with the launch of a cast with or without meshes.
template <typename Go> void launch_cast(int w, int h, const MeshSet& mesh, Go go) {
  auto with = [&](auto m) {
    using C = Cast<decltype(m)::value>;
    go(m, dim3((w + C::kX - 1) / C::kX, (h + C::kY - 1) / C::kY), C::kThreads);
  };
  if (mesh.num_objects > 0) with(std::true_type{});
  else with(std::false_type{});
}

int launch_gbuffer(const gi_view& view, const gi_prim* prims, int np, const MeshSet& mesh, float* albedo,
                   float* emissive, float* normal, float* moments, float* ndc, cudaStream_t stream) {
  const ViewArgs v = view_args(view);
  launch_cast(v.width, v.height, mesh, [&](auto m, dim3 grid, int threads) {
    gbuffer_kernel<decltype(m)::value><<<grid, threads, 0, stream>>>(v, prims, np, mesh, albedo, emissive, normal,
                                                                     moments, ndc);
  });
  GI_CHECK_LAUNCH("gbuffer_kernel");
  count_launches(1);
  return GI_OK;
}

int launch_shadow(const gi_view& view, const gi_prim* prims, int np, const MeshSet& mesh, float* out,
                  cudaStream_t stream) {
  const ViewArgs v = view_args(view);
  launch_cast(v.width, v.height, mesh, [&](auto m, dim3 grid, int threads) {
    shadow_kernel<decltype(m)::value><<<grid, threads, 0, stream>>>(v, prims, np, mesh, out);
  });
  GI_CHECK_LAUNCH("shadow_kernel");
  count_launches(1);
  return GI_OK;
}

}  // namespace
}  // namespace gi

using namespace gi;

extern "C" int gi_gbuffer(const gi_view* view, const gi_prim* prims, int num_prims, float* albedo, float* emissive,
                          float* normal, float* depth_moments, float* ndc_depth, void* stream) {
  GI_CHECK_ARG(view && prims && albedo && emissive && normal && depth_moments && ndc_depth, "gi_gbuffer: null");
  GI_CHECK_ARG(num_prims >= 1 && num_prims <= GI_MAX_PRIMS, "gi_gbuffer: bad primitive count");
  GI_CHECK_ARG(view->width >= 1 && view->height >= 1, "gi_gbuffer: bad viewport");
  GI_CHECK_ARG(aligned16(albedo) && aligned16(emissive) && aligned16(normal) && aligned16(depth_moments),
               "gi_gbuffer: unaligned buffer");
  return launch_gbuffer(*view, prims, num_prims, MeshSet{nullptr, nullptr, 0, 0}, albedo, emissive, normal,
                        depth_moments, ndc_depth, (cudaStream_t)stream);
}

static int check_mesh(const gi_prim* prims, int num_prims, const gi_mesh_object* objects, int num_objects,
                      const gi_triangle* tris, int num_tris, const char* who) {
  GI_CHECK_ARG(num_prims >= 0 && num_prims <= GI_MAX_PRIMS && (num_prims == 0 || prims), who);
  GI_CHECK_ARG(num_objects >= 0 && num_objects <= GI_MAX_MESH_OBJECTS && (num_objects == 0 || (objects && tris)),
               who);
  GI_CHECK_ARG(num_tris >= 0 && num_tris <= GI_MAX_TRIANGLES, who);
  GI_CHECK_ARG(num_prims + num_objects >= 1, who);
  return GI_OK;
}

extern "C" int gi_gbuffer_mesh(const gi_view* view, const gi_prim* prims, int num_prims,
                               const gi_mesh_object* objects, int num_objects, const gi_triangle* tris, int num_tris,
                               int cull, float* albedo, float* emissive, float* normal, float* depth_moments, float* ndc_depth,
                               void* stream) {
  GI_CHECK_ARG(view && albedo && emissive && normal && depth_moments && ndc_depth, "gi_gbuffer_mesh: null");
  int st = check_mesh(prims, num_prims, objects, num_objects, tris, num_tris, "gi_gbuffer_mesh: bad scene arrays");
  if (st) return st;
  GI_CHECK_ARG(cull == GI_CULL_NONE || cull == GI_CULL_BACK, "gi_gbuffer_mesh: unknown cull mode");
  GI_CHECK_ARG(view->width >= 1 && view->height >= 1, "gi_gbuffer_mesh: bad viewport");
  GI_CHECK_ARG(aligned16(albedo) && aligned16(emissive) && aligned16(normal) && aligned16(depth_moments),
               "gi_gbuffer_mesh: unaligned buffer");
  return launch_gbuffer(*view, prims, num_prims, MeshSet{objects, tris, num_objects, cull}, albedo, emissive, normal,
                        depth_moments, ndc_depth, (cudaStream_t)stream);
}

extern "C" int gi_shadow_map_mesh(const gi_view* light_view, const gi_prim* prims, int num_prims,
                                  const gi_mesh_object* objects, int num_objects, const gi_triangle* tris,
                                  int num_tris, int cull, float* shadow, void* stream) {
  GI_CHECK_ARG(light_view && shadow, "gi_shadow_map_mesh: null");
  int st = check_mesh(prims, num_prims, objects, num_objects, tris, num_tris, "gi_shadow_map_mesh: bad scene arrays");
  if (st) return st;
  GI_CHECK_ARG(cull == GI_CULL_NONE || cull == GI_CULL_BACK, "gi_shadow_map_mesh: unknown cull mode");
  return launch_shadow(*light_view, prims, num_prims, MeshSet{objects, tris, num_objects, cull}, shadow,
                       (cudaStream_t)stream);
}

extern "C" int gi_shadow_map(const gi_view* light_view, const gi_prim* prims, int num_prims, float* shadow,
                             void* stream) {
  GI_CHECK_ARG(light_view && prims && shadow, "gi_shadow_map: null");
  GI_CHECK_ARG(num_prims >= 1 && num_prims <= GI_MAX_PRIMS, "gi_shadow_map: bad primitive count");
  return launch_shadow(*light_view, prims, num_prims, MeshSet{nullptr, nullptr, 0, 0}, shadow, (cudaStream_t)stream);
}

extern "C" int gi_direct_light(const gi_view* view, const gi_view* light_view, const float* albedo,
                               const float* emissive, const float* normal, const float* ndc_depth, const float* shadow,
                               int shadow_size, float* out, void* stream) {
  GI_CHECK_ARG(view && light_view && albedo && emissive && normal && ndc_depth && shadow && out,
               "gi_direct_light: null");
  GI_CHECK_ARG(shadow_size >= 1, "gi_direct_light: bad shadow size");
  GI_CHECK_ARG(aligned16(albedo) && aligned16(emissive) && aligned16(normal) && aligned16(out),
               "gi_direct_light: unaligned buffer");
  ViewArgs v = view_args(*view), lv = view_args(*light_view);
  direct_kernel<<<grid2d(v.width, v.height), dim3(kTx, kTy), 0, (cudaStream_t)stream>>>(
      v, lv, albedo, emissive, normal, ndc_depth, shadow, shadow_size, out);
  GI_CHECK_LAUNCH("direct_kernel");
  count_launches(1);
  return GI_OK;
}
