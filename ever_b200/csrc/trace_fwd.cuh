// Forward trace kernels (included by trace_fwd_k{8,16,32}.cu, one k-buffer size per
// translation unit so the instantiations compile in parallel).
//
// Each ray's entry/exit events are integrated in order of t (update() with SH colour
// evaluated along the ray). Three traversals find them, with the same results:
//  - frustum phase (traversal 0, the default): the warp lists the leaves that its packet of
//    up to 32 rays can meet, and each lane takes its events from that list (below);
//  - gather rounds of packets (2, and what the frustum phase leaves): each ray's next KBUF
//    events go into a sorted register buffer and are then integrated, round after round. The
//    rays of a warp walk ONE node sequence together: each lane tests its own ray against
//    the node's two child boxes, __ballot_sync decides where the warp goes, and a per-warp
//    stack lives in shared memory. Node fetches are warp-uniform (one broadcast load);
//  - gather rounds per ray (1): each thread walks the tree alone (stack in shared memory).
//
// Reference: raygen loop splinetracers/fast_ellipsoid_splinetracer/slang/shaders.slang:171-235,
// intersection program :84-107 and any-hit k-buffer :117-164. Our rounds gather
// events strictly after the last gathered one in the total order (t, Morton position,
// entry-before-exit), so no round boundary of ours drops an event; the reference's own
// 16-event round boundaries are replayed while consuming (s16 below): an event tied with
// the 16th event of a reference round is dropped, and an exit beyond tmax counts only
// inside the reference round that consumed its entry. The result is the reference's
// event sequence for any KBUF.
#pragma once
#include <climits>

#include "camera.cuh"
#include "common.cuh"
#include "internal.cuh"

namespace ever {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kMaxMembers = 16;

template <int KBUF>
__device__ __forceinline__ void buf_insert(uint64_t (&buf)[KBUF], uint64_t k) {
#pragma unroll
  for (int i = 0; i < KBUF; ++i) {
    const uint64_t b = buf[i];
    const bool lt = k < b;
    buf[i] = lt ? k : b;
    k = lt ? b : k;
  }
}

// The same among the first M entries; returns the key that falls out behind them.
template <int M, int KBUF>
__device__ __forceinline__ uint64_t buf_insert_low(uint64_t (&buf)[KBUF], uint64_t k) {
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const uint64_t b = buf[i];
    const bool lt = k < b;
    buf[i] = lt ? k : b;
    k = lt ? b : k;
  }
  return k;
}

__device__ __forceinline__ Node load_node(const Node* __restrict__ nodes, int n) {
  const float4* p = reinterpret_cast<const float4*>(nodes + n);
  Node nd;
  nd.a = __ldg(p + 0);
  nd.b = __ldg(p + 1);
  nd.c = __ldg(p + 2);
  nd.d = __ldg(p + 3);
  return nd;
}

struct RaySlab {
  float3 invd, ood;
};

__device__ __forceinline__ RaySlab make_slab(const Ray& r) {
  auto inv = [](float d) { return 1.f / (fabsf(d) > 1e-20f ? d : copysignf(1e-20f, d)); };
  RaySlab s;
  s.invd = make_float3(inv(r.d.x), inv(r.d.y), inv(r.d.z));
  s.ood = make_float3(r.o.x * s.invd.x, r.o.y * s.invd.y, r.o.z * s.invd.z);
  return s;
}

// Slab test of [lo, hi] against [tlo, thi]; returns the entry distance or +inf on a miss.
__device__ __forceinline__ float slab(const RaySlab& s, float lx, float ly, float lz, float hx, float hy, float hz,
                                      float tlo, float thi) {
  const float ax = fmaf(lx, s.invd.x, -s.ood.x), bx = fmaf(hx, s.invd.x, -s.ood.x);
  const float ay = fmaf(ly, s.invd.y, -s.ood.y), by = fmaf(hy, s.invd.y, -s.ood.y);
  const float az = fmaf(lz, s.invd.z, -s.ood.z), bz = fmaf(hz, s.invd.z, -s.ood.z);
  const float tn = fmaxf(fmaxf(fminf(ax, bx), fminf(ay, by)), fmaxf(fminf(az, bz), tlo));
  const float tf = fminf(fminf(fmaxf(ax, bx), fmaxf(ay, by)), fminf(fmaxf(az, bz), thi));
  return tn <= tf ? tn : INFINITY;
}

__device__ __forceinline__ bool box_contains(float lx, float ly, float lz, float hx, float hy, float hz, float3 p) {
  return p.x >= lx && p.x <= hx && p.y >= ly && p.y <= hy && p.z >= lz && p.z <= hz;
}

// One leaf: the ellipsoid's entry/exit events that are candidates of this round
// (see the file comment) go into the sorted buffer.
template <int KBUF>
__device__ __forceinline__ void leaf_insert(const Record* __restrict__ recs, int j, const Ray& ray, uint64_t lower,
                                            float s16, float tmax, uint64_t (&buf)[KBUF]) {
  const Record R = load_record(recs, j);
  HitT H;
  if (!intersect(R, ray, H)) return;
  if (H.t0 > s16 && H.t0 <= tmax) {
    const uint64_t e = event_key(H.t0, j, 0);
    if (e > lower && e < buf[KBUF - 1]) buf_insert(buf, e);
  }
  if (H.t1 > s16 && (H.t1 <= tmax || (H.t0 > s16 && H.t0 <= tmax))) {
    const uint64_t e = event_key(H.t1, j, 1);
    if (e > lower && e < buf[KBUF - 1]) buf_insert(buf, e);
  }
}

// ---- per-ray traversal ----
template <int KBUF>
__device__ void gather_ray(const Node* __restrict__ nodes, const Record* __restrict__ recs, const Ray& ray,
                           const RaySlab& sl, uint64_t lower, float s16, float tmax, uint64_t (&buf)[KBUF],
                           int* st_node, float* st_t, int stride, int depth, uint32_t& status) {
  const float cap = fminf(tmax, kSentinel);
  // The last event may be an exit beyond tmax; others like it are still to be found at tmax.
  const float lo_t = fminf(fmaxf(lower ? key_t(lower) : 0.f, s16), cap);
  int sp = 0;
  int node = 0;
  for (;;) {
    const Node nd = load_node(nodes, node);
    const float hi = fminf(cap, key_t(buf[KBUF - 1]));  // an empty slot is NaN: fminf keeps cap
    const float tc[2] = {slab(sl, nd.a.x, nd.a.y, nd.a.z, nd.a.w, nd.b.x, nd.b.y, lo_t, hi),
                         slab(sl, nd.c.x, nd.c.y, nd.c.z, nd.c.w, nd.d.x, nd.d.y, lo_t, hi)};
    const int c[2] = {child_link(nd.b), child_link(nd.d)};
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (tc[k] != INFINITY && c[k] < 0) leaf_insert(recs, ~c[k], ray, lower, s16, tmax, buf);
    const bool i0 = tc[0] != INFINITY && c[0] >= 0;
    const bool i1 = tc[1] != INFINITY && c[1] >= 0;
    if (i0 && i1) {
      const bool first0 = tc[0] <= tc[1];
      if (sp < depth) {
        st_node[sp * stride] = first0 ? c[1] : c[0];
        st_t[sp * stride] = first0 ? tc[1] : tc[0];
        ++sp;
      } else {
        status |= EVER_STATUS_STACK_OVERFLOW;
      }
      node = first0 ? c[0] : c[1];
      continue;
    }
    if (i0 || i1) {
      node = i0 ? c[0] : c[1];
      continue;
    }
    bool found = false;
    while (sp > 0) {
      --sp;
      if (st_t[sp * stride] <= fminf(cap, key_t(buf[KBUF - 1]))) {
        node = st_node[sp * stride];
        found = true;
        break;
      }
    }
    if (!found) break;
  }
}

// ---- packet traversal: the warp walks one node sequence ----
template <int KBUF>
__device__ void gather_packet(const Node* __restrict__ nodes, const Record* __restrict__ recs, const Ray& ray,
                              const RaySlab& sl, bool act, uint64_t lower, float s16, float tmax,
                              uint64_t (&buf)[KBUF], int* wstack, int lane, int depth, uint32_t& status) {
  const float cap = fminf(tmax, kSentinel);
  const float lo_t = fminf(fmaxf(lower ? key_t(lower) : 0.f, s16), cap);  // as in gather_ray
  int sp = 0;
  int node = 0;
  for (;;) {
    const Node nd = load_node(nodes, node);
    float t0 = INFINITY, t1 = INFINITY;
    if (act) {
      const float hi = fminf(cap, key_t(buf[KBUF - 1]));
      t0 = slab(sl, nd.a.x, nd.a.y, nd.a.z, nd.a.w, nd.b.x, nd.b.y, lo_t, hi);
      t1 = slab(sl, nd.c.x, nd.c.y, nd.c.z, nd.c.w, nd.d.x, nd.d.y, lo_t, hi);
    }
    const unsigned m0 = __ballot_sync(kFull, t0 != INFINITY);
    const unsigned m1 = __ballot_sync(kFull, t1 != INFINITY);
    const int c0 = child_link(nd.b), c1 = child_link(nd.d);
    if (c0 < 0 && t0 != INFINITY) leaf_insert(recs, ~c0, ray, lower, s16, tmax, buf);
    if (c1 < 0 && t1 != INFINITY) leaf_insert(recs, ~c1, ray, lower, s16, tmax, buf);
    const bool g0 = c0 >= 0 && m0 != 0u, g1 = c1 >= 0 && m1 != 0u;
    if (g0 && g1) {
      // nearer child first, by majority of the lanes that hit either
      const unsigned pref0 = __ballot_sync(kFull, t0 <= t1 && t0 != INFINITY);
      const bool first0 = 2 * __popc(pref0) >= __popc(m0 | m1);
      if (sp < depth) {
        if (lane == 0) {
          const int far = first0 ? c1 : c0;
          wstack[sp] = far;
          asm volatile("prefetch.global.L1 [%0];" ::"l"(nodes + far));
        }
        ++sp;
      } else {
        status |= EVER_STATUS_STACK_OVERFLOW;
      }
      __syncwarp();
      node = first0 ? c0 : c1;
    } else if (g0 || g1) {
      node = g0 ? c0 : c1;
    } else {
      if (sp == 0) break;
      --sp;
      node = wstack[sp];
    }
  }
}

__device__ __forceinline__ void member_insert(int p, int j, int& n_mem, int (&mem_p)[kMaxMembers],
                                              int (&mem_j)[kMaxMembers]) {
  int jj = j;
  for (int q = 0; q < n_mem; ++q) {
    if (p < mem_p[q]) {
      const int tp = mem_p[q], tj = mem_j[q];
      mem_p[q] = p;
      mem_j[q] = jj;
      p = tp;
      jj = tj;
    }
  }
  mem_p[n_mem] = p;
  mem_j[n_mem] = jj;
  ++n_mem;
}

// Ellipsoid j contains the ray start (t0 <= 0 < t1): record it (sorted by original index);
// beyond kMaxMembers the rest are summed into `extra` in traversal order (status flag).
template <int DEG>
__device__ __forceinline__ void point_leaf(const Record* __restrict__ recs, const int32_t* __restrict__ order,
                                           const float* __restrict__ feats, int fst, const float* B, int bs,
                                           const Ray& ray, int j, int& n_mem, int (&mem_p)[kMaxMembers],
                                           int (&mem_j)[kMaxMembers], float4& extra, uint32_t& status) {
  const Record R = load_record(recs, j);
  HitT H;
  if (!(intersect(R, ray, H) && H.t0 <= 0.f && H.t1 > 0.f)) return;
  if (n_mem < kMaxMembers) {
    member_insert(__ldg(order + j), j, n_mem, mem_p, mem_j);
  } else {
    status |= EVER_STATUS_INIT_OVERFLOW;
    const float sg = R.r3.x;
    const float3 c = DEG == 0 ? dc_colour(R.r3) : sh_colour<DEG>(feats + int64_t(j) * fst, B, bs);
    extra.x = extra.x + sg;
    extra.y = extra.y + sg * c.x;
    extra.z = extra.z + sg * c.y;
    extra.w = extra.w + sg * c.z;
  }
}

// Point query for the ray start; PACKET: warp-uniform walk.
template <int DEG, bool PACKET>
__device__ int point_members(const Node* __restrict__ nodes, const Record* __restrict__ recs,
                             const int32_t* __restrict__ order, const float* __restrict__ feats, int fst,
                             const float* B, int bs, const Ray& ray, bool act,
                             int* stack, int stride, int depth, int lane, int (&mem_p)[kMaxMembers],
                             int (&mem_j)[kMaxMembers], float4& extra, uint32_t& status) {
  int n_mem = 0;
  int sp = 0;
  int node = 0;
  for (;;) {
    const Node nd = load_node(nodes, node);
    const bool h0 = act && box_contains(nd.a.x, nd.a.y, nd.a.z, nd.a.w, nd.b.x, nd.b.y, ray.o);
    const bool h1 = act && box_contains(nd.c.x, nd.c.y, nd.c.z, nd.c.w, nd.d.x, nd.d.y, ray.o);
    const int c0 = child_link(nd.b), c1 = child_link(nd.d);
    if (h0 && c0 < 0) point_leaf<DEG>(recs, order, feats, fst, B, bs, ray, ~c0, n_mem, mem_p, mem_j, extra, status);
    if (h1 && c1 < 0) point_leaf<DEG>(recs, order, feats, fst, B, bs, ray, ~c1, n_mem, mem_p, mem_j, extra, status);
    bool g0 = h0 && c0 >= 0, g1 = h1 && c1 >= 0;
    if (PACKET) {
      g0 = __any_sync(kFull, g0);
      g1 = __any_sync(kFull, g1);
    }
    if (g0 && g1) {
      if (sp < depth) {
        if (!PACKET || lane == 0) stack[sp * stride] = c1;
        ++sp;
      } else {
        status |= EVER_STATUS_STACK_OVERFLOW;
      }
      if (PACKET) __syncwarp();
      node = c0;
    } else if (g0 || g1) {
      node = g0 ? c0 : c1;
    } else {
      if (sp == 0) break;
      --sp;
      node = stack[sp * stride];
    }
  }
  return n_mem;
}

// Which scene a packet traces, and the per-launch constants.
struct SceneRef {
  const Node* nodes;
  const Record* recs;
  const float* features;
  const int32_t* order;  // Morton position -> original index
  int64_t N;
  int K;
};

struct TraceCtx {
  float tmin, tmax;
  int max_iters;
  EverForwardOut out;
  int depth;           // traversal stack entries in use (<= kStackDepth)
  const float* depth_hint;  // (R) nullable: per-ray guess of the stopping t
  LeftRays left;       // rays that the frustum phase leaves, for the rounds' own kernel
};

// One event of a ray's sorted sequence, integrated under the reference's round rules
// (shaders.slang:197-227): an event tied with the 16th event of a reference round is
// dropped, an exit beyond tmax counts only inside the round that consumed its entry, a
// t > 1e9 sentinel ends the ray. Returns true once the ray is finished.
template <int DEG>
__device__ __forceinline__ bool consume_event(const SceneRef& sc, const TraceCtx& C, const Ray& ray, const float* B,
                                              int bs, int64_t slot, uint64_t k, State& s, float4& last_dirac,
                                              int& iters, float& s16, int& cnt16, uint32_t& status) {
  const float t = key_t(k);
  const int j = key_pos(k);
  const int ex = key_exit(k);
  if (!(t > s16)) return false;  // tied with the 16th event of a reference round: dropped
  if (t > kSentinel) return true;
  const float4 r3 = __ldg(&sc.recs[j].r3);
  if (ex && t > C.tmax) {
    HitT H;
    intersect(load_record(sc.recs, j), ray, H);
    if (!(H.t0 > s16 && H.t0 <= C.tmax)) return false;
  }
  const float3 c = DEG == 0 ? dc_colour(r3) : sh_colour<DEG>(sc.features + int64_t(j) * feat_stride(sc.K), B, bs);
  const float dh = ex ? -r3.x : r3.x;
  const float4 dirac = make_float4(dh, dh * c.x, dh * c.y, dh * c.z);
  update(s, t, dirac);
  last_dirac = dirac;
  if (C.out.event_log) {
    if (iters < C.out.log_cap)
      C.out.event_log[slot * int64_t(C.out.log_cap) + iters] = 2 * j + (ex ? 0 : 1);
    else
      status |= EVER_STATUS_LOG_OVERFLOW;
  }
  if (C.out.touch_count) atomicAdd(C.out.touch_count + __ldg(sc.order + j), 1);
  ++iters;
  if (++cnt16 == kRefRound) {
    s16 = t;
    cnt16 = 0;
  }
  return !(s.logT < kLogCutoff && iters < C.max_iters);
}

// Integrates the gathered events in order. Returns true once the ray is finished.
template <int KBUF, int DEG>
__device__ __forceinline__ bool consume(const SceneRef& sc, const TraceCtx& C, const Ray& ray, const float* B,
                                        int bs, int64_t slot, uint64_t (&buf)[KBUF], State& s, float4& last_dirac,
                                        int& iters, float& s16, int& cnt16, uint64_t& lower, uint32_t& status) {
  const uint64_t last = buf[KBUF - 1];
  bool done = false;
  for (int n = 0; n < KBUF && !done; ++n) {
    const uint64_t k = buf[0];
#pragma unroll
    for (int i = 0; i < KBUF - 1; ++i) buf[i] = buf[i + 1];
    buf[KBUF - 1] = kEmptyKey;
    if (k == kEmptyKey) return true;  // nothing left beyond the last gathered event
    done = consume_event<DEG>(sc, C, ray, B, bs, slot, k, s, last_dirac, iters, s16, cnt16, status);
  }
  if (done || last == kEmptyKey) return true;
  lower = last;
  return false;
}

template <int DEG>
__device__ __forceinline__ void init_density(const SceneRef& sc, const float* B, int bs, int n_mem,
                                             const int (&mem_j)[kMaxMembers], float4 extra, uint32_t status,
                                             State& s) {
  const int fst = feat_stride(sc.K);
  for (int q = 0; q < n_mem; ++q) {
    const int j = mem_j[q];
    const float4 r3 = __ldg(&sc.recs[j].r3);
    const float sg = r3.x;
    const float3 c = DEG == 0 ? dc_colour(r3) : sh_colour<DEG>(sc.features + int64_t(j) * fst, B, bs);
    s.drgb.x = s.drgb.x + sg;
    s.drgb.y = s.drgb.y + sg * c.x;
    s.drgb.z = s.drgb.z + sg * c.y;
    s.drgb.w = s.drgb.w + sg * c.z;
  }
  if (status & EVER_STATUS_INIT_OVERFLOW) {
    s.drgb.x = s.drgb.x + extra.x;
    s.drgb.y = s.drgb.y + extra.y;
    s.drgb.z = s.drgb.z + extra.z;
    s.drgb.w = s.drgb.w + extra.w;
  }
}

__device__ __forceinline__ void write_outputs(const EverForwardOut& out, int64_t r, const State& s, float4 last_dirac,
                                              int iters, uint32_t status) {
  float* o = out.out + 5 * r;
  o[0] = s.C.x;
  o[1] = s.C.y;
  o[2] = s.C.z;
  o[3] = 1.f - expf(-s.logT);
  o[4] = s.dist_x - s.dist_y;
  if (out.states) {
    float4* st = reinterpret_cast<float4*>(out.states + 16 * r);
    st[0] = make_float4(s.dist_x, s.dist_y, s.cum_x, s.cum_y);
    st[1] = make_float4(0.f, 0.f, 0.f, s.t);
    st[2] = s.drgb;
    st[3] = make_float4(s.logT, s.C.x, s.C.y, s.C.z);
  }
  if (out.last_dirac) reinterpret_cast<float4*>(out.last_dirac)[r] = last_dirac;
  out.iters[r] = iters;
  if (out.ray_stats) {
    out.ray_stats[2 * r] = float(iters);
    out.ray_stats[2 * r + 1] = s.t;
  }
  if (status && out.status) atomicOr(out.status, int(status));
}

__device__ __forceinline__ Ray load_ray(const float* rayo, const float* rayd, int64_t r, float tmin) {
  const float3 ro = make_float3(rayo[3 * r], rayo[3 * r + 1], rayo[3 * r + 2]);
  const float3 rd = make_float3(rayd[3 * r], rayd[3 * r + 1], rayd[3 * r + 2]);
  return make_ray(ro, rd, tmin);
}

__device__ __forceinline__ SceneRef scene_of(const FwdParams& P) {
  return SceneRef{reinterpret_cast<const Node*>(P.nodes), reinterpret_cast<const Record*>(P.records), P.features,
                  P.order, P.N, P.K};
}

template <int KBUF, int DEG>
__global__ void __launch_bounds__(256) k_trace_fwd_ray(const FwdParams P) {
  extern __shared__ int smem[];
  const int tid = threadIdx.x, stride = blockDim.x;
  int* st_node = smem + tid;
  float* st_t = reinterpret_cast<float*>(smem + kStackDepth * stride) + tid;
  const int64_t gi = int64_t(blockIdx.x) * blockDim.x + tid;
  if (gi >= P.R) return;
  const int64_t r = P.ray_order ? int64_t(P.ray_order[gi]) : gi;
  const SceneRef sc = scene_of(P);
  const TraceCtx C{P.tmin, P.tmax, P.max_iters, P.out, P.stack_depth, P.depth_hint, P.left};
  const Ray ray = load_ray(P.rayo, P.rayd, r, P.tmin);
  const RaySlab sl = make_slab(ray);
  float B[16];
  sh_basis<DEG>(ray.rd, B);
  uint32_t status = 0;
  State s = empty_state();
  float4 last_dirac = make_float4(0.f, 0.f, 0.f, 0.f);
  int iters = 0;
  if (sc.N > 0) {
    int mem_p[kMaxMembers], mem_j[kMaxMembers];
    float4 extra = make_float4(0.f, 0.f, 0.f, 0.f);
    const int n_mem = point_members<DEG, false>(sc.nodes, sc.recs, sc.order, sc.features, feat_stride(sc.K), B, 1,
                                                ray, true,
                                                st_node, stride, C.depth, 0, mem_p, mem_j, extra, status);
    init_density<DEG>(sc, B, 1, n_mem, mem_j, extra, status, s);
    float s16 = 0.f;
    int cnt16 = 0;
    uint64_t lower = 0;
    bool done = C.max_iters <= 0;
    while (!done) {
      uint64_t buf[KBUF];
#pragma unroll
      for (int i = 0; i < KBUF; ++i) buf[i] = kEmptyKey;
      gather_ray<KBUF>(sc.nodes, sc.recs, ray, sl, lower, s16, C.tmax, buf, st_node, st_t, stride, C.depth,
                       status);
      done = consume<KBUF, DEG>(sc, C, ray, B, 1, gi, buf, s, last_dirac, iters, s16, cnt16, lower, status);
    }
  }
  write_outputs(C.out, r, s, last_dirac, iters, status);
}

// The SH basis of the ray's direction into the block's shared array (B[k * bs]).
template <int DEG>
__device__ __forceinline__ void store_basis(const Ray& ray, float* B, int bs) {
  float Bl[16];
  sh_basis<DEG>(ray.rd, Bl);
#pragma unroll
  for (int k = 0; k < (DEG + 1) * (DEG + 1); ++k) B[k * bs] = Bl[k];
}

// What a ray carries from one gather round to the next. cnt16 is not kept: it always equals
// iters % kRefRound (both count the consumed events from zero).
struct RayLoop {
  State s;
  float4 last_dirac;
  int iters;
  float s16;
  int cnt16;
  uint64_t lower;
  uint32_t status;
};

// Initial state of a ray: empty, plus the density of the ellipsoids its start lies in.
template <int DEG>
__device__ __forceinline__ RayLoop start_ray(const SceneRef& sc, const Ray& ray, bool valid, int* wstack, int depth,
                                             float* B,
                                             int bs, int lane) {
  RayLoop L;
  L.status = 0;
  L.s = empty_state();
  L.last_dirac = make_float4(0.f, 0.f, 0.f, 0.f);
  L.iters = 0;
  L.s16 = 0.f;
  L.cnt16 = 0;
  L.lower = 0;
  if (sc.N > 0) {
    int mem_p[kMaxMembers], mem_j[kMaxMembers];
    float4 extra = make_float4(0.f, 0.f, 0.f, 0.f);
    const int n_mem = point_members<DEG, true>(sc.nodes, sc.recs, sc.order, sc.features, feat_stride(sc.K), B, bs,
                                               ray, valid,
                                               wstack, 1, depth, lane, mem_p, mem_j, extra, L.status);
    init_density<DEG>(sc, B, bs, n_mem, mem_j, extra, L.status, L.s);
  }
  return L;
}

// Gather + consume rounds of a warp's packet until no lane is active or max_rounds rounds
// have run. Returns whether this lane's ray needs another round.
template <int KBUF, int DEG>
__device__ __forceinline__ bool run_rounds(const SceneRef& sc, const TraceCtx& C, const Ray& ray, const float* B, int bs,
                                           int64_t slot, int* wstack, int lane, bool act, RayLoop& L, int max_rounds) {
  const RaySlab sl = make_slab(ray);
  for (int round = 0; round < max_rounds && __any_sync(kFull, act); ++round) {
    uint64_t buf[KBUF];
#pragma unroll
    for (int i = 0; i < KBUF; ++i) buf[i] = kEmptyKey;
    gather_packet<KBUF>(sc.nodes, sc.recs, ray, sl, act, L.lower, L.s16, C.tmax, buf, wstack, lane, C.depth,
                        L.status);
    if (act)
      act = !consume<KBUF, DEG>(sc, C, ray, B, bs, slot, buf, L.s, L.last_dirac, L.iters, L.s16, L.cnt16, L.lower,
                                L.status);
  }
  return act;
}

// ---- packet frustum phase ----
// Bound by issued instructions (54% of the issue slots busy, ALU pipe 41%, DRAM 2%), so the
// phase is cut into steps that each keep the lanes busy:
//  - list_leaves: the warp bounds its rays by intervals (origins, inverse directions), walks
//    the BVH with one child box per lane and lists the leaves whose box some ray can meet;
//    each lane then tests one listed ellipsoid against the cone of the packet's
//    directions, which drops 40% of them (boxes of thin turned ellipsoids are mostly
//    empty), and the rest are sorted by the earliest t at which any ray can enter them;
//  - every lane tests the leaves in that order; a leaf's events on the lane's ray go into
//    its sorted buffer, and before the next leaf, whose events all lie at or beyond that
//    leaf's entry bound T, the events below T are final;
//  - order_events takes the final events in order, decides where the ray ends and logs them;
//  - ring_integrate integrates them later, most lanes at once.
// So each ray integrates exactly its sorted event sequence, as the rounds do. Where the
// leaves of the whole t range do not fit, the phase goes on in stages over t. At 1M
// ellipsoids / 1080p the forward's kernels took 6.26 ms before (one walk over whole nodes,
// no cone test, integration where an event became final, a second pass of stack rounds for
// overflowing packets) and take 3.6 ms; a packet issues 37k instructions, 66k before. The
// sweeps below were taken when it was 3.5 ms, by event times within one run.
// Rays in no order (no_order) have no list in common and go to the rounds at once.
// Events a lane holds in the frustum phase: more cost registers and compares, fewer cost the
// lanes that run out another pass over the list (kernel time at 1M ellipsoids / 1080p and for
// 100,000 dense ones at 800 x 800 with 8 / 10 / 12 / 16 events: 3.58 / 3.49 / 3.56 / 3.83 and
// 1.68 / 1.57 / 1.48 / 1.49 ms).
constexpr int frustum_buffer(int kbuf) { return kbuf == 32 ? 16 : (kbuf == 8 ? 8 : 10); }
constexpr int kLowEvents = 4;  // buffered events up to which an insertion moves only the first entries
constexpr int kHold = 4;       // leaves between two rounds of ordering (8: 3.51 ms)
constexpr int kWalkCap = 256;  // nodes waiting in the walk
// Leaves of a group's first stage. Fewer prune the walk sooner, but a group that needs more
// walks again. With 96: 3.68 against 3.60 ms then (dense 2.98 against 1.69); with 192: 3.49
// against 3.49 (2M ellipsoids 3.75 against 3.59).
constexpr int kFirstLeaves = 128;
constexpr int kStageLeaves = 256;  // leaves of a later stage
constexpr int kCandCap = kStageLeaves + 64;
// Cuts of a list that overflows in one walk, for packets with a cone (6 without one: such a
// group is better traced by the rounds). With 6 for all, packets through dense ellipsoids gave
// up and were halved again and again: one took 3.3 ms where all 20,000 take 1.6 ms. With 64 the
// wide packets of small views cut too long (batched views 4.4 -> 5.0 ms).
constexpr int kMaxCuts = 16;
constexpr int kMaxStages = 128;  // then the rounds take over
// Passes over a stage's list, after which the stage ends where its slowest lane is and the next
// lists half as many leaves (kShortList at least): where a ray is inside many ellipsoids at
// once, each pass tests every leaf for the few events that a lane's buffer takes (262,144 rays
// through 10,000 ellipsoids three times over 10.1 -> 7.3 ms; with 3 passes a dense uniform
// scene 1.02 -> 1.14 ms, with 8 the first 7.8).
constexpr int kMaxPasses = 5;
constexpr int kShortList = 96;
constexpr int kTileWords = 28;
constexpr int kStateWords = 14;  // of a lane's integration state: State (13), the last event's id
// Shared ints per warp: the walk's nodes with their entry bounds (before and after it, the
// traversal stack of the rounds; after it, the events' ring),
// the leaf keys (64-bit), the lanes' integration state, the packet's direction tile.
constexpr int kWarpInts = 2 * kWalkCap + 2 * kCandCap + kStateWords * 32 + kTileWords;

// Warp minimum / maximum; NaN lanes are ignored (a NaN ray meets nothing).
__device__ __forceinline__ float warp_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float rcp_approx(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

// Interval bounds of a packet's rays for the box test. On an axis whose directions share a
// sign, every ray enters a box through one plane (the upper one where the sign is negative)
// and leaves it through the other, and the bound of the entry comes from one end of the
// origins' interval: o_near; that of the exit from the other: o_far.
struct PacketBounds {
  float o_near[3], o_far[3];
  float imin[3], imax[3];  // inverse directions (as the per-ray slab test takes them)
  unsigned neg, free;      // axes with negative directions / with directions of both signs
};

// The packet's rays as a cone of directions, and the origin and direction intervals that
// the free axes need; one copy per warp in shared memory.
struct PacketTile {
  float o[3];      // the common point of the rays' lines (their origin before the tmin shift)
  float d0[3];     // centre direction; every ray's direction is a multiple of
  float e1[3];     //   d0 + a e1 + b e2 with |a|, |b| <= 1
  float e2[3];
  float omin[3], omax[3], dmin[3], dmax[3];  // free axes only
  float shift[3];  // how far rounding may have put a ray's start off its line; 0 with tmin = 0
};
static_assert(sizeof(PacketTile) <= kTileWords * sizeof(int), "tile words");

// Bounds over the lanes with `part` (all lanes take part in the reductions). Writes the tile;
// *area: its size, +inf when there is none (no common apex, or no narrow cone).
__device__ __forceinline__ PacketBounds packet_bounds(const Ray& ray, const RaySlab& sl, bool part, PacketTile* tile,
                                                      int lane, float* area) {
  PacketBounds P;
  const float o[3] = {ray.o.x, ray.o.y, ray.o.z}, d[3] = {ray.d.x, ray.d.y, ray.d.z};
  const float iv[3] = {sl.invd.x, sl.invd.y, sl.invd.z}, ap[3] = {ray.apex.x, ray.apex.y, ray.apex.z};
  P.neg = P.free = 0;
  bool common = true;
  float m[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float omin = warp_min(part ? o[a] : INFINITY), omax = warp_max(part ? o[a] : -INFINITY);
    const float dmin = warp_min(part ? d[a] : INFINITY), dmax = warp_max(part ? d[a] : -INFINITY);
    const float amin = warp_min(part ? ap[a] : INFINITY), amax = warp_max(part ? ap[a] : -INFINITY);
    P.imin[a] = warp_min(part ? iv[a] : INFINITY);
    P.imax[a] = warp_max(part ? iv[a] : -INFINITY);
    const bool neg = P.imax[a] < 0.f;
    if (neg) P.neg |= 1u << a;
    if (P.imin[a] < 0.f && P.imax[a] > 0.f) P.free |= 1u << a;
    P.o_near[a] = neg ? omin : omax;
    P.o_far[a] = neg ? omax : omin;
    common = common && amin == amax;
    m[a] = 0.5f * (dmin + dmax);
    // a start that is not the apex itself is rounded to half an ulp (2^-24 of its size), twice that here
    const float shift = 1.2e-7f * warp_max(part && o[a] != ap[a] ? fabsf(o[a]) : 0.f);
    if (lane == 0) {
      tile->o[a] = amin;
      tile->omin[a] = omin;
      tile->omax[a] = omax;
      tile->dmin[a] = dmin;
      tile->dmax[a] = dmax;
      tile->shift[a] = shift;
    }
  }
  // tangent plane of the middle direction, and the rays' rectangle in it: the smallest over a
  // few rotations. Only a bound is needed, so approximate reciprocals do (margins below).
  const float inv_m = rsqrtf(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
#pragma unroll
  for (int a = 0; a < 3; ++a) m[a] *= inv_m;
  const bool x_small = fabsf(m[0]) < 0.6f;
  float t1[3], t2[3];
  {  // t1 = m x axis
    const float ax = x_small ? 1.f : 0.f, ay = x_small ? 0.f : 1.f;
    t1[0] = -m[2] * ay;
    t1[1] = m[2] * ax;
    t1[2] = m[0] * ay - m[1] * ax;
    const float n = rsqrtf(t1[0] * t1[0] + t1[1] * t1[1] + t1[2] * t1[2]);
#pragma unroll
    for (int a = 0; a < 3; ++a) t1[a] *= n;
    t2[0] = m[1] * t1[2] - m[2] * t1[1];
    t2[1] = m[2] * t1[0] - m[0] * t1[2];
    t2[2] = m[0] * t1[1] - m[1] * t1[0];
  }
  const float dm = d[0] * m[0] + d[1] * m[1] + d[2] * m[2];
  const float k = 1.f / dm;
  const float u = (d[0] * t1[0] + d[1] * t1[1] + d[2] * t1[2]) * k;
  const float v = (d[0] * t2[0] + d[1] * t2[1] + d[2] * t2[2]) * k;
  float best = INFINITY, uc = 0.f, vc = 0.f, uh = 0.f, vh = 0.f, bc = 1.f, bs = 0.f;
  float cq = 1.f, sq = 0.f;
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {  // 0, 22.5, 45, 67.5 degrees
    const float x = cq * u + sq * v, y = cq * v - sq * u;
    const float x0 = warp_min(part ? x : INFINITY), x1 = warp_max(part ? x : -INFINITY);
    const float y0 = warp_min(part ? y : INFINITY), y1 = warp_max(part ? y : -INFINITY);
    const float a = (x1 - x0) * (y1 - y0);
    if (a < best) {
      best = a;
      uc = 0.5f * (x0 + x1);
      vc = 0.5f * (y0 + y1);
      uh = 0.5f * (x1 - x0);
      vh = 0.5f * (y1 - y0);
      bc = cq;
      bs = sq;
    }
    const float c = cq * 0.92387953f - sq * 0.38268343f;
    sq = cq * 0.38268343f + sq * 0.92387953f;
    cq = c;
  }
  // directions carry a few float roundings: 1e-6 of the unit tangent plane covers them
  uh = uh * 1.00001f + 1e-6f;
  vh = vh * 1.00001f + 1e-6f;
  *area = common && warp_min(part ? dm : INFINITY) > 0.5f ? uh * vh : INFINITY;
  if (lane == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float r1 = bc * t1[a] + bs * t2[a], r2 = bc * t2[a] - bs * t1[a];
      tile->d0[a] = m[a] + uc * r1 + vc * r2;
      tile->e1[a] = uh * r1;
      tile->e2[a] = vh * r2;
    }
  }
  __syncwarp();
  return P;
}

// A lower bound of the t at which any packet ray is in the box within [t_lo, cap], or +inf
// when no packet ray can meet it there. Interval products bound every ray's plane
// distances; the float rounding of the bound (a few ulps) is covered by widening it by a
// relative 1e-6. Axes whose direction changes sign bound no t: there the positions the
// packet reaches over the t range of the other axes must overlap the box.
__device__ __forceinline__ float packet_entry(const PacketBounds& P, const PacketTile* tile, float4 a, float4 b,
                                              float t_lo, float cap) {
  const float lo[3] = {a.x, a.y, a.z}, hi[3] = {a.w, b.x, b.y};
  float tn = 0.f, tf = cap;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const bool neg = P.neg >> q & 1u;
    const float dn = (neg ? hi[q] : lo[q]) - P.o_near[q], df = (neg ? lo[q] : hi[q]) - P.o_far[q];
    const float n = fminf(dn * P.imin[q], dn * P.imax[q]), f = fmaxf(df * P.imin[q], df * P.imax[q]);
    if (!(P.free >> q & 1u)) {
      tn = fmaxf(tn, n);
      tf = fminf(tf, f);
    }
  }
  tn = fmaxf(tn * 0.999999f, t_lo);  // tn >= 0; a product, so that an infinite bound stays one
  tf = tf + 1e-6f * fabsf(tf);
  if (!(tn <= tf)) return INFINITY;
  if (P.free) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      if (!(P.free >> q & 1u)) continue;
      const float d0 = tile->dmin[q], d1 = tile->dmax[q];
      const float xl = tile->omin[q] + fminf(fminf(tn * d0, tn * d1), fminf(tf * d0, tf * d1));
      const float xh = tile->omax[q] + fmaxf(fmaxf(tn * d0, tn * d1), fmaxf(tf * d0, tf * d1));
      const float tol = 1e-6f * (fabsf(xl) + fabsf(xh) + fabsf(tf));
      if (xh + tol < lo[q] || xl - tol > hi[q]) return INFINITY;
    }
  }
  return tn;
}

// Whether no ray of the packet's tile can meet ellipsoid j. In the ellipsoid's frame (unit
// sphere) the rays start at c and run along v0 + a v1 + b v2, |a|, |b| <= 1. They cross the
// plane through the centre normal to v0 in l + s' (a v1' + b v2'), v1' and v2' the parts of
// v1, v2 normal to v0, s' = s / (1 + a p1 + b p2): a parallelogram, once s' is replaced by
// its largest value. A ray's distance from the centre is at least its crossing point's
// times the cosine of its angle to v0, so the packet misses when the parallelogram stays
// farther than 1 / cos from the centre. In place of the radius 1 stands `rad`, which covers the
// float rounding of the exact test and of this one. Both work with W (x - mean), whose
// component i carries a few roundings of sum_a |W_ia| |x_a - mean_a| (about 18 times 2^-24 in
// all; 2e-6 is 33), which for a turned thin ellipsoid can be far more than the component;
// the roots along the ray add about 10 times 2^-24 of |c|. The exact test starts at the rounded
// rayo + tmin rayd, which lies off the ray's line by tile->shift: by as much as the coordinates
// are large, however near the ellipsoid. NaN never rejects.
__device__ __forceinline__ bool packet_misses(const PacketTile* T, const Record* __restrict__ recs, int j) {
  const float4* rp = reinterpret_cast<const float4*>(recs + j);
  const float4 r[3] = {__ldg(rp), __ldg(rp + 1), __ldg(rp + 2)};
  const float x = T->o[0] - r[0].w, y = T->o[1] - r[1].w, z = T->o[2] - r[2].w;
  float c[3], v0[3], v1[3], v2[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    c[i] = fmaf(r[i].z, z, fmaf(r[i].y, y, r[i].x * x));
    v0[i] = fmaf(r[i].z, T->d0[2], fmaf(r[i].y, T->d0[1], r[i].x * T->d0[0]));
    v1[i] = fmaf(r[i].z, T->e1[2], fmaf(r[i].y, T->e1[1], r[i].x * T->e1[0]));
    v2[i] = fmaf(r[i].z, T->e2[2], fmaf(r[i].y, T->e2[1], r[i].x * T->e2[0]));
  }
  auto dot = [](const float (&p)[3], const float (&q)[3]) { return fmaf(p[2], q[2], fmaf(p[1], q[1], p[0] * q[0])); };
  const float iv = rcp_approx(dot(v0, v0));
  const float s = -dot(c, v0) * iv, p1 = dot(v1, v0) * iv, p2 = dot(v2, v0) * iv;
  const float g = fabsf(p1) + fabsf(p2);
  float l[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    l[i] = fmaf(s, v0[i], c[i]);
    v1[i] = fmaf(-p1, v0[i], v1[i]);
    v2[i] = fmaf(-p2, v0[i], v2[i]);
  }
  const float k = rcp_approx(1.f - g), sk = s * k;
  const float q11 = dot(v1, v1), q22 = dot(v2, v2);
  const float tan2 = 2.f * (q11 + q22) * iv * k * k;
  const float A = dot(l, l), B1 = sk * dot(l, v1), B2 = sk * dot(l, v2), s2 = sk * sk;
  const float C11 = s2 * q11, C22 = s2 * q22, C12 = s2 * dot(v1, v2);
  const float det = C11 * C22 - C12 * C12;
  const bool inside = fabsf(B2 * C12 - B1 * C22) <= det && fabsf(B1 * C12 - B2 * C11) <= det;
  const float i1 = rcp_approx(C11), i2 = rcp_approx(C22);
  float f = INFINITY;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const float sg = e ? -1.f : 1.f;
    const float h1 = fmaf(sg, C12, B1), h2 = fmaf(sg, C12, B2);
    const float a = clampf(-h1 * i1, -1.f, 1.f), b = clampf(-h2 * i2, -1.f, 1.f);
    f = fminf(f, fmaf(a, fmaf(a, C11, 2.f * h1), fmaf(2.f * sg, B2, A + C22)));
    f = fminf(f, fmaf(b, fmaf(b, C22, 2.f * h2), fmaf(2.f * sg, B1, A + C11)));
  }
  const float ex = fmaf(2e-6f, fabsf(x), T->shift[0]), ey = fmaf(2e-6f, fabsf(y), T->shift[1]),
              ez = fmaf(2e-6f, fabsf(z), T->shift[2]);
  float rad = fmaf(5e-6f, fabsf(c[0]) + fabsf(c[1]) + fabsf(c[2]), 1.001f);
#pragma unroll
  for (int i = 0; i < 3; ++i) rad = fmaf(fabsf(r[i].z), ez, fmaf(fabsf(r[i].y), ey, fmaf(fabsf(r[i].x), ex, rad)));
  const float lim = (1.f + tan2) * (rad * rad) + 4e-6f * (A + C11 + C22);
  return g < 0.5f && !inside && f > lim && C11 + C22 < 1e5f;
}

// Drops the leaves that the packet's tile misses from cand[0, n), keeping the others.
__device__ __forceinline__ int cull_leaves(const PacketTile* tile, const Record* __restrict__ recs, uint64_t* cand,
                                           int from, int n, int lane) {
  int kept = from;
  const unsigned below = (1u << lane) - 1u;
#pragma unroll 1
  for (int base = from; base < n; base += 32) {
    const int i = base + lane;
    uint64_t key = kEmptyKey;
    bool keep = false;
    if (i < n) {
      key = cand[i];
      keep = !packet_misses(tile, recs, int(uint32_t(key)));
    }
    const unsigned m = __ballot_sync(kFull, keep);
    __syncwarp();
    if (keep) cand[kept + __popc(m & below)] = key;
    kept += __popc(m);
  }
  __syncwarp();
  return kept;
}

// Keeps the nearest `least` to `most` (ties permitting) of cand[0, n) and returns their
// number; every dropped leaf's entry bound is at least *cut. 0 when all entry bounds are equal.
__device__ __forceinline__ int nearer_leaves(uint64_t* cand, int n, int least, int most, int lane, float* cut) {
  uint32_t lo = 0, hi = 0x7f800000u;  // fewer than `least` bounds lie below lo, more than `most` below hi
  int kept = 0;
  uint32_t at = 0;
  while (hi - lo > 1) {
    at = lo + (hi - lo) / 2;
    int c = 0;
    for (int i = lane; i < n; i += 32) c += uint32_t(cand[i] >> 32) < at ? 1 : 0;
    kept = __reduce_add_sync(kFull, c);
    if (kept < least) lo = at;
    else if (kept > most) hi = at;
    else break;
  }
  if (kept < least || kept > most) {  // a run of equal bounds spans the range: cut below or above it
    int below = 0;
    for (int i = lane; i < n; i += 32) below += uint32_t(cand[i] >> 32) < lo ? 1 : 0;
    at = __reduce_add_sync(kFull, below) > 0 ? lo : hi;
  }
  *cut = __uint_as_float(at);
  int out = 0;
  const unsigned under = (1u << lane) - 1u;
  for (int base = 0; base < n; base += 32) {
    const int i = base + lane;
    const uint64_t key = i < n ? cand[i] : kEmptyKey;
    const bool keep = uint32_t(key >> 32) < at;
    const unsigned m = __ballot_sync(kFull, keep);
    __syncwarp();
    if (keep) cand[out + __popc(m & under)] = key;
    out += __popc(m);
  }
  __syncwarp();
  return out < n ? out : 0;
}

// Walk of the BVH with one child box per lane and 32 nodes at a time (two boxes per lane
// in flight: the walk waits on its loads), nearer siblings first, from a stack of nodes and
// their entry bounds in shared memory. Lists the leaf keys (entry bound bits << 32 |
// position) of the leaves the packet can meet within [t_lo, *cap] in cand[0, n). When more
// than `limit` remain, the nearest are kept and *cap is lowered to where they end. Returns
// n <= limit, or -1 when no cut clearly beyond t_lo leaves few enough (many leaves reach
// back to t_lo: stages would hardly advance) or too many cuts were needed (a group this
// wide gains nothing from a common list).
__device__ __forceinline__ int packet_leaves(const Node* __restrict__ nodes, const Record* __restrict__ recs,
                                             const PacketBounds& P, const PacketTile* tile, bool cull, float t_lo,
                                             float* cap, int limit, int* stack, uint64_t* cand, int lane) {
  float* bound = reinterpret_cast<float*>(stack + kWalkCap);
  if (lane == 0) {
    stack[0] = 0;
    bound[0] = t_lo;
  }
  __syncwarp();
  int sp = 1, nc = 0, checked = 0, cuts = 0;
  const unsigned below = (1u << lane) - 1u;
#pragma unroll 1
  while (sp > 0) {
    const int take = min(min(sp, 32), kWalkCap - sp);
    if (take == 0) return -1;
    sp -= take;
    float4 a[2], b[2];
    bool on[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = 16 * k + (lane >> 1);
      on[k] = i < take && bound[sp + i] <= *cap;
      if (on[k]) {
        const float4* p = reinterpret_cast<const float4*>(nodes + stack[sp + i]) + 2 * (lane & 1);
        a[k] = __ldg(p);
        b[k] = __ldg(p + 1);
      }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (k == 1 && take <= 16) break;
      const float te = on[k] ? packet_entry(P, tile, a[k], b[k], t_lo, *cap) : INFINITY;
      const int c = on[k] ? child_link(b[k]) : 0;
      const bool hit = te != INFINITY, in = hit && c >= 0, leaf = hit && c < 0;
      const float sib = __shfl_xor_sync(kFull, te, 1);
      const bool near = te < sib || (te == sib && (lane & 1));
      const unsigned mf = __ballot_sync(kFull, in && !near), mn = __ballot_sync(kFull, in && near);
      const unsigned ml = __ballot_sync(kFull, leaf);
      if (in) {
        const int q = sp + (near ? __popc(mf) + __popc(mn & below) : __popc(mf & below));
        stack[q] = c;
        bound[q] = te;
      }
      if (leaf) cand[nc + __popc(ml & below)] = (uint64_t(__float_as_uint(te)) << 32) | uint32_t(~c);
      sp += __popc(mf) + __popc(mn);
      nc += __popc(ml);
    }
    __syncwarp();
    if (nc > limit || sp == 0) {
      if (cull) nc = checked = cull_leaves(tile, recs, cand, checked, nc, lane);
      if (nc > limit) {
        nc = checked = nearer_leaves(cand, nc, limit / 2, limit - limit / 8, lane, cap);
        if (nc == 0 || nc > limit || !(*cap > 1.001f * t_lo + 1e-6f) || ++cuts > (cull ? kMaxCuts : 6))
          return -1;
      }
    }
  }
  return nc;
}

__device__ __forceinline__ uint64_t shfl_xor64(uint64_t v, int m) {
  const uint32_t lo = __shfl_xor_sync(kFull, uint32_t(v), m), hi = __shfl_xor_sync(kFull, uint32_t(v >> 32), m);
  return (uint64_t(hi) << 32) | lo;
}

// Sorts cand[0, n) ascending (n <= 32 * E): bitonic, key r * 32 + lane in register r, strides
// below 32 by shuffles, the others inside the lane. The stage loops stay rolled: unrolled
// they are thousands of instructions that run once per packet, and the instruction cache
// misses cost more than the loops.
template <int E>
__device__ __forceinline__ void sort_keys_r(uint64_t* cand, int n, int lane) {
  uint64_t k[E];
#pragma unroll
  for (int r = 0; r < E; ++r) k[r] = 32 * r + lane < n ? cand[32 * r + lane] : kEmptyKey;
#pragma unroll 1
  for (int size = 2; size <= 32 * E; size <<= 1) {
#pragma unroll
    for (int d = E / 2; d > 0; d >>= 1) {  // stride 32 d
      if (size <= 32 * d) continue;
#pragma unroll
      for (int r = 0; r < E; ++r) {
        if (r & d) continue;
        const bool up = ((32 * r) & size) == 0;
        const uint64_t x = k[r], y = k[r | d];
        const bool sw = (x > y) == up;
        k[r] = sw ? y : x;
        k[r | d] = sw ? x : y;
      }
    }
#pragma unroll 1
    for (int stride = min(size >> 1, 16); stride > 0; stride >>= 1) {
      const bool lower = (lane & stride) == 0;
#pragma unroll
      for (int r = 0; r < E; ++r) {
        const uint64_t o = shfl_xor64(k[r], stride);
        const bool up = ((32 * r + lane) & size) == 0;
        const bool less = o < k[r];
        k[r] = (less == (lower == up)) ? o : k[r];
      }
    }
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < E; ++r) cand[32 * r + lane] = k[r];
  __syncwarp();
}
__device__ __forceinline__ void sort_keys(uint64_t* cand, int n, int lane) {
  if (n <= 64) sort_keys_r<2>(cand, n, lane);
  else if (n <= 128) sort_keys_r<4>(cand, n, lane);
  else sort_keys_r<8>(cand, n, lane);
}
static_assert(kStageLeaves <= 256, "sort_keys takes up to 256 keys");

// The sorted leaf list of a group of the warp's rays (the lanes with `mine`) within [t_lo,
// cap]: bounds, walk and sort, over the warp's lists at smem[at]. A call of its own, so that
// the walk and the passes over its list keep their registers apart. Returns the number of leaves (packet_leaves) and the cap.
struct LeafList {
  int n;
  float cap;
  float area;  // of the group's tile of directions; +inf if its rays share no apex
};
__device__ __noinline__ LeafList list_leaves(const Node* nodes, const Record* recs, float3 o, float3 d, float3 apex,
                                             bool mine, float t_lo, float cap, int limit, int at, int lane) {
  extern __shared__ int smem[];
  int* walk = smem + at;
  uint64_t* cand = reinterpret_cast<uint64_t*>(walk + 2 * kWalkCap);
  PacketTile* tile = reinterpret_cast<PacketTile*>(walk + 2 * kWalkCap + 2 * kCandCap + kStateWords * 32);
  Ray ray;
  ray.o = o;
  ray.d = d;
  ray.apex = apex;
  float area;
  const PacketBounds P = packet_bounds(ray, make_slab(ray), mine, tile, lane, &area);
  const bool cull = area < INFINITY;
  const int n = packet_leaves(nodes, recs, P, tile, cull, t_lo, &cap, cull || limit < kFirstLeaves ? limit : kStageLeaves, walk, cand, lane);
  if (n > 0) sort_keys(cand, n, lane);
  return LeafList{n, cap, area};
}

// Events that the frustum phase has put in order but not yet integrated: a ring per lane in
// shared memory (over the walk's stack, which is done by then). The ordering step keeps only
// the density and optical-depth sums that decide when a ray ends; colour, distortion and the
// rest of the state stay in shared memory and take their events kRingBurst at a time, when
// some lane's ring is full, so that most lanes integrate together.
constexpr int kRing = kWalkCap / 32;  // events per lane
constexpr int kRingBurst = kRing / 2;
static_assert(kRing * 32 == kWalkCap, "the ring takes the walk's stack");

struct Ring {
  uint64_t* ev;  // [kRing][32]
  float* st;     // [kStateWords][32]
  int head, n;   // this lane's first event and their number
};

__device__ __forceinline__ void ring_state_store(float* st, int lane, const State& s) {
  const float v[13] = {s.dist_x, s.dist_y, s.cum_x, s.cum_y, s.t, s.drgb.x, s.drgb.y, s.drgb.z, s.drgb.w,
                       s.logT,   s.C.x,    s.C.y,   s.C.z};
#pragma unroll
  for (int i = 0; i < 13; ++i) st[32 * i + lane] = v[i];
}
__device__ __forceinline__ State ring_state_load(const float* st, int lane) {
  float v[13];
#pragma unroll
  for (int i = 0; i < 13; ++i) v[i] = st[32 * i + lane];
  State s;
  s.dist_x = v[0];
  s.dist_y = v[1];
  s.cum_x = v[2];
  s.cum_y = v[3];
  s.t = v[4];
  s.drgb = make_float4(v[5], v[6], v[7], v[8]);
  s.logT = v[9];
  s.C = make_float3(v[10], v[11], v[12]);
  return s;
}

// Control point of an event: +-density and +-density * colour.
template <int DEG>
__device__ __forceinline__ float4 event_dirac(const SceneRef& sc, const float* B, int bs, uint32_t id) {
  const int j = int(id >> 1);
  const float4 r3 = __ldg(&sc.recs[j].r3);
  const float3 c = DEG == 0 ? dc_colour(r3) : sh_colour<DEG>(sc.features + int64_t(j) * feat_stride(sc.K), B, bs);
  const float dh = (id & 1u) ? -r3.x : r3.x;
  return make_float4(dh, dh * c.x, dh * c.y, dh * c.z);
}

// Integrates up to `most` of each lane's waiting events.
template <int DEG>
__device__ __forceinline__ void ring_integrate(const SceneRef& sc, const float* B, int bs, Ring& q, int lane,
                                               int most) {
  const int n = min(q.n, most);
  if (n > 0) {
    State s = ring_state_load(q.st, lane);
    uint32_t id = 0;
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      const uint64_t k = q.ev[((q.head + i) & (kRing - 1)) * 32 + lane];
      id = uint32_t(k);
      update(s, key_t(k), event_dirac<DEG>(sc, B, bs, id));
    }
    ring_state_store(q.st, lane, s);
    q.st[32 * 13 + lane] = __uint_as_float(id);
    q.head += n;
    q.n -= n;
  }
  __syncwarp();
}

// The entry root of ellipsoid j; a call, since only exits beyond tmax need it.
__device__ __noinline__ float entry_time(const Record* recs, int j, float3 o, float3 d) {
  Ray ray;
  ray.o = o;
  ray.d = d;
  HitT H;
  intersect(load_record(recs, j), ray, H);
  return H.t0;
}

// Takes every lane's next events, all before T: in order, under the reference's round rules
// (as consume_event), into the event log and the lane's ring. Clears live and act of a
// lane whose ray ends. drain: also integrates what is left in the rings.
template <int FBUF, int DEG>
__device__ __forceinline__ void order_events(const SceneRef& sc, const TraceCtx& C, const Ray& ray, const float* B,
                                             int bs, int64_t slot, int lane, uint64_t T, uint64_t (&buf)[FBUF],
                                             Ring& q, RayLoop& L, float& sigma, float& t_last, float& depth,
                                             bool& live, bool& act, bool drain) {
#pragma unroll 1
  for (;;) {
    const bool want = live && buf[0] < T;
    const bool any = __any_sync(kFull, want);
    // the one place that integrates: a full ring, or the end of a pass with events waiting
    if (__any_sync(kFull, any ? want && q.n == kRing : drain && q.n > 0))
      ring_integrate<DEG>(sc, B, bs, q, lane, kRingBurst);
    else if (!any)
      break;
    if (want) {
      const uint64_t k = buf[0];
#pragma unroll
      for (int i = 0; i < FBUF - 1; ++i) buf[i] = buf[i + 1];
      buf[FBUF - 1] = kEmptyKey;
      L.lower = k;
      const float t = key_t(k);
      const int j = key_pos(k), ex = key_exit(k);
      bool take = t > L.s16;
      bool done = false;
      if (take && t > kSentinel) {
        take = false;
        done = true;
      }
      if (take && ex && t > C.tmax) {
        const float t0 = entry_time(sc.recs, j, ray.o, ray.d);
        take = t0 > L.s16 && t0 <= C.tmax;
      }
      if (take) {
        const float rho = __ldg(&sc.recs[j].r3.x);
        const float area = fmaxf(sigma * fmaxf(t - t_last, 0.f), 0.f);
        depth = fmaxf(area + depth, 0.f);
        sigma = sigma + (ex ? -rho : rho);
        t_last = t;
        q.ev[((q.head + q.n) & (kRing - 1)) * 32 + lane] = k;
        ++q.n;
        if (C.out.event_log) {
          if (L.iters < C.out.log_cap)
            C.out.event_log[slot * int64_t(C.out.log_cap) + L.iters] = 2 * j + (ex ? 0 : 1);
          else
            L.status |= EVER_STATUS_LOG_OVERFLOW;
        }
        if (C.out.touch_count) atomicAdd(C.out.touch_count + __ldg(sc.order + j), 1);
        ++L.iters;
        if ((L.iters & (kRefRound - 1)) == 0) L.s16 = t;
        done = !(depth < kLogCutoff && L.iters < C.max_iters);
      }
      if (done) live = act = false;
    }
  }
}

// The lanes of `todo` to trace as one group: all of them, or those before a gap in the order
// of directions more than 12 times the usual one (a launch order that leaves one patch of
// directions for a distant one inside the packet: the union of both would meet far too much).
__device__ __forceinline__ unsigned pick_group(const Ray& ray, unsigned todo, int lane) {
  const float px = __shfl_up_sync(kFull, ray.d.x, 1), py = __shfl_up_sync(kFull, ray.d.y, 1),
              pz = __shfl_up_sync(kFull, ray.d.z, 1);
  const bool pair = lane > 0 && ((todo >> (lane - 1)) & 3u) == 3u;
  const float gap = pair ? fabsf(ray.d.x - px) + fabsf(ray.d.y - py) + fabsf(ray.d.z - pz) : 0.f;
  const float most = warp_max(gap);
  float sum = gap;
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(kFull, sum, m);
  // the mean of the gaps up to the mean of all: what neighbours are apart
  const bool small = pair && gap * float(__popc(todo & (todo >> 1))) <= sum;
  float usual = small ? gap : 0.f;
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) usual += __shfl_xor_sync(kFull, usual, m);
  const int n = __popc(__ballot_sync(kFull, small));
  if (!(most * float(n) > 12.f * usual)) return todo;
  const int at = __ffs(__ballot_sync(kFull, pair && gap == most)) - 1;
  const unsigned before = todo & ((1u << at) - 1u);
  return before ? before : todo;
}

// Whether the rays of `todo` come in no order: 16 or more, neighbours apart by more than a
// fifth of the whole range of directions or of origins (random points: a third; runs of a
// curve or a tile: a tenth to a sixth). No common list serves them.
__device__ __forceinline__ bool no_order(const Ray& ray, unsigned todo, int lane) {
  const bool part = todo >> lane & 1u, pair = lane > 0 && ((todo >> (lane - 1)) & 3u) == 3u;
  const int pairs = __popc(todo & (todo >> 1));
  const float v[6] = {ray.d.x, ray.d.y, ray.d.z, ray.o.x, ray.o.y, ray.o.z};
  bool out = false;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    float gap = 0.f, range = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float x = h ? v[3 + a] : v[a], y = __shfl_up_sync(kFull, x, 1);
      gap += pair ? fabsf(x - y) : 0.f;
      range += warp_max(part ? x : -INFINITY) - warp_min(part ? x : INFINITY);
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) gap += __shfl_xor_sync(kFull, gap, m);
    out = out || gap > 0.2f * range * float(pairs);
  }
  return out && pairs >= 15;
}

// The lower half of a group's lanes.
__device__ __forceinline__ unsigned half_group(unsigned grp, int lane) {
  const bool low = (grp >> lane & 1u) && 2 * __popc(grp & ((1u << lane) - 1u)) < __popc(grp);
  return __ballot_sync(kFull, low);
}

// The frustum phase of a warp's packet, in stages over t: a stage lists the leaves of the
// next t range (the whole scene, unless they do not fit or a depth hint ends it early) and
// takes every event in it. The packet is traced as one group of lanes, or in several where
// its directions leave a gap or a stage's leaves are met by few of its lanes. Returns whether
// this lane's ray still needs rounds (L then holds its state after its last integrated event,
// L.lower that event's key): only where more leaves than the list holds reach over one t.
template <int KBUF, int DEG>
__device__ __forceinline__ bool frustum_phase(const SceneRef& sc, const TraceCtx& C, const Ray& ray, const float* B,
                                              int bs, int64_t slot, int64_t r, int at, int lane, bool act,
                                              RayLoop& L) {
  extern __shared__ int smem[];
  constexpr int FBUF = frustum_buffer(KBUF);
  if (!__any_sync(kFull, act)) return act;
  const float cap_all = fminf(C.tmax, kSentinel);
  int* walk = smem + at;  // the warp's lists
  uint64_t* cand = reinterpret_cast<uint64_t*>(walk + 2 * kWalkCap);
  Ring q{reinterpret_cast<uint64_t*>(walk), reinterpret_cast<float*>(cand + kCandCap), 0, 0};
  ring_state_store(q.st, lane, L.s);
  // the ordering step's own copy of what decides the ray's end
  float sigma = L.s.drgb.x, t_last = L.s.t, depth = L.s.logT;
  const int first = L.iters;
  float t_done = 0.f;  // every event of this lane's ray before it has been taken
  float whole = INFINITY;  // tile area of the group a half was taken from
  int limit = kFirstLeaves;
  bool halved = false;     // the last list did not fit
  unsigned todo = __ballot_sync(kFull, act), grp = pick_group(ray, todo, lane);
  if (grp == todo && no_order(ray, todo, lane)) return act;
#pragma unroll 1
  for (int stage = 0; todo && stage < kMaxStages; ++stage) {
    const bool mine = grp >> lane & 1u;
    const float t_lo = warp_min(mine ? t_done : INFINITY);
    float cap = cap_all;
    // With a depth hint a group's first stage covers t up to its largest guessed stopping t
    // (plus 5%). A poor guess costs time, never correctness.
    if (C.depth_hint && t_lo == 0.f) {
      const float h = warp_max(mine ? C.depth_hint[r] : -INFINITY);
      if (h > 0.f && 1.05f * h + 1e-3f < cap) cap = 1.05f * h + 1e-3f;
    }
    const LeafList list = list_leaves(sc.nodes, sc.recs, ray.o, ray.d, ray.apex, mine, t_lo, cap,
                                      t_lo == 0.f ? min(limit, kFirstLeaves) : limit, at, lane);
    int nc = list.n;
    const bool cut = list.cap < cap;
    cap = list.cap;
    // half a group's lanes cover as much as all did: directions in no order, for the rounds
    if (list.area > 0.7f * whole) break;
    whole = INFINITY;
    // More leaves than the list holds reach over one t. Where they do so at the start, fewer rays
    // would hardly meet fewer of them; farther on, half a packet may do once (1,000 large
    // ellipsoids among 50,000, 262,144 rays: halved down to single rays 157 ms, once anywhere
    // 40, once beyond the start 38, never 35, the rounds alone 31; 200,000 faint ones in four
    // views as one batch: once 47 ms, never 65).
    if (nc < 0) {
      if (limit < kFirstLeaves) {
        limit = kStageLeaves;
        continue;
      }
      if (halved || t_lo == 0.f || __popc(grp) == 1 || !(list.area < INFINITY)) break;
      halved = true;
      whole = list.area;
      grp = half_group(grp, lane);
      continue;
    }
    halved = false;
    // events from `end` on belong to the next stage
    const uint64_t end = uint64_t(cap < cap_all ? __float_as_uint(cap) : 0x7f800000u) << 32;
    // A leaf whose bound lies at or past the cut (the walk's margins list a few) has no event
    // before it, and must not raise T past it: a leaf left off the list may come first there.
    while (nc > 0 && cand[nc - 1] >= end) --nc;
    // Passes over the list: one, unless a lane's buffer overflows. It then keeps its smallest
    // events and takes those; the events from `over` (the smallest it dropped) on are
    // collected again by another pass.
    bool pending = mine;
    int hits = 0, passes = 0;
#pragma unroll 1
    do {
      uint64_t buf[FBUF];
#pragma unroll
      for (int i = 0; i < FBUF; ++i) buf[i] = kEmptyKey;
      uint64_t over = kEmptyKey;
      bool live = pending;
#pragma unroll 1
      for (int ci = 0;; ++ci) {
        // every 32 leaves, the lanes start the loads of the next 32 records into L1 (one each),
        // so the broadcast record loads of the loop below rarely wait on L2
        if ((ci & 31) == 0 && ci + lane < nc)
          asm volatile("prefetch.global.L1 [%0];" ::"l"(sc.recs + int(uint32_t(cand[ci + lane]))));
        const uint64_t ck = ci < nc ? cand[ci] : kEmptyKey;
        // events below T are final: no leaf still to come has an event before T
        const uint64_t T = ci < nc ? (ck & ~uint64_t(0xffffffffu)) : end;
        const bool stop = ci >= nc || !__any_sync(kFull, live);
        // ordering waits for a few leaves' events, so that more lanes take part in it
        if (stop || (ci & (kHold - 1)) == 0 || __any_sync(kFull, live && buf[FBUF - 2] != kEmptyKey))
          order_events<FBUF, DEG>(sc, C, ray, B, bs, slot, lane, T, buf, q, L, sigma, t_last, depth, live, act,
                                  stop);
        if (stop) break;
        live = live && T < over;
        // few buffered events in every lane (nearly always): an insertion moves only the first
        const bool low = !__any_sync(kFull, live && buf[kLowEvents] != kEmptyKey);
        if (live) {
          const int j = int(uint32_t(ck));
          const Record R = load_record(sc.recs, j);
          HitT H;
          if (intersect(R, ray, H)) {
            ++hits;
            const bool in0 = H.t0 > L.s16 && H.t0 <= C.tmax;
            const bool in1 = H.t1 > L.s16 && (H.t1 <= C.tmax || in0);
            uint64_t e0 = event_key(H.t0, j, 0), e1 = event_key(H.t1, j, 1);
            e0 = in0 && e0 > L.lower && e0 < over ? e0 : kEmptyKey;
            e1 = in1 && e1 > L.lower && e1 < over ? e1 : kEmptyKey;
            if (low) {
              buf_insert_low<kLowEvents + 2>(buf, e0);
              buf_insert_low<kLowEvents + 2>(buf, e1);
            } else {
              e0 = buf_insert_low<FBUF>(buf, e0);
              e1 = e1 < e0 ? buf_insert_low<FBUF>(buf, e1) : e1;
              over = min(over, min(e0, e1));
            }
          }
        }
      }
      pending = pending && act && over < end;
    } while (__any_sync(kFull, pending) && ++passes < kMaxPasses);
    const bool ended = __any_sync(kFull, pending);
    if (ended) limit = max(kShortList, limit / 2);
    else if (limit >= kFirstLeaves) limit = kStageLeaves;
    if (mine) {
      t_done = pending ? fminf(fmaxf(t_lo, key_t(L.lower)), cap_all) : cap;  // exits may lie beyond tmax
      if (!pending && cap >= cap_all) act = false;
    }
    const unsigned left = __ballot_sync(kFull, act);
    // a list that had to be cut short and that fewer than one lane in 32 met on average: the
    // group is too wide
    const bool wide = __reduce_add_sync(kFull, hits) * 32 < nc * __popc(grp);
    todo &= left;
    grp &= left;
    if (!grp) {
      grp = pick_group(ray, todo, lane);
    } else if (cut && wide && __popc(grp) > 1) {
      whole = list.area;
      grp = half_group(grp, lane);
    }
  }
  L.cnt16 = L.iters & (kRefRound - 1);
  L.s = ring_state_load(q.st, lane);
  if (L.iters > first) L.last_dirac = event_dirac<DEG>(sc, B, bs, __float_as_uint(q.st[32 * 13 + lane]));
  __syncwarp();
  return act;
}

// A ray that needs more rounds parks its loop state in its own output rows: `states` in
// the final layout, with s16 and the 64-bit key bound of the next round in the three
// padding words, `last_dirac` and `iters`. Its status flags are raised now.
__device__ __forceinline__ void park_ray(const EverForwardOut& out, int64_t r, const RayLoop& L) {
  float4* st = reinterpret_cast<float4*>(out.states + 16 * r);
  st[0] = make_float4(L.s.dist_x, L.s.dist_y, L.s.cum_x, L.s.cum_y);
  st[1] = make_float4(L.s16, __uint_as_float(uint32_t(L.lower)), __uint_as_float(uint32_t(L.lower >> 32)), L.s.t);
  st[2] = L.s.drgb;
  st[3] = make_float4(L.s.logT, L.s.C.x, L.s.C.y, L.s.C.z);
  reinterpret_cast<float4*>(out.last_dirac)[r] = L.last_dirac;
  out.iters[r] = L.iters;
  if (L.status && out.status) atomicOr(out.status, int(L.status));
}

__device__ __forceinline__ RayLoop resume_ray(const EverForwardOut& out, int64_t r) {
  const float4* st = reinterpret_cast<const float4*>(out.states + 16 * r);
  const float4 a = st[0], b = st[1], c = st[2], d = st[3];
  RayLoop L;
  L.s.dist_x = a.x;
  L.s.dist_y = a.y;
  L.s.cum_x = a.z;
  L.s.cum_y = a.w;
  L.s.t = b.w;
  L.s.drgb = c;
  L.s.logT = d.x;
  L.s.C = make_float3(d.y, d.z, d.w);
  L.s16 = b.x;
  L.lower = uint64_t(__float_as_uint(b.y)) | (uint64_t(__float_as_uint(b.z)) << 32);
  L.last_dirac = reinterpret_cast<const float4*>(out.last_dirac)[r];
  L.iters = out.iters[r];
  L.cnt16 = L.iters % kRefRound;
  L.status = 0;
  return L;
}

// Rounds that a packet runs itself on the rays that the frustum phase leaves it. Inside this
// kernel they have 16 warps per SM and the L1 that the lists leave, in their own 20 and nearly
// all of it; but a few rays there would run alone. So the first packets of a launch (as many as
// are resident) run two rounds, which is all that most such rays need (100,000 uniform
// ellipsoids all around, 262,144 rays: 2.8 ms, with every packet left at once 3.5); what
// they leave, and every later packet's rays, are the other kernel's (1,000 large ellipsoids
// among 50,000: 37 ms, with all rounds here 50).
constexpr int kRoundsHere = 2;
__device__ __forceinline__ int rounds_here(const LeftRays& left, int lane) {
  if (!left.words) return INT_MAX;
  uint32_t n = 0;
  if (lane == 0) n = atomicAdd(left.words + kLeftPackets, 1u);
  return __shfl_sync(kFull, n, 0) < left.packets_min ? kRoundsHere : 0;
}

// Lists the rays m of the packet of slots [first, first + 32).
__device__ __forceinline__ void leave_rays(const LeftRays& left, unsigned m, int64_t first, int lane) {
  if (lane != 0) return;
  left.masks[first >> 5] = m;
  left.list[atomicAdd(left.words + kLeftGroups, 1u)] = int32_t(first >> 5);
}

// The rounds that finish what the frustum phase leaves: rarely anything, so they are a call
// (inlined, they would cost the whole kernel registers), with its arguments in local memory.
struct RoundsCall {
  SceneRef sc;
  TraceCtx C;
  Ray ray;
  const float* B;
  int bs, lane;
  int64_t slot;
  int* wstack;
  bool act;
  RayLoop L;
  int rounds;
};
template <int KBUF, int DEG>
__device__ __noinline__ void rounds_call(RoundsCall* a) {
  RayLoop L = a->L;
  a->act = run_rounds<KBUF, DEG>(a->sc, a->C, a->ray, a->B, a->bs, a->slot, a->wstack, a->lane, a->act, L, a->rounds);
  a->L = L;
}

// One warp traces one packet of up to 32 rays against one scene (lanes with valid=false
// only take part in the warp-wide votes). FRUSTUM: the frustum phase, else rounds only.
template <int KBUF, int DEG, bool FRUSTUM>
__device__ __forceinline__ void trace_packet(const SceneRef& sc, const TraceCtx& C, const Ray& ray, int64_t r,
                                             bool valid, int64_t slot, int* wstack, float* B, int bs, int lane) {
  store_basis<DEG>(ray, B, bs);
  RayLoop L = start_ray<DEG>(sc, ray, valid, wstack, C.depth, B, bs, lane);
  bool act = valid && C.max_iters > 0 && sc.N > 0;
  if (FRUSTUM) {
    act = frustum_phase<KBUF, DEG>(sc, C, ray, B, bs, slot, r, int(threadIdx.x >> 5) * kWarpInts, lane, act, L);
    if (__any_sync(kFull, act)) {
      const int rounds = rounds_here(C.left, lane);
      if (rounds > 0) {
        RoundsCall a{sc, C, ray, B, bs, lane, slot, wstack, act, L, rounds};
        rounds_call<KBUF, DEG>(&a);
        L = a.L;
        act = a.act;
      }
      if (const unsigned m = __ballot_sync(kFull, act)) {
        leave_rays(C.left, m, slot - lane, lane);
        if (act) park_ray(C.out, r, L);
        valid = valid && !act;  // the outputs of those are the rounds' to write
      }
    }
  } else {
    run_rounds<KBUF, DEG>(sc, C, ray, B, bs, slot, wstack, lane, act, L, INT_MAX);
  }
  if (valid) write_outputs(C.out, r, L.s, L.last_dirac, L.iters, L.status);
  __syncwarp();
}

// Resident blocks per SM that the register budget of the packet kernels targets: 16 warps
// (128 registers) with the frustum phase, which is bound by instructions and not by latency
// (20 warps, with spills: 4.0 against 3.6 ms at 1M ellipsoids / 1080p); 20 warps (96
// registers) for the rounds, whose traversal is latency-bound.
template <int BLOCK, bool FRUSTUM = true>
struct FwdMinBlocks {
  static constexpr int value = BLOCK == 256 ? 2 : (FRUSTUM ? 512 : 640) / BLOCK;
};

template <int KBUF, int DEG, int BLOCK>
__global__ void __launch_bounds__(BLOCK, FwdMinBlocks<BLOCK>::value) k_trace_fwd_packet(const FwdParams P) {
  extern __shared__ int smem[];
  if (P.left.words && __ldg(P.left.words + kLeftVotes) >= P.left.votes_min) return;  // the rounds trace this launch
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int* wstack = smem + warp * kWarpInts;  // traversal stack, and the frustum phase's lists over it
  float* B = reinterpret_cast<float*>(smem + (blockDim.x / 32) * kWarpInts) + tid;  // B[k * blockDim.x]
  const int64_t gi = (int64_t(blockIdx.x) * (blockDim.x / 32) + warp) * P.lanes + lane;
  const bool valid = lane < P.lanes && gi < P.R;  // every lane stays for the warp-wide ballots
  const int64_t r = valid ? (P.ray_order ? int64_t(P.ray_order[gi]) : gi) : 0;
  const TraceCtx C{P.tmin, P.tmax, P.max_iters, P.out, P.stack_depth, P.depth_hint, P.left};
  const Ray ray = load_ray(P.rayo, P.rayd, r, P.tmin);
  trace_packet<KBUF, DEG, true>(scene_of(P), C, ray, r, valid, gi, wstack, B, blockDim.x, lane);
}

// Regrouped forward, one pass. PASS 0 takes every slot in order and runs the first gather
// round; PASS 1 runs one more round and PASS 2 every remaining round, each for the slots in
// `list` (count entries): the rays that the previous pass left active, packed into full
// warps in slot order. A pass 0 or 1 with fewer than `split_min` rays runs every remaining
// round instead (a later pass would hold too few rays to fill the GPU, and its latency-bound
// tail would run alone). Passes 0 and 1 park the rays that still need rounds and write one
// lane mask per warp (mask[position / 32]); the other rays write their outputs.
// Camera passes (CAM): slots are the camera's (camera.cuh); a slot's pixel ray is made in
// the kernel, padding slots take part only in the warp votes, and the event log has one
// column per slot.
struct PassCamera {
  CameraParams cam;
  const float* jitter;
  int64_t num_slots;
};

template <int KBUF, int DEG, int BLOCK, int PASS, bool CAM>
__global__ void __launch_bounds__(BLOCK, FwdMinBlocks<BLOCK, false>::value)
    k_trace_fwd_pass(const FwdParams P, const int32_t* __restrict__ list, const uint32_t* __restrict__ count,
                     uint32_t* __restrict__ mask, int64_t split_min, const PassCamera Q) {
  extern __shared__ int smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int* wstack = smem + warp * kStackDepth;
  float* B = reinterpret_cast<float*>(smem + (blockDim.x / 32) * kStackDepth) + tid;
  const int64_t gi = int64_t(blockIdx.x) * blockDim.x + tid;  // slot (PASS 0) or list position
  const int64_t slots = CAM ? Q.num_slots : P.R;
  const int64_t n = PASS == 0 ? slots : int64_t(*count);
  if ((gi & ~int64_t(31)) >= n) return;  // the whole warp lies beyond the list
  const int64_t slot = gi < n ? (PASS == 0 ? gi : int64_t(list[gi])) : 0;
  int64_t r = 0;
  bool valid = gi < n;
  if (CAM) {
    r = valid ? camera_slot_pixel(Q.cam, slot) : -1;
    valid = r >= 0;
  } else if (valid) {
    r = P.ray_order ? int64_t(P.ray_order[slot]) : slot;
  }
  if (!valid) r = 0;
  const SceneRef sc = scene_of(P);
  const TraceCtx C{P.tmin, P.tmax, P.max_iters, P.out, P.stack_depth, P.depth_hint, P.left};
  Ray ray;
  if (CAM) {
    float3 ro, rd;
    camera_ray(Q.cam, Q.jitter, r, ro, rd);
    ray = make_ray(ro, rd, P.tmin);
  } else {
    ray = load_ray(P.rayo, P.rayd, r, P.tmin);
  }
  store_basis<DEG>(ray, B, blockDim.x);
  RayLoop L;
  bool act;
  if (PASS == 0) {
    L = start_ray<DEG>(sc, ray, valid, wstack, C.depth, B, blockDim.x, lane);
    act = valid && C.max_iters > 0 && sc.N > 0;
  } else {
    if (valid) L = resume_ray(P.out, r);
    act = valid;
  }
  const bool last = PASS == 2 || n < split_min;
  act = run_rounds<KBUF, DEG>(sc, C, ray, B, blockDim.x, slot, wstack, lane, act, L, last ? INT_MAX : 1);
  if (PASS < 2 && mask) {
    const unsigned m = __ballot_sync(kFull, act);
    if (lane == 0) mask[gi >> 5] = m;
  }
  if (valid) {
    if (PASS < 2 && act)
      park_ray(P.out, r, L);
    else
      write_outputs(C.out, r, L.s, L.last_dirac, L.iters, L.status);
  }
}

// Rays in no order (random rays, shuffled pixels, the sorted pixels of many views) are traced by
// the gather rounds. Inside the frustum kernel these have 16 warps per SM and the L1 that the
// lists leave; in their own kernel 20 and nearly all of it: 262,144 random rays against 20,000
// ellipsoids 13.7 and 9.1 ms, against 300,000 22.7 and 15.6 ms; random pixels of 100 views 13.8
// and 8.6 ms. So one block looks at up to kVotePackets full packets, evenly spaced, and counts
// those in no order. More than half of them: the rounds take the launch. A launch with fewer
// (pixels of 8 views: an eighth) is the frustum kernel's, whose own rounds overlap with its
// other packets. The vote takes 6 us (256 packets in its block: 15) and the
// empty second launch 2.
constexpr uint32_t kVotePackets = 64;
__global__ void __launch_bounds__(1024) k_order_vote(const FwdParams P, uint32_t packets) {
  __shared__ uint32_t votes;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) votes = 0;
  __syncthreads();
  uint32_t n = 0;
#pragma unroll
  for (uint32_t q = 0; q < kVotePackets / 32; ++q) {
    const uint32_t v = 32 * q + threadIdx.x / 32;
    if (v >= packets) break;
    const int64_t gi = P.R / 32 * v / packets * 32 + lane;  // full packets only
    n += no_order(load_ray(P.rayo, P.rayd, P.ray_order ? int64_t(P.ray_order[gi]) : gi, P.tmin), kFull, lane) ? 1u : 0u;
  }
  if (lane == 0 && n) atomicAdd(&votes, n);
  __syncthreads();
  if (threadIdx.x < kLeftWords) P.left.words[threadIdx.x] = threadIdx.x == kLeftVotes ? votes : 0u;
}

// The rounds of a launch in no order, or of the rays that the frustum kernel has parked in the
// list. Persistent (an empty launch of one block per packet takes 10 us at full HD): warps take
// 32 slots at a time from a device counter.
constexpr int kLeftBlock = 128;
template <int KBUF, int DEG, bool CAM>
__global__ void __launch_bounds__(kLeftBlock, FwdMinBlocks<kLeftBlock, false>::value)
    k_trace_fwd_left(const FwdParams P, const PassCamera Q) {
  extern __shared__ int smem[];
  const bool all = !CAM && __ldg(P.left.words + kLeftVotes) >= P.left.votes_min;
  const int64_t n = all ? P.R : 32 * int64_t(__ldg(P.left.words + kLeftGroups));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int* wstack = smem + warp * kStackDepth;
  float* B = reinterpret_cast<float*>(smem + (kLeftBlock / 32) * kStackDepth) + tid;
  const SceneRef sc = scene_of(P);
  const TraceCtx C{P.tmin, P.tmax, P.max_iters, P.out, P.stack_depth, P.depth_hint, {}};
  while (n > 0) {
    uint32_t packet = 0;
    if (lane == 0) packet = atomicAdd(P.left.words + kLeftTaken, 1u);
    packet = __shfl_sync(kFull, packet, 0);
    const int64_t gi = int64_t(packet) * 32 + lane;
    if (int64_t(packet) * 32 >= n) break;
    const int32_t group = all ? int32_t(packet) : P.left.list[packet];
    const bool valid = all ? gi < n : P.left.masks[group] >> lane & 1u;
    const int64_t slot = valid ? 32 * int64_t(group) + lane : 0;
    int64_t r = slot;
    if (CAM) r = valid ? camera_slot_pixel(Q.cam, slot) : 0;
    else if (P.ray_order) r = valid ? int64_t(P.ray_order[slot]) : 0;
    Ray ray;
    if (CAM) {
      float3 ro, rd;
      camera_ray(Q.cam, Q.jitter, r, ro, rd);
      ray = make_ray(ro, rd, P.tmin);
    } else {
      ray = load_ray(P.rayo, P.rayd, r, P.tmin);
    }
    store_basis<DEG>(ray, B, kLeftBlock);
    RayLoop L;
    bool act = valid;
    if (all) {
      L = start_ray<DEG>(sc, ray, valid, wstack, C.depth, B, kLeftBlock, lane);
      act = valid && C.max_iters > 0 && sc.N > 0;
    } else if (valid) {
      L = resume_ray(P.out, r);
    }
    run_rounds<KBUF, DEG>(sc, C, ray, B, kLeftBlock, slot, wstack, lane, act, L, INT_MAX);
    if (valid) write_outputs(C.out, r, L.s, L.last_dirac, L.iters, L.status);
    __syncwarp();
  }
}

// Camera trace: rays are made from the camera in the kernel (no ray arrays). The launch
// covers the camera's slots, 32 per 8x4 pixel tile, so a warp traces one tile; outputs are
// written by pixel, event-log columns are slots.
template <int KBUF, int DEG, int BLOCK>
__global__ void __launch_bounds__(BLOCK, FwdMinBlocks<BLOCK>::value)
    k_trace_fwd_camera(const FwdParams P, const CameraParams cam, const float* __restrict__ jitter,
                       int64_t num_slots) {
  extern __shared__ int smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int* wstack = smem + warp * kWarpInts;  // traversal stack, and the frustum phase's lists over it
  float* B = reinterpret_cast<float*>(smem + (blockDim.x / 32) * kWarpInts) + tid;
  const int64_t gi = (int64_t(blockIdx.x) * (blockDim.x / 32) + warp) * P.lanes + lane;
  const int64_t p = lane < P.lanes && gi < num_slots ? camera_slot_pixel(cam, gi) : -1;
  const bool valid = p >= 0;
  const TraceCtx C{P.tmin, P.tmax, P.max_iters, P.out, P.stack_depth, P.depth_hint, P.left};
  float3 ro, rd;
  camera_ray(cam, jitter, valid ? p : 0, ro, rd);
  const Ray ray = make_ray(ro, rd, P.tmin);
  trace_packet<KBUF, DEG, true>(scene_of(P), C, ray, valid ? p : 0, valid, gi, wstack, B, blockDim.x, lane);
}

// Persistent batched forward: warps take 32-slot packets from a device counter until
// all views are done. Each packet lies inside one view, hence one scene.
template <int KBUF, int DEG, int BLOCK, bool FRUSTUM>
__global__ void __launch_bounds__(BLOCK, FwdMinBlocks<BLOCK, FRUSTUM>::value)
    k_trace_fwd_batched(const BatchFwdParams P) {
  extern __shared__ int smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kInts = FRUSTUM ? kWarpInts : kStackDepth;  // traversal stack, and the frustum phase's lists over it
  int* wstack = smem + warp * kInts;
  float* B = reinterpret_cast<float*>(smem + (blockDim.x / 32) * kInts) + tid;
  const TraceCtx C{P.tmin, P.tmax, P.max_iters, P.out, P.stack_depth, nullptr, {}};
  const int lanes = FRUSTUM ? P.lanes : 32;  // a divisor of 32: a packet never mixes views
  const int64_t num_packets = P.num_slots / lanes;
  for (;;) {
    unsigned int pk = 0;
    if (lane == 0) pk = atomicAdd(P.work_counter, 1u);
    pk = __shfl_sync(kFull, pk, 0);
    if (int64_t(pk) >= num_packets) break;
    const int64_t first = int64_t(pk) * lanes, slot = first + lane;
    int v = 0;  // the view holding this packet (few views: linear scan, warp-uniform)
    while (v + 1 < P.num_views && P.views[v + 1].slot_offset <= first) ++v;
    const BatchScene bs_ = P.scenes[P.views[v].scene];
    const SceneRef sc{reinterpret_cast<const Node*>(bs_.nodes), reinterpret_cast<const Record*>(bs_.records),
                      bs_.features, bs_.order, bs_.N, bs_.K};
    const int32_t r = lane < lanes ? P.slot_ray[slot] : -1;
    const Ray ray = load_ray(P.rayo, P.rayd, r >= 0 ? r : 0, P.tmin);
    trace_packet<KBUF, DEG, FRUSTUM>(sc, C, ray, r, r >= 0, slot, wstack, B, blockDim.x, lane);
  }
}

// Dynamic shared memory of a packet kernel: per warp its frustum-phase lists (or, for rounds
// only, its traversal stack), per thread the SH basis of its ray.
template <int DEG>
size_t packet_smem(int block, bool frustum = true) {
  return size_t(frustum ? kWarpInts : kStackDepth) * (block / 32) * sizeof(int) +
         size_t((DEG + 1) * (DEG + 1)) * block * sizeof(float);
}

// Dynamic shared memory above the 48 KB default needs the kernel's opt-in.
template <class Kern>
cudaError_t prepare(Kern kern, size_t smem) {
  if (smem <= size_t(48) * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
}

// Rays per packet. A launch that leaves warps idle takes fewer rays in each: a warp's time is
// the chain of its packet's leaves and events, and narrower packets have fewer (kernel time
// with 32 / 16 / 8 / 4 rays: 4,096 rays against 1,000 ellipsoids 115 / 71 / 55 / 50 us, 9,471
// rays against 20,000 400 / 262 / 177 / 91 us). Halved while the launch then still fits the
// resident warps (16 per SM); 4 rays at least (2: 82 us, the walk is repeated too often).
inline int packet_lanes(int64_t rays) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int lanes = 32;
  while (lanes > 4 && rays <= int64_t(sms) * 16 * (lanes / 2)) lanes /= 2;
  return lanes;
}

// Before the frustum kernel: the vote of a launch of full packets (it clears the words), or the
// words cleared.
inline cudaError_t left_begin(FwdParams& P, int64_t slots, bool cam, cudaStream_t st) {
  const uint32_t packets = uint32_t(std::min<int64_t>(slots / 32, kVotePackets));
  if (P.lanes < 32 || packets == 0 || P.max_iters <= 0) P.left.words = nullptr;  // no iterations: no rounds
  if (!P.left.words) return cudaSuccess;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  P.left.packets_min = uint32_t(16 * sms);  // the resident warps
  if (cam) {
    P.left.votes_min = UINT32_MAX;
    return cudaMemsetAsync(P.left.words, 0, kLeftWords * sizeof(uint32_t), st);
  }
  P.left.votes_min = packets / 2 + 1;
  k_order_vote<<<1, 1024, 0, st>>>(P, packets);
  return cudaGetLastError();
}
template <int KBUF, int DEG, bool CAM>
cudaError_t left_finish(const FwdParams& P, const PassCamera& Q, cudaStream_t st) {
  if (!P.left.words) return cudaGetLastError();
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t smem = packet_smem<DEG>(kLeftBlock, false);
  if (cudaError_t e_ = prepare(k_trace_fwd_left<KBUF, DEG, CAM>, smem)) return e_;
  k_trace_fwd_left<KBUF, DEG, CAM>
      <<<sms * FwdMinBlocks<kLeftBlock, false>::value, kLeftBlock, smem, st>>>(P, Q);
  return cudaGetLastError();
}

// Gather rounds only, one pass that runs them all.
template <int KBUF, int DEG, int BLOCK, bool CAM>
cudaError_t launch_rounds_b(const FwdParams& P, const PassCamera& Q, cudaStream_t st) {
  const int64_t n = CAM ? Q.num_slots : P.R;
  const size_t smem = packet_smem<DEG>(BLOCK, false);
  if (cudaError_t e_ = prepare(k_trace_fwd_pass<KBUF, DEG, BLOCK, 0, CAM>, smem)) return e_;
  k_trace_fwd_pass<KBUF, DEG, BLOCK, 0, CAM>
      <<<unsigned((n + BLOCK - 1) / BLOCK), BLOCK, smem, st>>>(P, nullptr, nullptr, nullptr, INT64_MAX, Q);
  return cudaGetLastError();
}
template <int KBUF, int DEG, bool CAM>
cudaError_t launch_rounds(const FwdParams& P, const PassCamera& Q, int block, cudaStream_t st) {
  switch (block) {
    case 64: return launch_rounds_b<KBUF, DEG, 64, CAM>(P, Q, st);
    case 128: return launch_rounds_b<KBUF, DEG, 128, CAM>(P, Q, st);
    default: return launch_rounds_b<KBUF, DEG, 256, CAM>(P, Q, st);
  }
}

template <int KBUF, int DEG>
cudaError_t launch_t(const FwdParams& P0, int block, int traversal, cudaStream_t st) {
  FwdParams P = P0;
  P.lanes = traversal == 0 ? packet_lanes(P.R) : 32;
  const int64_t grid = (P.R + P.lanes * (block / 32) - 1) / (P.lanes * (block / 32));
  if (traversal == 1) {
    const size_t smem = size_t(kStackDepth) * block * (sizeof(int) + sizeof(float));
    auto kern = k_trace_fwd_ray<KBUF, DEG>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return e;
    kern<<<unsigned(grid), block, smem, st>>>(P);
  } else if (traversal == 2) {
    return launch_rounds<KBUF, DEG, false>(P, PassCamera{}, block, st);
  } else {
    if (cudaError_t e_ = left_begin(P, P.R, false, st)) return e_;
    const size_t smem = packet_smem<DEG>(block);
    switch (block) {
      case 64: {
        if (cudaError_t e_ = prepare(k_trace_fwd_packet<KBUF, DEG, 64>, smem)) return e_;
        k_trace_fwd_packet<KBUF, DEG, 64><<<unsigned(grid), 64, smem, st>>>(P);
        break;
      }
      case 128: {
        if (cudaError_t e_ = prepare(k_trace_fwd_packet<KBUF, DEG, 128>, smem)) return e_;
        k_trace_fwd_packet<KBUF, DEG, 128><<<unsigned(grid), 128, smem, st>>>(P);
        break;
      }
      default: {
        if (cudaError_t e_ = prepare(k_trace_fwd_packet<KBUF, DEG, 256>, smem)) return e_;
        k_trace_fwd_packet<KBUF, DEG, 256><<<unsigned(grid), 256, smem, st>>>(P);
        break;
      }
    }
    return left_finish<KBUF, DEG, false>(P, PassCamera{}, st);
  }
  return cudaGetLastError();
}

template <int KBUF>
cudaError_t launch_k(const FwdParams& P, int deg, int block, int traversal, cudaStream_t st) {
  switch (deg) {
    case 0: return launch_t<KBUF, 0>(P, block, traversal, st);
    case 1: return launch_t<KBUF, 1>(P, block, traversal, st);
    case 2: return launch_t<KBUF, 2>(P, block, traversal, st);
    default: return launch_t<KBUF, 3>(P, block, traversal, st);
  }
}

template <int KBUF, int DEG, int BLOCK, bool CAM>
cudaError_t launch_regrouped_b(const FwdParams& P, const RegroupScratch& W, const PassCamera& Q, cudaStream_t st) {
  const int64_t n = CAM ? Q.num_slots : P.R;
  const unsigned grid = unsigned((n + BLOCK - 1) / BLOCK);
  const size_t smem = packet_smem<DEG>(BLOCK, false);
  if (cudaError_t e_ = prepare(k_trace_fwd_pass<KBUF, DEG, BLOCK, 0, CAM>, smem)) return e_;
  k_trace_fwd_pass<KBUF, DEG, BLOCK, 0, CAM><<<grid, BLOCK, smem, st>>>(P, nullptr, nullptr, W.mask0, W.split_min, Q);
  cudaError_t e = regroup_compact(W.mask0, nullptr, n, nullptr, W.offsets, W.list1, W.count1, st);
  if (e != cudaSuccess) return e;
  if (cudaError_t e_ = prepare(k_trace_fwd_pass<KBUF, DEG, BLOCK, 1, CAM>, smem)) return e_;
  k_trace_fwd_pass<KBUF, DEG, BLOCK, 1, CAM><<<grid, BLOCK, smem, st>>>(P, W.list1, W.count1, W.mask1, W.split_min, Q);
  e = regroup_compact(W.mask1, W.count1, n, W.list1, W.offsets, W.list2, W.count2, st);
  if (e != cudaSuccess) return e;
  if (cudaError_t e_ = prepare(k_trace_fwd_pass<KBUF, DEG, BLOCK, 2, CAM>, smem)) return e_;
  k_trace_fwd_pass<KBUF, DEG, BLOCK, 2, CAM><<<grid, BLOCK, smem, st>>>(P, W.list2, W.count2, nullptr, 0, Q);
  return cudaGetLastError();
}

template <int KBUF, int DEG, bool CAM>
cudaError_t launch_regrouped_t(const FwdParams& P, const RegroupScratch& W, const PassCamera& Q, int block,
                               cudaStream_t st) {
  switch (block) {
    case 64: return launch_regrouped_b<KBUF, DEG, 64, CAM>(P, W, Q, st);
    case 128: return launch_regrouped_b<KBUF, DEG, 128, CAM>(P, W, Q, st);
    default: return launch_regrouped_b<KBUF, DEG, 256, CAM>(P, W, Q, st);
  }
}

template <int KBUF, bool CAM>
cudaError_t launch_regrouped_c(const FwdParams& P, const RegroupScratch& W, const PassCamera& Q, int deg, int block,
                               cudaStream_t st) {
  switch (deg) {
    case 0: return launch_regrouped_t<KBUF, 0, CAM>(P, W, Q, block, st);
    case 1: return launch_regrouped_t<KBUF, 1, CAM>(P, W, Q, block, st);
    case 2: return launch_regrouped_t<KBUF, 2, CAM>(P, W, Q, block, st);
    default: return launch_regrouped_t<KBUF, 3, CAM>(P, W, Q, block, st);
  }
}

// cam: null for ray arrays, else the camera (its slots) and the per-pixel jitter
template <int KBUF>
cudaError_t launch_regrouped_k(const FwdParams& P, const RegroupScratch& W, const CameraParams* cam,
                               const float* jitter, int deg, int block, cudaStream_t st) {
  PassCamera Q{};
  if (!cam) return launch_regrouped_c<KBUF, false>(P, W, Q, deg, block, st);
  Q.cam = *cam;
  Q.jitter = jitter;
  Q.num_slots = camera_slots(*cam);
  return launch_regrouped_c<KBUF, true>(P, W, Q, deg, block, st);
}

template <int KBUF, int DEG>
cudaError_t launch_camera_t(const FwdParams& P0, const CameraParams& cam, const float* jitter, int block,
                            bool frustum, cudaStream_t st) {
  const int64_t num_slots = camera_slots(cam);
  if (!frustum) return launch_rounds<KBUF, DEG, true>(P0, PassCamera{cam, jitter, num_slots}, block, st);
  FwdParams P = P0;
  P.lanes = packet_lanes(num_slots);
  const unsigned grid = unsigned((num_slots + P.lanes * (block / 32) - 1) / (P.lanes * (block / 32)));
  if (cudaError_t e_ = left_begin(P, num_slots, true, st)) return e_;
  const size_t smem = packet_smem<DEG>(block);
  switch (block) {
    case 64: {
      if (cudaError_t e_ = prepare(k_trace_fwd_camera<KBUF, DEG, 64>, smem)) return e_;
      k_trace_fwd_camera<KBUF, DEG, 64><<<grid, 64, smem, st>>>(P, cam, jitter, num_slots);
      break;
    }
    case 128: {
      if (cudaError_t e_ = prepare(k_trace_fwd_camera<KBUF, DEG, 128>, smem)) return e_;
      k_trace_fwd_camera<KBUF, DEG, 128><<<grid, 128, smem, st>>>(P, cam, jitter, num_slots);
      break;
    }
    default: {
      if (cudaError_t e_ = prepare(k_trace_fwd_camera<KBUF, DEG, 256>, smem)) return e_;
      k_trace_fwd_camera<KBUF, DEG, 256><<<grid, 256, smem, st>>>(P, cam, jitter, num_slots);
      break;
    }
  }
  return left_finish<KBUF, DEG, true>(P, PassCamera{cam, jitter, num_slots}, st);
}

template <int KBUF>
cudaError_t launch_camera_k(const FwdParams& P, const CameraParams& cam, const float* jitter, int deg, int block,
                            cudaStream_t st) {
  const bool f = P.frustum != 0;
  switch (deg) {
    case 0: return launch_camera_t<KBUF, 0>(P, cam, jitter, block, f, st);
    case 1: return launch_camera_t<KBUF, 1>(P, cam, jitter, block, f, st);
    case 2: return launch_camera_t<KBUF, 2>(P, cam, jitter, block, f, st);
    default: return launch_camera_t<KBUF, 3>(P, cam, jitter, block, f, st);
  }
}

template <int KBUF, int DEG, int BLOCK, bool FRUSTUM>
cudaError_t launch_batched_b(const BatchFwdParams& P0, cudaStream_t st) {
  BatchFwdParams P = P0;
  P.lanes = FRUSTUM ? packet_lanes(P.num_slots) : 32;
  const size_t smem = packet_smem<DEG>(BLOCK, FRUSTUM);
  if (cudaError_t e_ = prepare(k_trace_fwd_batched<KBUF, DEG, BLOCK, FRUSTUM>, smem)) return e_;
  k_trace_fwd_batched<KBUF, DEG, BLOCK, FRUSTUM><<<P.grid, BLOCK, smem, st>>>(P);
  return cudaGetLastError();
}

template <int KBUF, int DEG>
cudaError_t launch_batched_t(const BatchFwdParams& P, int block, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(P.work_counter, 0, sizeof(unsigned int), st);
  if (e != cudaSuccess) return e;
  const bool f = P.frustum != 0;
  switch (block) {
    case 64: return f ? launch_batched_b<KBUF, DEG, 64, true>(P, st) : launch_batched_b<KBUF, DEG, 64, false>(P, st);
    case 128: return f ? launch_batched_b<KBUF, DEG, 128, true>(P, st) : launch_batched_b<KBUF, DEG, 128, false>(P, st);
    default: return f ? launch_batched_b<KBUF, DEG, 256, true>(P, st) : launch_batched_b<KBUF, DEG, 256, false>(P, st);
  }
}

template <int KBUF>
cudaError_t launch_batched_k(const BatchFwdParams& P, int deg, int block, cudaStream_t st) {
  switch (deg) {
    case 0: return launch_batched_t<KBUF, 0>(P, block, st);
    case 1: return launch_batched_t<KBUF, 1>(P, block, st);
    case 2: return launch_batched_t<KBUF, 2>(P, block, st);
    default: return launch_batched_t<KBUF, 3>(P, block, st);
  }
}

}  // namespace
}  // namespace ever
