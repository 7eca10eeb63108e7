// mega.cu -- the persistent render kernel: every camera sample of a render
// (or of a whole batch of renders) in ONE launch.
//
// PixelSamplerRenderer::render (src/renderer/pixel_sampler_renderer.cpp:24-109)
// calls PathTraceRenderer::eval_pixel_li (src/renderer/path_trace_renderer.cpp:27-210)
// once per camera sample, the samples of a pixel in order from one pcg32
// stream. Here a lane owns a pixel (a path slot) at a time and runs its
// samples one after another with the path state in registers; when the
// pixel's samples are done it claims the next unrendered pixel of any job
// (one atomic per warp). Each loop iteration processes one path vertex of
// every owning lane, in phases:
//
//   trace    every ray of the warp's pool: shadow rays, MIS rays and the
//            continuation or camera rays of the owners' next vertices
//   finish   the vertex's direct lighting, film updates of ended samples
//   vertex   emission, escape to the environment light, BSDF sample, the MIS
//            sample, throughput, Russian roulette, the next ray
//   lights   light samples of the warp's vertices, dealt out over all lanes
//
// All random draws of a vertex happen in its vertex phase, so the rays of its
// light samples and MIS sample and the path's next ray are independent, and
// so is the next sample's camera ray when the path ends there: they are traced
// together, any lane walking any ray, and the lights phase likewise takes
// (vertex, light) pairs from a dense list. One walk and one light evaluation
// per vertex are then on a path's serial chain instead of one per light, and
// lanes whose vertex has fewer rays do not idle.
//
// The arithmetic, the order of random draws and the order of the sums are
// those of the wavefront kernels of render.cu (k_logic, k_material, k_glass,
// k_nee, mis_contribution), so a pixel gets the same film bit for bit either
// way; only the work is arranged for small renders, where the wavefront's
// launches per path vertex over a few thousand slots cannot fill the GPU.
// Guided rendering and instrumented renders (stage times, visit counts) use
// the wavefront.

#define TRG_MATH_OUT_OF_LINE  // tr_math.cuh: this kernel holds every material's code

#include <cuda_runtime.h>

#include "mega.h"
#include "traverse.cuh"

namespace trg {

namespace {

constexpr unsigned kFull = 0xffffffffu;

// A warp's ray pool in shared memory, three float4 per ray:
//   a: origin, t_max
//   b: direction, who (owner lane | kind << 5 | light << 7 | scene << 12)
//   c: shadow rays: the light sample's contribution | the remembered occluder's
//      slot (-1: none), after the walk kBlocked | the occluding slot if blocked;
//      others, after the walk: t_attr, alpha, beta | primitive (-1: miss)
// Continuation and MIS rays lie at the front and stay for the iteration;
// shadow rays follow, walked in several rounds if they do not fit at once.
constexpr int kPool = 128;
constexpr size_t kPoolBytes = 3 * kPool * sizeof(float4);
constexpr int kBlocked = 1 << 30;
enum : int { RAY_NEXT = 0, RAY_MIS = 1, RAY_SHADOW = 2 };
__device__ __forceinline__ int who_of(int owner, int kind, int light, int scene) {
  return owner | kind << 5 | light << 7 | scene << 12;
}

// Walks rays [from, n) of the pool: the speculative while-while of
// persistent_traverse, closest-hit and any-hit rays side by side, finished
// lanes taking the next ray once fewer than kPoolRefill walk. Every lane of
// the warp calls it. Returns this lane's count of rays answered by their
// remembered occluder.
constexpr int kPoolRefill = 24;
__device__ __noinline__ unsigned int pool_trace(const DScene& sc, float4* pool, int from, int n, int cache, int* err) {
  float4 *pa = pool, *pb = pool + kPool, *pc = pool + 2 * kPool;
  const unsigned int below = (1u << (threadIdx.x & 31u)) - 1u;
  TravLane<false, false, false, true> L;
  VisitCount vc;
  bool live = false;
  int ray = -1, next = from;
  unsigned int hits = 0;
  __syncwarp();
  for (;;) {
    const unsigned int idle = __ballot_sync(kFull, !live);
    if (next < n) {
      const int mine = next + __popc(idle & below);
      next += __popc(idle);
      if (!live && mine < n) {
        ray = mine;
        const float4 a = pa[ray], b = pb[ray];
        const int who = __float_as_int(b.w), scene = who >> 12;
        const f3 o = mk3(a.x, a.y, a.z), d = mk3(b.x, b.y, b.z);
        L.any = ((who >> 5) & 3) == RAY_SHADOW;
        const float t_min = L.any ? kEps : 0.0f;
        const int oc = L.any && cache ? __float_as_int(pc[ray].w) : -1;
        if (oc >= 0 && occluded_by_slot(sc, scene, oc, o, d, t_min, a.w)) {
          pc[ray].w = __int_as_float(kBlocked | oc);
          ++hits;
        } else {
          live = L.start(sc, scene, o, d, t_min, a.w, vc, false);
          if (!live && !L.any) pc[ray] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
        }
      }
    } else if (idle == kFull) {
      break;
    }
    if (!__any_sync(kFull, live)) continue;
    for (;;) {
      for (;;) {
        if (live && L.cnt > 0 && L.pc == 0) L.postpone();
        if (!__any_sync(kFull, live && L.pc == 0)) break;
        bool ended = false;
        if (live && L.cnt == 0) {
          if (!L.interior(sc, err, vc)) {
            if (L.failed || L.pc == 0) ended = true;
            else L.cnt = -1;
          }
        }
        if (ended) {
          live = false;
          if (!L.any) pc[ray] = make_float4(L.h.t_attr, L.h.alpha, L.h.beta, __int_as_float(L.h.prim));
        }
      }
      if (live) {
        live = L.postponed_leaf(sc, vc);
        if (!live) {
          if (!L.any) pc[ray] = make_float4(L.h.t_attr, L.h.alpha, L.h.beta, __int_as_float(L.h.prim));
          else if (L.occluded) pc[ray].w = __int_as_float(kBlocked | L.h.prim);
        }
      }
      const int walking = __popc(__ballot_sync(kFull, live));
      if (walking == 0 || (walking < kPoolRefill && next < n)) break;
    }
  }
  __syncwarp();
  return hits;
}

// Material dispatch limited to the kinds of the instantiation (the sampler
// out of line: one copy serves the path's and the MIS sample).
template <unsigned MASK>
__device__ __noinline__ BsdfSample m_sample(const Bsdf& b, int kind, float u, float v, float w) {
  if ((MASK & MK_DISNEY12) && kind == MAT_DISNEY12) return b.disney_sample(u, v, w);
  if ((MASK & MK_METAL) && kind == MAT_METAL) return b.metal_sample(u, v, w);
  if ((MASK & MK_DISNEY15) && kind == MAT_DISNEY15) return b.d15_sample(u, v, w);
  return b.phong_sample_agg(u, v, w);
}
template <unsigned MASK>
__device__ __forceinline__ void m_value(const Bsdf& b, int kind, f3 wi, f3& f, float& pdf) {
  if ((MASK & MK_DISNEY12) && kind == MAT_DISNEY12) b.disney_value(wi, f, pdf);
  else if ((MASK & MK_METAL) && kind == MAT_METAL) b.metal_value(wi, f, pdf);
  else if ((MASK & MK_DISNEY15) && kind == MAT_DISNEY15) b.d15_value(wi, f, pdf);
  else b.phong_value(wi, f, pdf);
}

// The per-lane state of one pixel slot.
struct Path {
  int slot;  // -1: none
  const JobDev* J;
  unsigned long long st;
  int sample, depth, sdepth;
  bool spec;      // the ray continues a delta sample (emission it reaches counts)
  bool has_ray;   // the path has a next ray
  f3 o, d, coef, L;
  float px, py;
  unsigned int finished;
};

// start_sample of render.cu: the slot's next camera sample, finishing samples
// that Russian roulette ends before their first vertex.
__device__ __forceinline__ bool start_sample(Path& p) {
  const JobDev& J = *p.J;
  const int pix = p.slot - J.slot_base;
  const int x = pix % J.W, y = pix / J.W;
  while (p.sample < J.spp) {
    const float fu = Pcg::next(p.st), fv = Pcg::next(p.st);
    const float lu = Pcg::next(p.st), lv = Pcg::next(p.st);
    const float px = (float)x + fu, py = (float)y + fv;
    f3 o, d;
    camera_ray(J.cam, px / (float)J.W, py / (float)J.H, lu, lv, o, d);
    f3 coef = mk3(1.0f, 1.0f, 1.0f);
    bool dead = false;
    if (0 > J.min_depth) {  // Russian roulette at depth 0
      if (Pcg::next(p.st) > 0.9f) dead = true;
      else coef = divs(coef, 0.9f);
    }
    if (!dead && !valid3(coef)) dead = true;
    if (dead) {
      film_add(J, p.slot, px, py, mk3(0.0f, 0.0f, 0.0f));
      ++p.finished;
      ++p.sample;
      continue;
    }
    p.o = o;
    p.d = d;
    p.coef = coef;
    p.L = mk3(0.0f, 0.0f, 0.0f);
    p.px = px;
    p.py = py;
    p.depth = 0;
    p.sdepth = 0;
    p.spec = false;
    return true;
  }
  return false;
}

__device__ __forceinline__ f3 film_value(f3 L) {
  return valid3(L) ? L : mk3(0.0f, 0.0f, 0.0f);  // eval_pixel_li returns {} (path_trace_renderer.cpp:204-209)
}

__device__ __forceinline__ f3 shfl3(f3 v, int src) {
  return mk3(__shfl_sync(kFull, v.x, src), __shfl_sync(kFull, v.y, src), __shfl_sync(kFull, v.z, src));
}
__device__ __forceinline__ unsigned long long shfl64(unsigned long long v, int src) {
  const unsigned int lo = __shfl_sync(kFull, (unsigned int)v, src), hi = __shfl_sync(kFull, (unsigned int)(v >> 32), src);
  return (unsigned long long)hi << 32 | lo;
}

// One (vertex, light) pair (k_nee): the light sample of light `l` at pos, its
// contribution cc and shadow ray sd, dist. Returns whether there is one.
template <unsigned MASK>
__device__ __forceinline__ bool light_item(const DScene& sc, const DLight& lt, const Bsdf& bsdf, int kind, f3 pos,
                                           f3 coef, float2 uv, f3& cc, f3& sd, float& dist) {
  f3 to_light, Le;
  float lpdf;
  if ((MASK & MK_ENV) && lt.env >= 0) {
    // sample_environment_light (src/renderer/direct_illumination.cpp:73-106)
    f3 lpos;
    if (!env_sample(sc.envs[lt.env], pos, uv.x, uv.y, Le, lpdf, lpos) || black(Le)) return false;
    to_light = lpos - pos;
  } else {
    // sample_area_light (src/renderer/direct_illumination.cpp:35-71) via
    // UniformSampleTriangle (src/shape/triangle.cpp:61-97)
    const float su0 = sqrtf(uv.x);
    const float bx = 1.0f - su0, by = uv.y * su0;
    const f3 lpos = scale(lt.A, bx) + scale(lt.B, by) + scale(lt.C, 1.0f - bx - by);
    const f3 sp2ref = pos - lpos;
    if (!(dot(lt.gz, sp2ref) > 0.0f)) return false;
    const float dist2 = len2f(sp2ref);
    lpdf = area_to_solid_pdf(lt.area_pdf * dist2, dot(lt.gz, sp2ref), dist2);
    if (!lpdf) return false;
    to_light = lpos - pos;
    Le = lt.emission;
  }
  bool too_close;
  dist = dist_minus_eps(len2f(to_light), too_close);
  if (too_close) return false;
  to_light = normalize(to_light);
  f3 bf;
  float bpdf;
  m_value<MASK>(bsdf, kind, to_light, bf, bpdf);
  if (black(bf)) return false;
  const f3 fl = muls(mulc(Le, bf), abs_cos(to_light, bsdf.g.z));
  const float w = power_heuristic(lpdf, bpdf);
  cc = mulc(coef, divs(muls(fl, w), lpdf));
  sd = normalize(to_light);
  return true;
}

template <unsigned MASK, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) k_mega(MegaLaunch P) {
  extern __shared__ float4 pools[];
  const DScene& sc = P.sc;
  const int lane = (int)(threadIdx.x & 31u);
  const unsigned int below = (1u << lane) - 1u;
  float4* pool = pools + (threadIdx.x >> 5) * (3 * kPool);
  float4 *pa = pool, *pb = pool + kPool, *pc = pool + 2 * kPool;
  DMat* const tmat = (MASK & MK_MAPS) ? P.mt + (size_t)blockIdx.x * blockDim.x + threadIdx.x : nullptr;
  Path p;
  p.slot = -1;
  p.has_ray = false;
  p.finished = 0;
  bool done = lane >= P.lanes;
  long long steps = 0, max_steps = 0;  // vertex bound of the current pixel
  int oc[kMegaLights];                 // the slot that last blocked each light's shadow ray (-1: none)
  bool claimed = false;                // a pixel claimed in this iteration: oc is to be cleared
  unsigned long long n_ext = 0, n_sh = 0, n_vert = 0, n_hits = 0;
  // the vertex whose light is being gathered: what its light samples need,
  // its MIS ray, and the sample that ends with it (its film update is due
  // once its direct lighting is known)
  Isect is;
  Bsdf bsdf;
  int kind = 0, mcode = 0, scene = 0, light_base = 0, env = -1;
  unsigned int nee_mask = 0;
  unsigned long long st_lights = 0;  // the stream before the light samples' draws
  f3 coef_prev = mk3(0.0f, 0.0f, 0.0f), mo = coef_prev, md = coef_prev, mf = coef_prev;
  float mpdf = 0.0f, mcos = 0.0f;
  bool vertex = false, mis = false, mis_trace = false;
  bool due = false, restart = false;  // a film update is due; the next sample starts after it
  f3 due_L = coef_prev;
  float due_x = 0.0f, due_y = 0.0f;
  int due_slot = 0;
  const JobDev* due_J = nullptr;
  for (;;) {
    // owners without a ray claim pixels until they have one or none are left
    for (;;) {
      const bool want = !done && !p.has_ray && !restart;
      const unsigned need = __ballot_sync(kFull, want);
      if (!need) break;
      const int leader = __ffs(need) - 1;
      unsigned int base = 0;
      if (lane == leader) base = atomicAdd(P.fetch, (unsigned int)__popc(need));
      base = __shfl_sync(kFull, base, leader);
      if (want) {
        const unsigned int s = base + (unsigned int)__popc(need & below);
        if (s < (unsigned int)P.nslots) {
          p.slot = (int)s;
          p.J = &job_of(P.jobs, P.njobs, p.slot);
          const int pix = p.slot - p.J->slot_base;
          const int x = pix % p.J->W, y = pix / p.J->W;
          p.st = Pcg::seed((int)(p.J->seed_base + (unsigned)y * (unsigned)p.J->W + (unsigned)x));
          p.sample = 0;
          claimed = true;
          steps = 0;
          max_steps = (long long)p.J->spp * ((long long)p.J->max_depth + 2 + ((MASK & MK_GLASS) ? kMaxSpecularDepth : 0));
          p.has_ray = start_sample(p);
        } else {
          done = true;
        }
      }
    }
    // the pool's front: the owners' next rays, then their MIS rays
    const unsigned int m_next = __ballot_sync(kFull, p.has_ray), m_mis = __ballot_sync(kFull, mis_trace);
    const int i_next = __popc(m_next & below), i_mis = __popc(m_next) + __popc(m_mis & below);
    const int front = __popc(m_next) + __popc(m_mis);
    if (p.has_ray) {
      pa[i_next] = make_float4(p.o.x, p.o.y, p.o.z, kRealMax);
      pb[i_next] = make_float4(p.d.x, p.d.y, p.d.z, __int_as_float(who_of(lane, RAY_NEXT, 0, p.J->scene)));
    }
    if (mis_trace) {
      pa[i_mis] = make_float4(mo.x, mo.y, mo.z, kRealMax);
      pb[i_mis] = make_float4(md.x, md.y, md.z, __int_as_float(who_of(lane, RAY_MIS, 0, scene)));
    }
    n_ext += (p.has_ray ? 1 : 0) + (mis_trace ? 1 : 0);
    // the block goes through the phases together: one phase's code in the
    // instruction cache at a time (free-running warps took 2.8 times as long
    // on a 256x256x16 Cornell box)
    __syncthreads();

    // ---- lights: the (vertex, light) pairs of the warp, 32 at a time
    f3 direct = mk3(0.0f, 0.0f, 0.0f);
    int n_items = __popc(nee_mask), first_item = n_items;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(kFull, first_item, off);
      if (lane >= off) first_item += y;
    }
    const int items = __shfl_sync(kFull, first_item, 31);
    first_item -= n_items;
    int n = front, traced = 0, mine = 0, n_mine = 0;  // mine, n_mine: this owner's shadow rays in the pool
    for (int c0 = 0;; c0 += 32) {
      bool ray = false;
      f3 cc, sd, pos;
      float dist = 0.0f;
      int owner = 0, l = 0, osc = 0;
      if (c0 < items) {
        // lane k takes pair c0 + k; its owner is the last lane whose pairs
        // start at or before it (a lane without pairs starts where the next does)
        const int it = c0 + lane;
        for (int step = 16; step > 0; step >>= 1)
          if (__shfl_sync(kFull, first_item, owner + step) <= it) owner += step;
        const int start = __shfl_sync(kFull, first_item, owner);
        unsigned int mask = __shfl_sync(kFull, nee_mask, owner);
        const bool on = it < items;
        for (int k = it - start; on && k > 0; --k) mask &= mask - 1u;
        l = on ? __ffs((int)mask) - 1 : 0;
        unsigned long long st = shfl64(st_lights, owner);
        pos = shfl3(is.pos, owner);
        Bsdf b;
        b.g.x = shfl3(bsdf.g.x, owner);
        b.g.y = shfl3(bsdf.g.y, owner);
        b.g.z = shfl3(bsdf.g.z, owner);
        b.s.x = shfl3(bsdf.s.x, owner);
        b.s.y = shfl3(bsdf.s.y, owner);
        b.s.z = shfl3(bsdf.s.z, owner);
        b.lwo = shfl3(bsdf.lwo, owner);
        const int bits = __shfl_sync(kFull, (bsdf.wo_g ? 1 : 0) | (bsdf.wo_fr ? 2 : 0) | (bsdf.same_n ? 4 : 0) | kind << 3, owner);
        b.wo_g = bits & 1;
        b.wo_fr = bits & 2;
        b.same_n = bits & 4;
        const int mc = __shfl_sync(kFull, mcode, owner);
        const f3 coef = shfl3(coef_prev, owner);
        const int lb = __shfl_sync(kFull, light_base, owner);
        osc = __shfl_sync(kFull, scene, owner);
        if (on) {
          b.m = (MASK & MK_MAPS) && mc < 0 ? tmat + (owner - lane) : sc.mats + mc;
          for (int k = 0; k < l; ++k) Pcg::skip<5>(st);  // five draws a light, the first two place the sample
          const float u = Pcg::next(st), v = Pcg::next(st);
          ray = light_item<MASK>(sc, sc.lights[lb + l], b, bits >> 3, pos, coef, make_float2(u, v), cc, sd, dist);
        }
      }
      const unsigned int m_ray = __ballot_sync(kFull, ray);
      n_sh += ray;
      if (ray) {
        const int e = n + __popc(m_ray & below);
        pa[e] = make_float4(pos.x, pos.y, pos.z, dist);
        pb[e] = make_float4(sd.x, sd.y, sd.z, __int_as_float(who_of(owner, RAY_SHADOW, l, osc)));
        pc[e] = make_float4(cc.x, cc.y, cc.z, __int_as_float(-1));
      }
      __syncwarp();
      {
        // the owner's share of this round: pairs [lo, hi) of the chunk
        const int lo = min(max(first_item - c0, 0), 32), hi = min(max(first_item + n_items - c0, 0), 32);
        const unsigned int below_lo = lo >= 32 ? kFull : (1u << lo) - 1u, below_hi = hi >= 32 ? kFull : (1u << hi) - 1u;
        if (n_mine == 0) mine = n + __popc(m_ray & below_lo);
        const int k0 = n + __popc(m_ray & below_lo), k1 = n + __popc(m_ray & below_hi);
        for (int e = k0; e < k1; ++e)  // the light's last occluder is the owner's to know
          pc[e].w = __int_as_float(oc[(__float_as_int(pb[e].w) >> 7) & 31]);
        n_mine += k1 - k0;
      }
      n += __popc(m_ray);
      // the last round, or a full pool: walk it and add the shadow rays' answers
      const bool more = c0 + 32 < items;
      if (!more || n + 32 > kPool) {
        if (!more) __syncthreads();
        // ---- trace (k_extend, k_shadow)
        n_hits += pool_trace(sc, pool, traced, n, P.occluder_cache && sc.slot_leaf, P.err);
        for (int e = mine; e < mine + n_mine; ++e) {
          const float4 c = pc[e];
          const int w = __float_as_int(c.w);
          if (w >= 0 && (w & kBlocked)) oc[(__float_as_int(pb[e].w) >> 7) & 31] = w & ~kBlocked;
          else direct = direct + mk3(c.x, c.y, c.z);
        }
        __syncwarp();
        n = traced = front;
        n_mine = 0;
      }
      if (!more) break;
    }

    // a new pixel, which may be another scene's, starts without occluders; until
    // here they were those of the pixel before, whose last vertex was gathered
    if (claimed) {
      for (int l = 0; l < kMegaLights; ++l) oc[l] = -1;
      claimed = false;
    }

    // ---- finish: the MIS ray's emission, weighted against the light
    //      (mis_contribution of render.cu, direct_illumination.cpp:144-198), the
    //      vertex's direct lighting, the film update of a sample that ended
    if (mis) {
      float4 mh = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
      if (mis_trace) mh = pc[i_mis];  // a ray that can reach no light is not traced: its closest hit would give zero
      const int pid = __float_as_int(mh.w);
      f3 c = mk3(0.0f, 0.0f, 0.0f);
      if (pid < 0) {
        if ((MASK & MK_ENV) && env >= 0) {
          const DEnv& e = sc.envs[env];
          const f3 Le = env_emit(e, md);
          if (!black(Le)) {
            const f3 f = muls(mulc(Le, mf), mcos);
            const float w = power_heuristic(mpdf, env_pdf(e, md));
            c = divs(muls(f, w), mpdf);
          }
        }
      } else {
        const DPrim& pr = sc.prims[pid];
        if (pr.emissive) {
          const f3 gz = sc.tshade[pr.shape].gz;
          if (dot(gz, -md) > 0.0f) {
            const f3 f = muls(mulc(pr.emission, mf), mcos);
            const f3 pos = mo + scale(md, mh.x);
            const float lpdf = light_pdf_at(pr.area, mo, pos, gz);
            const float w = power_heuristic(mpdf, lpdf);
            c = divs(muls(f, w), mpdf);
          }
        }
      }
      direct = direct + mulc(coef_prev, c);
    }
    if (vertex) {
      if (due) film_add(*due_J, due_slot, due_x, due_y, film_value(due_L + direct));
      else p.L = p.L + direct;
    }
    vertex = mis = mis_trace = due = false;
    nee_mask = 0;
    float4 hit = make_float4(__int_as_float(-1), 0.0f, 0.0f, 0.0f);
    const bool arrived = p.has_ray;  // the next ray's hit is known
    if (arrived) {
      const float4 c = pc[i_next];
      hit = make_float4(c.w, c.x, c.y, c.z);
    }
    if (restart) {
      restart = false;
      p.has_ray = start_sample(p);
    }
    if (!__syncthreads_or(arrived || p.has_ray || !done)) break;

    // ---- vertex (k_logic, then k_material / k_glass)
    if (arrived) {
      bool ended = false;  // the sample ended at this hit without direct lighting
      bool term = false;
      ++n_vert;
      p.has_ray = false;
      if (++steps > max_steps) {
        atomicOr(P.err, 2);
        p.slot = -1;
      } else {
        const int pid = __float_as_int(hit.x);
        if (pid < 0) {
          // a camera ray or one after a delta sample left the scene: the
          // environment light's radiance along it (path_trace_renderer.cpp:66-81)
          if ((MASK & MK_ENV) && (p.depth == 0 || p.spec) && p.J->env >= 0)
            p.L = p.L + mulc(p.coef, env_emit(sc.envs[p.J->env], p.d));
          ended = true;
        } else {
          const DPrim& pr = sc.prims[pid];
          if ((p.depth == 0 || p.spec) && pr.emissive) {
            // emission seen by the camera ray or after a delta sample
            const f3 gz = sc.tshade[pr.shape].gz;
            if (dot(gz, -p.d) > 0.0f) p.L = p.L + mulc(p.coef, pr.emission);
          }
          kind = sc.mats[pr.material].kind;
          make_isect(sc, hit, p.o, p.d, is);
          mcode = pr.material;
          bsdf.m = sc.mats + mcode;
          if ((MASK & MK_MAPS) && bsdf.m->tex_any) {  // image maps: the material at this hit's uv
            float u, v;
            hit_uv(sc, hit, p.o, p.d, u, v);
            material_at(sc, pr.material, u, v, tmat);
            bsdf.m = tmat;
            mcode = -1;
          }
          bsdf.g = is.g;
          bsdf.s = is.s;
          bsdf.look_from(is.wo);
          if ((MASK & MK_GLASS) && kind == MAT_GLASS) {
            // k_glass: a delta sample, no direct lighting
            const float u0 = Pcg::next(p.st);
            Pcg::skip<2>(p.st);  // the rest of sample3()
            const BsdfSample bs = bsdf.glass_sample(u0);
            bool t = black(bs.f) || bs.pdf < kEps;
            if (!t) {
              const bool counted = p.sdepth >= kMaxSpecularDepth;
              if (!counted) ++p.sdepth;
              p.coef = mulc(p.coef, divs(muls(bs.f, abs_cos(is.g.z, bs.wi)), bs.pdf));
              t = !valid3(p.coef);
              if (!t) {
                if (counted) ++p.depth;
                if (p.depth >= p.J->max_depth) {
                  t = true;
                } else if (p.depth > p.J->min_depth) {
                  if (Pcg::next(p.st) > 0.9f) t = true;
                  else {
                    p.coef = divs(p.coef, 0.9f);
                    if (!valid3(p.coef)) t = true;
                  }
                }
              }
            }
            if (t) {
              ended = true;
            } else {
              p.o = is.eps_offset(bs.wi);
              p.d = normalize(normalize(bs.wi));
              p.spec = true;
              p.has_ray = true;
            }
          } else {
            const float u0 = Pcg::next(p.st), u1 = Pcg::next(p.st), u2 = Pcg::next(p.st);
            const BsdfSample bs = m_sample<MASK>(bsdf, kind, u0, u1, u2);
            if (black(bs.f) || bs.pdf < kEps) {
              ended = true;
            } else {
              vertex = true;
              // next-event estimation draws on every light (sample_area_light):
              // five each, taken in the lights phase from here on
              const JobDev& J = *p.J;
              st_lights = p.st;
              scene = J.scene;
              light_base = J.light_base;
              env = J.env;
              const float pos_mag = fabsf(is.pos.x) + fabsf(is.pos.y) + fabsf(is.pos.z);
              for (int l = 0; l < J.nl; ++l) {
                // a vertex well behind a light's plane gets nothing from it
                // (k_material's skip)
                const DLight& lt = sc.lights[J.light_base + l];
                const float side = dot(lt.gz, is.pos - lt.A);
                const float tol = 1e-4f * (pos_mag + lt.extent);
                Pcg::skip<5>(p.st);
                if (!(side < -tol)) nee_mask |= 1u << l;
              }
              // the MIS BSDF ray (sample_bsdf, src/renderer/direct_illumination.cpp:144-155)
              const float v0 = Pcg::next(p.st), v1 = Pcg::next(p.st), v2 = Pcg::next(p.st);
              const BsdfSample ms = m_sample<MASK>(bsdf, kind, v0, v1, v2);
              if (ms.valid()) {
                const f3 wi = normalize(ms.wi);
                mo = is.eps_offset(wi);
                md = normalize(wi);
                mpdf = ms.pdf;
                mcos = abs_cos(is.g.z, md);
                mf = ms.f;
                mis = true;
                mis_trace = mis_may_hit_light(sc, J, mo, md);
              }
              coef_prev = p.coef;
              p.coef = mulc(p.coef, divs(muls(bs.f, abs_cos(is.g.z, bs.wi)), bs.pdf));
              term = !valid3(p.coef);
              if (!term) {
                ++p.depth;
                if (p.depth >= J.max_depth) {
                  term = true;
                } else if (p.depth > J.min_depth) {
                  if (Pcg::next(p.st) > 0.9f) term = true;
                  else {
                    p.coef = divs(p.coef, 0.9f);
                    if (!valid3(p.coef)) term = true;
                  }
                }
              }
              if (!term) {
                p.o = is.eps_offset(bs.wi);
                p.d = normalize(normalize(bs.wi));
                p.spec = false;
                p.has_ray = true;
              }
            }
          }
        }
        if (ended || term) {
          // the sample is over: its film update, now or once its direct
          // lighting is known, and the pixel's next sample (samples that end
          // before their first vertex, min_depth below 0, update the film as
          // they start: they wait for the update that is due)
          if (ended) film_add(*p.J, p.slot, p.px, p.py, film_value(p.L));
          due = term;
          due_L = p.L;
          due_x = p.px;
          due_y = p.py;
          due_slot = p.slot;
          due_J = p.J;
          ++p.finished;
          ++p.sample;
          restart = due && p.J->min_depth < 0;
          if (!restart) p.has_ray = start_sample(p);
        }
      }
    }
  }
  // statistics (warp sums, one atomic per warp)
  const unsigned long long sums[5] = {p.finished, n_ext, n_sh, n_vert, n_hits};
  const int where[5] = {0, 1, 2, 3, 8};
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    unsigned long long v = sums[k];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(kFull, v, off);
    if (lane == 0 && v) atomicAdd(P.stats + where[k], v);
  }
}

constexpr unsigned kMaskPhong = MK_PHONG;
constexpr unsigned kMaskPD = MK_PHONG | MK_DISNEY12;
constexpr unsigned kMaskAll = MK_PHONG | MK_DISNEY12 | MK_GLASS | MK_METAL | MK_DISNEY15 | MK_ENV | MK_MAPS;

template <unsigned MASK, int THREADS>
cudaError_t launch(const MegaLaunch& P, int grid, cudaStream_t st) {
  constexpr size_t smem = (size_t)(THREADS / 32) * kPoolBytes;
  const cudaError_t e = cudaFuncSetAttribute((const void*)k_mega<MASK, THREADS>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_mega<MASK, THREADS><<<grid, THREADS, smem, st>>>(P);
  return cudaGetLastError();
}

template <int THREADS>
cudaError_t launch(const MegaLaunch& P, unsigned mask, int grid, cudaStream_t st) {
  if (mask == kMaskPhong) return launch<kMaskPhong, THREADS>(P, grid, st);
  if (mask == kMaskPD) return launch<kMaskPD, THREADS>(P, grid, st);
  return launch<kMaskAll, THREADS>(P, grid, st);
}

}  // namespace

unsigned mega_kernel_mask(const DScene& sc, bool has_disney12) {
  if (sc.has_glass || sc.has_metal || sc.has_disney15 || sc.has_env || sc.has_textures) return kMaskAll;
  return has_disney12 ? kMaskPD : kMaskPhong;
}

cudaError_t launch_mega(const MegaLaunch& P, unsigned mask, const MegaShape& shape, cudaStream_t st) {
  return shape.threads == kMegaFewThreads ? launch<kMegaFewThreads>(P, mask, shape.grid, st)
                                          : launch<kMegaThreads>(P, mask, shape.grid, st);
}

}  // namespace trg
