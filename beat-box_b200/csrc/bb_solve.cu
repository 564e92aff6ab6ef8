// bb_solve.cu -- PGS_SOFT and AVBD contact solvers.
//
// Reference: PGS_SOFT::pre_step / solve (src/shaders/simulation/solvers.slang:142-279) run
// per colour (RB_sim.slang:1408-1578) in the order of RBM:1369-1389 (pre-step, I solve sweeps,
// integrate positions RB_sim.slang:1287-1326, I relax sweeps), each sweep colours 0..31 then
// the serial overflow bucket.  AVBD (src/shaders/simulation/avbd.slang): body colouring
// (:812-981), prepare (:70-128), warm start (:390-473), support depth (:667-724), primal
// (:478-658) with the 6x6 LDL^T of avbd_solve6 (:329-387), dual (:728-808), finalize
// (:132-202), post-stabilisation sweeps (RBM:1400-1425).
//
// B200 design: each solver phase is ONE persistent cooperative kernel that walks compact
// colour buckets, instead of the reference's (2I+1) x 33 dispatches that each scan every
// manifold and filter by colour.  The PGS_SOFT sweeps order the updates of a body by a tag in its
// velocity words; the AVBD sweeps separate colours with a grid barrier.  The 6x6 block solve
// stays in registers.
#include "bb_common.cuh"
#include <algorithm>

#include "bb_kernels.cuh"

// ---------------------------------------------------------------------------------------
// PGS_SOFT
__device__ __forceinline__ Sym3 load_iw(const DevState& d, uint32_t i) {
  float4 a = d.iw[2 * i], b = d.iw[2 * i + 1];
  return Sym3{a.x, a.y, a.z, a.w, b.x, b.y};
}
__device__ __forceinline__ bool awake(uint32_t f) { return (f & BB_BODY_DYNAMIC) && !(f & BB_BODY_SLEEPING); }

// Quaternion integration (extensions.slang:148-166)
__device__ __forceinline__ Quatf apply_angular_velocity(Quatf rot, float3 w, float dt) {
  float angle = len3(w) * dt;
  Quatf q;
  if (angle > 0.0001f) {
    float3 axis = w * (1.0f / len3(w));
    float half = angle / 2.0f;
    float sh, ch;
    sincosf(half, &sh, &ch);
    q = Quatf{axis.x * sh, axis.y * sh, axis.z * sh, ch};
  } else {
    float3 dr = w * dt * 0.5f;
    q = Quatf{dr.x, dr.y, dr.z, 1.0f};
  }
  return q_normalize(q_mul(q, rot));
}

// ---- PGS_SOFT arithmetic of one contact ---------------------------------------------------

// Every operation below is an explicitly rounded intrinsic (fma where a product feeds a sum),
// so the compiler has nothing left to contract: each inlined copy of this arithmetic produces
// the same bits.
__device__ __forceinline__ float3 xadd(float3 a, float3 b) {
  return make_float3(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z));
}
__device__ __forceinline__ float3 xsub(float3 a, float3 b) {
  return make_float3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z));
}
__device__ __forceinline__ float3 xscale(float3 a, float s) {
  return make_float3(__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s));
}
__device__ __forceinline__ float3 xaxpy(float3 a, float s, float3 y) {  // a * s + y
  return make_float3(__fmaf_rn(a.x, s, y.x), __fmaf_rn(a.y, s, y.y), __fmaf_rn(a.z, s, y.z));
}
__device__ __forceinline__ float xdot(float3 a, float3 b) {
  return __fmaf_rn(a.z, b.z, __fmaf_rn(a.y, b.y, __fmul_rn(a.x, b.x)));
}
__device__ __forceinline__ float3 xcross(float3 a, float3 b) {
  return make_float3(__fmaf_rn(a.y, b.z, -__fmul_rn(a.z, b.y)), __fmaf_rn(a.z, b.x, -__fmul_rn(a.x, b.z)),
                     __fmaf_rn(a.x, b.y, -__fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float3 xsym(const Sym3& s, float3 v) {
  return make_float3(__fmaf_rn(s.xz, v.z, __fmaf_rn(s.xy, v.y, __fmul_rn(s.xx, v.x))),
                     __fmaf_rn(s.yz, v.z, __fmaf_rn(s.yy, v.y, __fmul_rn(s.xy, v.x))),
                     __fmaf_rn(s.zz, v.z, __fmaf_rn(s.yz, v.y, __fmul_rn(s.xz, v.x))));
}
// v_a -= P m_a, w_a -= I_a (r1 x P), v_b += P m_b, w_b += I_b (r2 x P)
__device__ __forceinline__ void xapply(float3 P, float3 r1, float3 r2, float ima, float imb, const Sym3& IA,
                                       const Sym3& IB, float3& va, float3& wa, float3& vb, float3& wb) {
  va = xaxpy(P, -ima, va);
  wa = xsub(wa, xsym(IA, xcross(r1, P)));
  vb = xaxpy(P, imb, vb);
  wb = xadd(wb, xsym(IB, xcross(r2, P)));
}

// soft-constraint coefficients of a manifold (solvers.slang:150-158)
struct SoftCoef {
  float bf, mcoef, icoef, inv_h;
};
__device__ __forceinline__ SoftCoef pgs_soft_coef(float ima, float imb, float h, float hertz) {
  const float ch = (ima == 0.f || imb == 0.f) ? __fmul_rn(2.0f, hertz) : hertz;
  const float zeta = 10.0f;
  const float omega = __fmul_rn(2.0f * 3.14159265359f, ch);
  const float ho = __fmul_rn(h, omega);
  const float den = __fadd_rn(2.0f * zeta, ho);
  const float c = __fmul_rn(ho, den);
  SoftCoef s;
  s.bf = __fdiv_rn(omega, den);
  s.icoef = __fdiv_rn(1.0f, __fadd_rn(1.0f, c));
  s.mcoef = __fmul_rn(c, s.icoef);
  s.inv_h = h > 0.f ? __fdiv_rn(1.0f, h) : 0.f;
  return s;
}

// effective mass of one row along direction u: 1 / (m_a + m_b + (r1 x u) I_a (r1 x u) + ...)
__device__ __forceinline__ float xrow_mass(float3 r1, float3 r2, float3 u, float ima, float imb, const Sym3& IA,
                                           const Sym3& IB) {
  const float3 c1 = xcross(r1, u), c2 = xcross(r2, u);
  const float k = __fadd_rn(__fadd_rn(__fadd_rn(ima, imb), xdot(c1, xsym(IA, c1))), xdot(c2, xsym(IB, c2)));
  return k == 0.f ? 0.f : __fdiv_rn(1.0f, k);
}

// rows of one contact (solvers.slang:160-190): R1 = (r1, normal mass), R2 = (r2, tangent
// mass 0), K = (tangent mass 1, bias, mass coefficient, impulse coefficient)
__device__ __forceinline__ void pgs_contact_rows(float4 pp, float3 aa, float3 ab, float3 n, float3 t0, float3 t1,
                                                 float ima, float imb, const Sym3& IA, const Sym3& IB,
                                                 const SoftCoef& s, float4& R1, float4& R2, float4& K) {
  const float3 r1 = xsub(f3(pp), aa), r2 = xsub(f3(pp), ab);
  const float nmass = xrow_mass(r1, r2, n, ima, imb, IA, IB);
  const float tm0 = xrow_mass(r1, r2, t0, ima, imb, IA, IB);
  const float tm1 = xrow_mass(r1, r2, t1, ima, imb, IA, IB);
  const float pen = pp.w;
  const float bias_value = pen > 0.f ? __fmul_rn(pen, s.inv_h) : fmaxf(__fmul_rn(s.bf, pen), -4.0f);
  R1 = f4(r1, nmass);
  R2 = f4(r2, tm0);
  K = make_float4(tm1, bias_value, s.mcoef, s.icoef);
}

// warm start of one contact: apply the accumulated impulse (solvers.slang:191-195)
__device__ __forceinline__ void pgs_contact_warm(float3 r1, float3 r2, float4 lam, float3 n, float3 t0, float3 t1,
                                                 bool fric, float ima, float imb, const Sym3& IA, const Sym3& IB,
                                                 float3& va, float3& wa, float3& vb, float3& wb) {
  float3 P = xscale(n, lam.x);
  if (fric) P = xaxpy(t1, lam.z, xaxpy(t0, lam.y, P));
  xapply(P, r1, r2, ima, imb, IA, IB, va, wa, vb, wb);
}

// relative velocity at the contact: (v_b + w_b x r2) - (v_a + w_a x r1)
__device__ __forceinline__ float3 xrel(float3 r1, float3 r2, float3 va, float3 wa, float3 vb, float3 wb) {
  return xsub(xadd(vb, xcross(wb, r2)), xadd(va, xcross(wa, r1)));
}

// one contact of PGS_SOFT::solve (solvers.slang:209-277): two friction rows, then the normal row.
// Both friction rows take their impulse from the same relative velocity (computed once, before
// either is applied, as the reference does), so their two impulses are applied as one sum: the
// same result up to rounding, with one body update instead of two.
__device__ __forceinline__ void pgs_contact_solve(float4 R1, float4 R2, float4 K, float4& lam, float3 n, float3 t0,
                                                  float3 t1, float mu, bool use_bias, bool accum, bool fric, float ima,
                                                  float imb, const Sym3& IA, const Sym3& IB, float3& va, float3& wa,
                                                  float3& vb, float3& wb) {
  const float3 r1 = f3(R1), r2 = f3(R2);
  if (fric) {
    const float3 rv = xrel(r1, r2, va, wa, vb, wb);
    float imp_t[2] = {lam.y, lam.z}, ti[2];
    const float tmass[2] = {R2.w, K.x};
    const float maxf = __fmul_rn(mu, lam.x);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float3 t = k == 0 ? t0 : t1;
      ti[k] = __fmul_rn(tmass[k], -xdot(rv, t));
      if (accum) {
        const float old = imp_t[k];
        imp_t[k] = fminf(fmaxf(__fadd_rn(old, ti[k]), -maxf), maxf);
        ti[k] = __fsub_rn(imp_t[k], old);
      } else {
        ti[k] = fminf(fmaxf(ti[k], -maxf), maxf);
      }
    }
    xapply(xaxpy(t1, ti[1], xscale(t0, ti[0])), r1, r2, ima, imb, IA, IB, va, wa, vb, wb);
    lam.y = imp_t[0];
    lam.z = imp_t[1];
  }
  const float vn = xdot(xrel(r1, r2, va, wa, vb, wb), n);
  float bias = 0.f, ms = 1.f, is = 0.f;
  if (K.y > 0.f) {
    bias = K.y;
  } else if (use_bias) {
    bias = K.y;
    ms = K.z;
    is = K.w;
  }
  float imp = __fsub_rn(__fmul_rn(__fmul_rn(-R1.w, ms), __fadd_rn(vn, bias)), __fmul_rn(is, lam.x));
  if (accum) {
    const float old = lam.x;
    lam.x = fmaxf(__fadd_rn(old, imp), 0.f);
    imp = __fsub_rn(lam.x, old);
  } else {
    imp = fmaxf(imp, 0.f);
  }
  xapply(xscale(n, imp), r1, r2, ima, imb, IA, IB, va, wa, vb, wb);
}

// PGS_SOFT::pre_step (solvers.slang:143-196) of one manifold slot: rows, then warm start
__device__ void pgs_pre_step_slot(const DevState& d, const Params& p, int cur, uint32_t slot, uint2 b, float h,
                                  float hertz) {
  const uint32_t fa = d.flags[b.x], fb = d.flags[b.y];
  if (!awake(fa) && !awake(fb)) return;
  const float ima = d.pos[b.x].w, imb = d.pos[b.y].w;
  const Sym3 IA = load_iw(d, b.x), IB = load_iw(d, b.y);
  float3 va = f3(d.vel[b.x]), wa = f3(d.omega[b.x]), vb = f3(d.vel[b.y]), wb = f3(d.omega[b.y]);
  const float3 n = f3(d.m_normal[cur][slot]);
  const float3 t0 = f3(d.m_t0[cur][slot]), t1 = f3(d.m_t1[cur][slot]);
  const float3 aa = f3(d.m_anchor_a[cur][slot]), ab = f3(d.m_anchor_b[cur][slot]);
  const int cc = d.m_keycc[cur][slot].y;
  const bool accum = p.flags & BB_SIM_ACCUM_IMPULSE, fric = p.flags & BB_SIM_FRICTION;
  const SoftCoef s = pgs_soft_coef(ima, imb, h, hertz);
  for (int j = 0; j < cc; ++j) {
    const uint32_t ci = slot * BB_MAX_CONTACTS + j;
    float4 R1, R2, K;
    pgs_contact_rows(d.c_pos[cur][ci], aa, ab, n, t0, t1, ima, imb, IA, IB, s, R1, R2, K);
    d.c_r1[ci] = R1;
    d.c_r2[ci] = R2;
    d.c_k[ci] = K;
    float4 lam = d.c_lam[cur][ci];
    // the reference writes its mass coefficient / tangent masses into the persistent contact
    d.c_lam[cur][ci] = make_float4(lam.x, lam.y, lam.z, s.mcoef);
    float4 kt4 = d.c_kt[cur][ci];
    d.c_kt[cur][ci] = make_float4(R2.w, K.x, kt4.z, kt4.w);
    if (accum) pgs_contact_warm(f3(R1), f3(R2), lam, n, t0, t1, fric, ima, imb, IA, IB, va, wa, vb, wb);
  }
  if (fa & BB_BODY_DYNAMIC) {
    d.vel[b.x] = f4(va, d.vel[b.x].w);
    d.omega[b.x] = f4(wa, 0.f);
  }
  if (fb & BB_BODY_DYNAMIC) {
    d.vel[b.y] = f4(vb, d.vel[b.y].w);
    d.omega[b.y] = f4(wb, 0.f);
  }
}

// PGS_SOFT::solve (solvers.slang:199-278) of one manifold slot
__device__ void pgs_solve_slot(const DevState& d, const Params& p, int cur, uint32_t slot, uint2 b, bool use_bias) {
  const uint32_t fa = d.flags[b.x], fb = d.flags[b.y];
  if (!awake(fa) && !awake(fb)) return;
  const float ima = d.pos[b.x].w, imb = d.pos[b.y].w;
  const Sym3 IA = load_iw(d, b.x), IB = load_iw(d, b.y);
  float4 va4 = d.vel[b.x], vb4 = d.vel[b.y];
  float3 va = f3(va4), wa = f3(d.omega[b.x]), vb = f3(vb4), wb = f3(d.omega[b.y]);
  const float mu = sqrtf(d.iinv[b.x].w * d.iinv[b.y].w);
  const float3 n = f3(d.m_normal[cur][slot]);
  const float3 t0 = f3(d.m_t0[cur][slot]), t1 = f3(d.m_t1[cur][slot]);
  const int cc = d.m_keycc[cur][slot].y;
  const bool accum = p.flags & BB_SIM_ACCUM_IMPULSE, fric = p.flags & BB_SIM_FRICTION;
  for (int j = 0; j < cc; ++j) {
    const uint32_t ci = slot * BB_MAX_CONTACTS + j;
    float4 lam = d.c_lam[cur][ci];
    pgs_contact_solve(d.c_r1[ci], d.c_r2[ci], d.c_k[ci], lam, n, t0, t1, mu, use_bias, accum, fric, ima, imb, IA, IB,
                      va, wa, vb, wb);
    d.c_lam[cur][ci] = lam;
  }
  if (fa & BB_BODY_DYNAMIC) {
    d.vel[b.x] = f4(va, va4.w);
    d.omega[b.x] = f4(wa, 0.f);
  }
  if (fb & BB_BODY_DYNAMIC) {
    d.vel[b.y] = f4(vb, vb4.w);
    d.omega[b.y] = f4(wb, 0.f);
  }
}

// integrate one body (RB_sim.slang:1287-1326) and refresh its world inverse inertia
// Compiled once (not inlined) so every path integrates with the same instructions.
__device__ __noinline__ void pgs_integrate_body(float4* pos, float4* rot, float4 vel, float4 omega,
                                                const float4* iinv, const float4* ioff, bool full, float4* iw,
                                                uint32_t i, float h, bool tq) {
  const float4 ps = pos[i];
  const float3 v = f3(vel);
  pos[i] = make_float4(ps.x + v.x * h, ps.y + v.y * h, ps.z + v.z * h, ps.w);
  const Quatf q = apply_angular_velocity(q_from(rot[i]), f3(omega), h);
  rot[i] = q_to4(q);
  const Sym3 s = body_world_inv_inertia(iinv, ioff, full, i, q, tq);
  iw[2 * i] = make_float4(s.xx, s.xy, s.xz, s.yy);
  iw[2 * i + 1] = make_float4(s.yz, s.zz, 0.f, 0.f);
}
__device__ __noinline__ void pgs_world_inertia_body(const float4* rot, const float4* iinv, const float4* ioff,
                                                    bool full, float4* iw, uint32_t i, bool tq) {
  const Sym3 s = body_world_inv_inertia(iinv, ioff, full, i, q_from(rot[i]), tq);
  iw[2 * i] = make_float4(s.xx, s.xy, s.xz, s.yy);
  iw[2 * i + 1] = make_float4(s.yz, s.zz, 0.f, 0.f);
}
__device__ __forceinline__ void pgs_world_inertia(const DevState& d, uint32_t i, bool tq) {
  pgs_world_inertia_body(d.rot, d.iinv, d.iinv_off, d.full_inertia != 0, d.iw, i, tq);
}
__device__ __forceinline__ void pgs_integrate(const DevState& d, uint32_t i, float h, bool tq) {
  pgs_integrate_body(d.pos, d.rot, d.vel[i], d.omega[i], d.iinv, d.iinv_off, d.full_inertia != 0, d.iw, i, h, tq);
}

// ---------------------------------------------------------------------------------------
// PGS_SOFT on colours: one persistent cooperative kernel without a barrier between colours.
//
// The sweeps give every body the ordered sequence of its manifolds by colour, and a manifold's
// result depends only on its two bodies' velocities.  So each body's velocity carries a tag: the
// number of updates it has had.  An item (a manifold) of sweep s waits until its two bodies
// carry s * degree + rank (the body's swept manifolds, and the item's place among them), runs,
// and stores them with the tag one higher.  Velocity and tag share one 16-byte word, loaded
// and stored as one (b128, relaxed, gpu scope), so a wait is the load of the data itself: no
// barrier, no fence and no separate flag.  The same order on every body as one barrier per
// colour gives, hence the same bits.
//
// Items are taken 32 at a time, a tile: a warp's lanes, all of one colour, so none waits for
// another lane of its warp.  Warp w of W runs the tiles w, w + W, ... in (sweep, colour)
// order, every wait points at an earlier tile, and all blocks are resident: no deadlock.
// Within a colour the items are sorted by contact count, so a tile's lanes run equally long.
//
// Layout: a compact copy in colour order.  Per item 88 bytes in planes of float4 (a warp reads
// 512 consecutive bytes), per contact 40 bytes: (position, normal mass), (tangent masses),
// (impulses, bias).  Contact j of a tile's lanes is stored lane after lane (those that have a
// contact j), after contact j - 1 of all: dense, and one run per load.  The lever arms are
// the contact's position minus the two anchors, as the pre-step forms them.
#define BB_PGS_THREADS 64
#define BB_PGS_PER_SM 4
#define BB_PGS_PF 4  // contacts of an item loaded together
// Sweeps between two grid barriers at most: a block that has no tiles, or is done with its own, waits
// for the others at the next barrier, and this bounds that wait however many sweeps are asked for.
#define BB_PGS_RUN 64u

// body i's tagged velocities (linear, angular) next to each other, in row scratch this solver
// does not use
__device__ __forceinline__ float4* pgs_vw(const DevState& d) { return d.c_k; }
__device__ __forceinline__ float2* pgs_tmass(const DevState& d) { return reinterpret_cast<float2*>(d.c_r2); }
__device__ __forceinline__ float2* pgs_anchor(const DevState& d) { return reinterpret_cast<float2*>(d.flow_rec); }

__device__ __forceinline__ float4 ld_tagged(const float4* p) {
  unsigned long long lo, hi;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  return make_float4(__uint_as_float(uint32_t(lo)), __uint_as_float(uint32_t(lo >> 32)), __uint_as_float(uint32_t(hi)),
                     __uint_as_float(uint32_t(hi >> 32)));
}
__device__ __forceinline__ void st_tagged(float4* p, float3 v, uint32_t tag) {
  const unsigned long long lo = (unsigned long long)__float_as_uint(v.x) | ((unsigned long long)__float_as_uint(v.y) << 32);
  const unsigned long long hi = (unsigned long long)__float_as_uint(v.z) | ((unsigned long long)tag << 32);
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}"
               :
               : "l"(p), "l"(lo), "l"(hi)
               : "memory");
}

// tiles of the colour lists: first tile of each colour (from the colour count on: the number of
// tiles) and first item of each colour
struct PgsTiles {
  uint32_t first[BB_MAX_COLORS + 1];
  uint32_t start[BB_MAX_COLORS + 2];
};
__device__ __forceinline__ void pgs_tiles(const DevState& d, PgsTiles& ft) {
  if (threadIdx.x < 32u) {
    const uint32_t lane = threadIdx.x;
    const uint32_t s0 = d.bucket_start[lane], s1 = d.bucket_start[lane + 1];
    uint32_t v = lane < d.ctr->gc_colors ? (s1 - s0 + 31u) / 32u : 0u;
    const uint32_t own = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, v, o);
      if (int(lane) >= o) v += u;
    }
    ft.first[lane] = v - own;
    ft.start[lane] = s0;
    if (lane == 31u) {
      ft.first[32] = v;
      ft.start[32] = s1;
      ft.start[33] = d.bucket_start[BB_MAX_COLORS + 1];
    }
  }
  __syncthreads();
}
// item of this lane in tile t (BB_NONE past the colour's end)
__device__ __forceinline__ uint32_t pgs_tile_item(const PgsTiles& ft, uint32_t t) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t c = uint32_t(__popc(__ballot_sync(0xFFFFFFFFu, ft.first[lane] <= t))) - 1u;
  const uint32_t k = ft.start[c] + (t - ft.first[c]) * 32u + lane;
  return k < ft.start[c + 1] ? k : BB_NONE;
}

// item record: x, y: bodies, bit 31 = dynamic; z: contact count | rank on a << 4 | degree of a
// << 9 | rank on b << 15 | degree of b << 20; w: first contact of the item's tile (overflow:
// of the item)
#define PGS_BODY(x) ((x) & 0x7FFFFFFFu)

// before a solve, per body: world inverse inertia and, for the colour sweeps, tagged velocities and no
// colours yet
__global__ void k_pgs_bodies(const DevState d, uint32_t n, Params p, bool sweeps) {
  const bool tq = p.quirks & BB_QUIRK_INERTIA_TRANSPOSE;
  float4* vw = pgs_vw(d);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    pgs_world_inertia(d, i, tq);
    if (!sweeps) continue;
    d.flow_counter[i] = 0u;
    vw[2 * size_t(i)] = f4(f3(d.vel[i]), 0.f);
    vw[2 * size_t(i) + 1] = f4(f3(d.omega[i]), 0.f);
  }
}

// per swept item (colours and overflow): contact count, to be scanned; its colour in the masks of
// its dynamic bodies (a body's rank and degree are bit counts of its mask)
__global__ void k_pgs_count(const DevState d, int cur) {
  const uint32_t end = d.bucket_start[BB_MAX_COLORS + 1], over = d.bucket_start[BB_MAX_COLORS];
  const uint32_t* list = d.bucket_vals[1];
  if (blockIdx.x == 0 && threadIdx.x == 0) d.ctr->pgs_manifolds = end;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < end; k += gridDim.x * blockDim.x) {
    const uint32_t m = list[k], slot = d.man_slot[cur][m];
    d.pgs_slot[k] = slot;
    d.pgs_cnt[k] = uint32_t(d.m_keycc[cur][slot].y);
    if (k >= over) continue;
    const uint2 b = d.m_bodies[cur][slot];
    const uint32_t bit = 1u << d.gc_color[m];
    if (d.flags[b.x] & BB_BODY_DYNAMIC) atomicOr(&d.flow_counter[b.x], bit);
    if (d.flags[b.y] & BB_BODY_DYNAMIC) atomicOr(&d.flow_counter[b.y], bit);
  }
}

// records, frames and contact rows of every swept item (the pre-step's row half; no body is
// touched), a warp per tile.  Bound by memory latency: an item's slot is a random line in each
// array.  Positions and impulses of BB_PGS_PF contacts load before the first row is formed (the
// stores of one contact may alias the next one's loads, so one by one they ran in turn) and only
// the tangent masses of the stored contact are written.  With the same grouping in k_pgs_finish
// the solve of 1M boxes (3 M manifolds) fell 7.39 -> 7.20 ms, of 1,024 worlds 1.89 -> 1.86 ms; two
// contacts at a time, or 80 registers for a third block per SM, gave 7.22 and 7.29 ms.
__global__ void k_pgs_build(const DevState d, Params p, int cur, float h) {
  __shared__ PgsTiles ft;
  pgs_tiles(d, ft);
  const float inv_h = h > 0.f ? 1.0f / h : 0.f;
  const float hertz = fminf(p.contact_hertz, inv_h * 0.3333333333333333f);
  const uint32_t T = ft.first[BB_MAX_COLORS], over = ft.start[BB_MAX_COLORS], end = ft.start[BB_MAX_COLORS + 1];
  const uint32_t TO = T + (end - over + 31u) / 32u;  // and the overflow bucket's tiles
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u, nw = gridDim.x * (blockDim.x >> 5);
  const uint32_t* list = d.bucket_vals[1];
  const size_t P = d.pair_capacity;
  for (uint32_t t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < TO; t += nw) {
    uint32_t k = BB_NONE;
    if (t < T) k = pgs_tile_item(ft, t);
    else if (over + (t - T) * 32u + lane < end) k = over + (t - T) * 32u + lane;
    const bool ov = t >= T;
    const uint32_t cc = k != BB_NONE ? d.pgs_cnt[k] : 0u, c0 = k != BB_NONE ? d.pgs_coff[k] : 0u;
    const uint32_t base = __shfl_sync(0xFFFFFFFFu, c0, 0);
    uint32_t slot = 0;
    float3 n{}, t0{}, t1{}, aa{}, ab{};
    float ima = 0.f, imb = 0.f;
    Sym3 IA{}, IB{};
    if (k != BB_NONE) {
      slot = d.pgs_slot[k];
      const uint2 b = d.m_bodies[cur][slot];
      const bool da = d.flags[b.x] & BB_BODY_DYNAMIC, db = d.flags[b.y] & BB_BODY_DYNAMIC;
      ima = d.pos[b.x].w;
      imb = d.pos[b.y].w;
      n = f3(d.m_normal[cur][slot]);
      t0 = f3(d.m_t0[cur][slot]);
      t1 = f3(d.m_t1[cur][slot]);
      aa = f3(d.m_anchor_a[cur][slot]);
      ab = f3(d.m_anchor_b[cur][slot]);
      IA = load_iw(d, b.x);
      IB = load_iw(d, b.y);
      const uint32_t below = ov ? 0u : (1u << d.gc_color[list[k]]) - 1u;
      const uint32_t ma = da ? d.flow_counter[b.x] : 0u, mb = db ? d.flow_counter[b.y] : 0u;
      d.pgs_rec[k] = make_uint4(b.x | (da ? 0x80000000u : 0u), b.y | (db ? 0x80000000u : 0u),
                                cc | uint32_t(__popc(ma & below)) << 4 | uint32_t(__popc(ma)) << 9 |
                                    uint32_t(__popc(mb & below)) << 15 | uint32_t(__popc(mb)) << 20,
                                ov ? c0 : base);
      d.pgs_frame[k] = f4(n, ima);
      d.pgs_frame[P + k] = f4(t0, imb);
      d.pgs_frame[2 * P + k] = f4(t1, sqrtf(d.iinv[b.x].w * d.iinv[b.y].w));
      d.pgs_mass[k] = f4(aa, ab.x);
      pgs_anchor(d)[k] = make_float2(ab.y, ab.z);
    }
    const SoftCoef s = pgs_soft_coef(ima, imb, h, hertz);
    uint32_t off = base;
    for (uint32_t j0 = 0; __any_sync(0xFFFFFFFFu, cc > j0); j0 += BB_PGS_PF) {
      float4 pp[BB_PGS_PF], lam[BB_PGS_PF];
#pragma unroll
      for (uint32_t u = 0; u < BB_PGS_PF; ++u) {
        const size_t ci = size_t(slot) * BB_MAX_CONTACTS + j0 + u;
        if (cc > j0 + u) {
          pp[u] = d.c_pos[cur][ci];
          lam[u] = d.c_lam[cur][ci];
        }
      }
#pragma unroll
      for (uint32_t u = 0; u < BB_PGS_PF; ++u) {
        const uint32_t j = j0 + u, m = __ballot_sync(0xFFFFFFFFu, cc > j);
        if (cc > j) {
          const size_t ci = size_t(slot) * BB_MAX_CONTACTS + j, r = ov ? c0 + j : off + uint32_t(__popc(m & lt));
          float4 R1, R2, K;
          pgs_contact_rows(pp[u], aa, ab, n, t0, t1, ima, imb, IA, IB, s, R1, R2, K);
          d.c_r1[r] = f4(f3(pp[u]), R1.w);
          pgs_tmass(d)[r] = make_float2(R2.w, K.x);
          d.pgs_lam[r] = make_float4(lam[u].x, lam[u].y, lam[u].z, K.y);
          // the reference writes its tangent masses into the persistent contact
          *reinterpret_cast<float2*>(&d.c_kt[cur][ci]) = make_float2(R2.w, K.x);
        }
        off += uint32_t(__popc(m));
      }
    }
  }
}

// contacts [first, first + BB_PGS_PF) of a tile's lanes, and where their impulses live
struct PgsRows {
  float4 A[BB_PGS_PF], L[BB_PGS_PF];
  float2 B[BB_PGS_PF];
  uint32_t at[BB_PGS_PF];
};
__device__ __forceinline__ void pgs_rows_load(const DevState& d, uint32_t cc, uint32_t first, uint32_t& off, PgsRows& x) {
  const uint32_t lt = (1u << (threadIdx.x & 31u)) - 1u;
#pragma unroll
  for (int j = 0; j < BB_PGS_PF; ++j) {
    const bool has = cc > first + uint32_t(j);
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, has);
    x.at[j] = off + uint32_t(__popc(m & lt));
    off += uint32_t(__popc(m));
    if (has) {
      x.A[j] = d.c_r1[x.at[j]];
      x.B[j] = pgs_tmass(d)[x.at[j]];
      x.L[j] = d.pgs_lam[x.at[j]];
    }
  }
}

struct PgsItem {
  float3 n, t0, t1, aa, ab;
  float ima, imb, mu, cm, ci;  // inverse masses, friction, soft coefficients
};
// the two soft-coefficient pairs (solvers.slang:150-158): a contact with a static body, and not
struct PgsCoef {
  float m[2], i[2];
};
__device__ __forceinline__ PgsItem pgs_item_load(const DevState& d, uint32_t k) {
  const size_t P = d.pair_capacity;
  const float4 f0 = d.pgs_frame[k], f1 = d.pgs_frame[P + k], f2 = d.pgs_frame[2 * P + k], f3_ = d.pgs_mass[k];
  const float2 g = pgs_anchor(d)[k];
  PgsItem x;
  x.n = f3(f0);
  x.ima = f0.w;
  x.t0 = f3(f1);
  x.imb = f1.w;
  x.t1 = f3(f2);
  x.mu = f2.w;
  x.aa = f3(f3_);
  x.ab = make_float3(f3_.w, g.x, g.y);
  return x;
}
// (apart from the load: its use of the masses would wait for them before the rows are asked for)
__device__ __forceinline__ void pgs_item_coef(PgsItem& x, const PgsCoef& co) {
  const bool fixed = x.ima == 0.f || x.imb == 0.f;
  x.cm = fixed ? co.m[1] : co.m[0];
  x.ci = fixed ? co.i[1] : co.i[0];
}

// One contact of an item, in a solve or relax sweep, and in the warm start.  PLAIN: impulses are
// accumulated and friction is on (the defaults), known at compile time: a contact is one dependent
// chain of some 40 operations, and each branch on a run-time flag in it costs as much as five of them.
template <bool PLAIN>
__device__ __forceinline__ void pgs_run_contact(const PgsItem& x, float4 A, float2 B, float4& L, bool use_bias, uint32_t flags,
                                                const Sym3& IA, const Sym3& IB, float3& va, float3& wa, float3& vb,
                                                float3& wb) {
  const bool accum = PLAIN || (flags & BB_SIM_ACCUM_IMPULSE), fric = PLAIN || (flags & BB_SIM_FRICTION);
  const float3 r1 = xsub(f3(A), x.aa), r2 = xsub(f3(A), x.ab);
  const float bias = L.w;
  float4 lam = L;
  pgs_contact_solve(f4(r1, A.w), f4(r2, B.x), make_float4(B.y, bias, x.cm, x.ci), lam, x.n, x.t0, x.t1, x.mu, use_bias, accum,
                    fric, x.ima, x.imb, IA, IB, va, wa, vb, wb);
  L = make_float4(lam.x, lam.y, lam.z, bias);
}
template <bool PLAIN>
__device__ __forceinline__ void pgs_warm_contact(const PgsItem& x, float4 A, float4 L, uint32_t flags, const Sym3& IA,
                                                 const Sym3& IB, float3& va, float3& wa, float3& vb, float3& wb) {
  pgs_contact_warm(xsub(f3(A), x.aa), xsub(f3(A), x.ab), L, x.n, x.t0, x.t1, PLAIN || (flags & BB_SIM_FRICTION), x.ima, x.imb,
                   IA, IB, va, wa, vb, wb);
}

// gives up a tagged wait past the world's limit, or when another wait already did
__device__ __forceinline__ bool pgs_gave_up(DevCounters* c, uint32_t spins) {
  if ((spins & 63u) != 0u) return false;
  const uint32_t lim = *reinterpret_cast<volatile const uint32_t*>(&c->wait_limit);
  if (spins > (lim ? lim : BB_SPIN_LIMIT)) {
    raise_wait_error(c, BB_SITE_FLOW);
    return true;
  }
  return (*reinterpret_cast<volatile const uint32_t*>(&c->error_flags) & BB_ERRF_SPIN_LIMIT) != 0;
}

// sweeps [s0, s1): those below warm are the warm start, those below mid solve, the rest relax
template <bool PLAIN>
__device__ __forceinline__ void pgs_sweeps(const DevState& d, const Params& p, const PgsTiles& ft, const PgsCoef& co,
                                           uint32_t s0, uint32_t s1, uint32_t warm, uint32_t mid, bool& dead) {
  const uint32_t T = ft.first[BB_MAX_COLORS];
  const uint32_t w0 = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, nw = gridDim.x * (BB_PGS_THREADS / 32);
  if (w0 >= T || s0 >= s1) return;
  const bool single = w0 + nw >= T;  // this warp's only tile stays in registers
  float4* vw = pgs_vw(d);
  uint32_t t = w0, s = s0;
  uint32_t k = pgs_tile_item(ft, t);
  uint4 rec = make_uint4(0, 0, 0, 0);
  if (k != BB_NONE) rec = d.pgs_rec[k];
  PgsItem x;
  PgsRows r;
  Sym3 IA, IB;
  bool fresh = true;
  uint32_t off = 0;
  for (;;) {
    // this warp's next tile and its record, a tile ahead
    uint32_t tn = t + nw, sn = s;
    if (tn >= T) {
      tn = w0;
      ++sn;
    }
    const uint32_t kn = pgs_tile_item(ft, tn);
    uint4 rn = make_uint4(0, 0, 0, 0);
    if (kn != BB_NONE) rn = d.pgs_rec[kn];
    const bool on = k != BB_NONE;
    const uint32_t a = PGS_BODY(rec.x), b = PGS_BODY(rec.y), cc = rec.z & 15u;
    const uint32_t na = s * ((rec.z >> 9) & 63u) + ((rec.z >> 4) & 31u), nb = s * (rec.z >> 20) + ((rec.z >> 15) & 31u);
    // The body loads go first: their first round trip overlaps the rows'.
    float4 va4, wa4, vb4, wb4;
    va4 = wa4 = vb4 = wb4 = make_float4(0.f, 0.f, 0.f, 0.f);
    auto bodies = [&](bool la, bool lb) {
      if (la) {
        va4 = ld_tagged(vw + 2 * size_t(a));
        wa4 = ld_tagged(vw + 2 * size_t(a) + 1);
      }
      if (lb) {
        vb4 = ld_tagged(vw + 2 * size_t(b));
        wb4 = ld_tagged(vw + 2 * size_t(b) + 1);
      }
    };
    bodies(on, on);
    if (fresh) {
      off = __shfl_sync(0xFFFFFFFFu, rec.w, 0);
      if (on) {
        x = pgs_item_load(d, k);
        IA = load_iw(d, a);
        IB = load_iw(d, b);
      }
      pgs_rows_load(d, cc, 0, off, r);
    }
    // the rows beyond the first BB_PGS_PF contacts, for tiles that have them
    const bool deep = __any_sync(0xFFFFFFFFu, cc > BB_PGS_PF);
    PgsRows y;
    if (deep) {
      uint32_t off2 = off;
      pgs_rows_load(d, cc, BB_PGS_PF, off2, y);
    }
    for (uint32_t spins = 0;;) {
      const bool okA = !on || (__float_as_uint(va4.w) == na && __float_as_uint(wa4.w) == na);
      const bool okB = !on || (__float_as_uint(vb4.w) == nb && __float_as_uint(wb4.w) == nb);
      if (__all_sync(0xFFFFFFFFu, okA && okB) || dead) break;
      bodies(!okA, !okB);
      dead = __any_sync(0xFFFFFFFFu, pgs_gave_up(d.ctr, ++spins));
    }
    float3 va = f3(va4), wa = f3(wa4), vb = f3(vb4), wb = f3(wb4);
    pgs_item_coef(x, co);
    if (s < warm) {
#pragma unroll
      for (int j = 0; j < BB_PGS_PF; ++j)
        if (cc > uint32_t(j)) pgs_warm_contact<PLAIN>(x, r.A[j], r.L[j], p.flags, IA, IB, va, wa, vb, wb);
      if (deep) {
#pragma unroll
        for (int j = 0; j < BB_PGS_PF; ++j)
          if (cc > uint32_t(BB_PGS_PF + j)) pgs_warm_contact<PLAIN>(x, y.A[j], y.L[j], p.flags, IA, IB, va, wa, vb, wb);
      }
    } else {
      const bool use_bias = s < mid;
#pragma unroll
      for (int j = 0; j < BB_PGS_PF; ++j)
        if (cc > uint32_t(j)) pgs_run_contact<PLAIN>(x, r.A[j], r.B[j], r.L[j], use_bias, p.flags, IA, IB, va, wa, vb, wb);
      if (deep) {
#pragma unroll
        for (int j = 0; j < BB_PGS_PF; ++j)
          if (cc > uint32_t(BB_PGS_PF + j))
            pgs_run_contact<PLAIN>(x, y.A[j], y.B[j], y.L[j], use_bias, p.flags, IA, IB, va, wa, vb, wb);
      }
    }
    // the bodies first: other warps wait for them
    if (rec.x >> 31) {
      st_tagged(vw + 2 * size_t(a), va, na + 1u);
      st_tagged(vw + 2 * size_t(a) + 1, wa, na + 1u);
    }
    if (rec.y >> 31) {
      st_tagged(vw + 2 * size_t(b), vb, nb + 1u);
      st_tagged(vw + 2 * size_t(b) + 1, wb, nb + 1u);
    }
    if (s >= warm) {
#pragma unroll
      for (int j = 0; j < BB_PGS_PF; ++j) {
        if (cc > uint32_t(j)) d.pgs_lam[r.at[j]] = r.L[j];
        if (deep && cc > uint32_t(BB_PGS_PF + j)) d.pgs_lam[y.at[j]] = y.L[j];
      }
    }
    if (sn >= s1) return;
    t = tn;
    s = sn;
    k = kn;
    rec = rn;
    fresh = !single;
  }
}

// One sweep over the overflow bucket, items [o0, o1): serially in manifold order by one warp, between
// grid barriers (plain loads and stores of the velocities; tags stay as they are).  Bound by the
// chain of its items: BB_PGS_OVER of them load at once, a lane each, then run one after the other,
// and an item's velocities go to the later lanes with the same body by shuffles.  One thread that
// loaded item after item and passed velocities through memory took 1.6 us per item of four contacts:
// 144 boxes on one dynamic plate (113 items, 84 sweeps per step) 19.8 -> 14.3 ms per step, a pile of
// 2,000 after one colouring round (3,443 items) 34.3 -> 19.8 ms.  The contacts wait in shared memory:
// in local arrays they cost the tiles' code 1.6 % (1,024 worlds), and 32 items' shared memory
// takes L1 from the tiles' rows (0.4 %).
#define BB_PGS_OVER 16u
__device__ __forceinline__ void pgs_overflow(const DevState& d, const Params& p, uint32_t o0, uint32_t o1, int mode,
                                             const PgsCoef& co) {
  __shared__ float4 A[BB_MAX_CONTACTS][BB_PGS_OVER], L[BB_MAX_CONTACTS][BB_PGS_OVER];
  __shared__ float2 B[BB_MAX_CONTACTS][BB_PGS_OVER];
  constexpr uint32_t ALL = 0xFFFFFFFFu;
  const uint32_t lane = threadIdx.x & 31u;
  float4* vw = pgs_vw(d);
  for (uint32_t k0 = o0; k0 < o1; k0 += BB_PGS_OVER) {
    const uint32_t count = min(BB_PGS_OVER, o1 - k0), k = k0 + min(lane, count - 1u);
    const uint4 rec = d.pgs_rec[k];
    const uint32_t a = PGS_BODY(rec.x), b = PGS_BODY(rec.y), cc = lane < count ? rec.z & 15u : 0u;
    PgsItem x = pgs_item_load(d, k);
    const Sym3 IA = load_iw(d, a), IB = load_iw(d, b);
    const float4 va4 = vw[2 * size_t(a)], wa4 = vw[2 * size_t(a) + 1], vb4 = vw[2 * size_t(b)], wb4 = vw[2 * size_t(b) + 1];
#pragma unroll 1
    for (uint32_t j = 0; j < cc; ++j) {
      A[j][lane] = d.c_r1[rec.w + j];
      B[j][lane] = pgs_tmass(d)[rec.w + j];
      L[j][lane] = d.pgs_lam[rec.w + j];
    }
    float3 va = f3(va4), wa = f3(wa4), vb = f3(vb4), wb = f3(wb4);
    pgs_item_coef(x, co);
    for (uint32_t l = 0; l < count; ++l) {
      if (lane == l) {
#pragma unroll 1
        for (uint32_t j = 0; j < cc; ++j) {
          float4 lam = L[j][lane];
          if (mode == 0) {
            pgs_warm_contact<false>(x, A[j][lane], lam, p.flags, IA, IB, va, wa, vb, wb);
          } else {
            pgs_run_contact<false>(x, A[j][lane], B[j][lane], lam, mode == 1, p.flags, IA, IB, va, wa, vb, wb);
            d.pgs_lam[rec.w + j] = lam;
          }
        }
      }
      __syncwarp();
      // (a dynamic body's bit 31 is set: only those are handed on)
      const uint32_t la = __shfl_sync(ALL, rec.x, int(l)), lb = __shfl_sync(ALL, rec.y, int(l));
      float f[12] = {va.x, va.y, va.z, wa.x, wa.y, wa.z, vb.x, vb.y, vb.z, wb.x, wb.y, wb.z};
#pragma unroll
      for (int q = 0; q < 12; ++q) f[q] = __shfl_sync(ALL, f[q], int(l));
      if (rec.x >> 31 && (rec.x == la || rec.x == lb)) {
        va = rec.x == la ? make_float3(f[0], f[1], f[2]) : make_float3(f[6], f[7], f[8]);
        wa = rec.x == la ? make_float3(f[3], f[4], f[5]) : make_float3(f[9], f[10], f[11]);
      }
      if (rec.y >> 31 && (rec.y == la || rec.y == lb)) {
        vb = rec.y == la ? make_float3(f[0], f[1], f[2]) : make_float3(f[6], f[7], f[8]);
        wb = rec.y == la ? make_float3(f[3], f[4], f[5]) : make_float3(f[9], f[10], f[11]);
      }
    }
    // (lanes that share a body hold the same velocities of it by now)
    if (rec.x >> 31) {
      vw[2 * size_t(a)] = f4(va, va4.w);
      vw[2 * size_t(a) + 1] = f4(wa, wa4.w);
    }
    if (rec.y >> 31) {
      vw[2 * size_t(b)] = f4(vb, vb4.w);
      vw[2 * size_t(b) + 1] = f4(wb, wb4.w);
    }
    __syncwarp();
  }
}

template <bool PLAIN>
__global__ void __launch_bounds__(BB_PGS_THREADS, BB_PGS_PER_SM) k_pgs_soft(const DevState d, Params p, uint32_t n, float h) {
  __shared__ PgsTiles ft;
  // test switch (bb_debug_wait_limit): the last block leaves, so the others' waits for it run out
  if (gridDim.x > 1 && blockIdx.x == gridDim.x - 1 && d.ctr->abandon_block) return;
  pgs_tiles(d, ft);
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  const bool tq = p.quirks & BB_QUIRK_INERTIA_TRANSPOSE;
  const float inv_h = h > 0.f ? 1.0f / h : 0.f;
  const float hertz = fminf(p.contact_hertz, inv_h * 0.3333333333333333f);
  const SoftCoef c0 = pgs_soft_coef(1.f, 1.f, h, hertz), c1 = pgs_soft_coef(0.f, 1.f, h, hertz);
  const PgsCoef co{{c0.mcoef, c1.mcoef}, {c0.icoef, c1.icoef}};
  uint32_t* sync = &d.ctr->sync_count[1];
  uint32_t epoch = 0;
  float4* vw = pgs_vw(d);
  bool dead = false;
  const uint32_t warm = (p.flags & BB_SIM_ACCUM_IMPULSE) ? 1u : 0u, mid = warm + p.iterations, last = mid + p.relax_iterations;
  const uint32_t o0 = ft.start[BB_MAX_COLORS], o1 = ft.start[BB_MAX_COLORS + 1];
  bool integrated = !(p.flags & BB_SIM_ADVECTION);
  for (uint32_t s = 0;;) {
    if (s == mid && !integrated) {
      grid_sync(d.ctr, sync, epoch);
      for (uint32_t i = tid; i < n; i += stride)
        if (awake(d.flags[i]))
          pgs_integrate_body(d.pos, d.rot, vw[2 * size_t(i)], vw[2 * size_t(i) + 1], d.iinv, d.iinv_off,
                             d.full_inertia != 0, d.iw, i, h, tq);
      grid_sync(d.ctr, sync, epoch);
      integrated = true;
    }
    if (s >= last) break;
    const uint32_t e = o0 != o1 ? s + 1u : min(s < mid ? mid : last, s + BB_PGS_RUN);
    pgs_sweeps<PLAIN>(d, p, ft, co, s, e, warm, mid, dead);
    if (o0 != o1) {  // overflow bucket: serial, in manifold order
      grid_sync(d.ctr, sync, epoch);
      if (tid < 32u) pgs_overflow(d, p, o0, o1, s < warm ? 0 : s < mid ? 1 : 2, co);
      grid_sync(d.ctr, sync, epoch);
    } else if (e - s == BB_PGS_RUN) {
      grid_sync(d.ctr, sync, epoch);
    }
    s = e;
  }
}

// after the sweeps: impulses back to the persistent contacts (with the mass coefficient the
// reference leaves there), velocities back to the bodies
__global__ void k_pgs_finish(const DevState d, Params p, int cur, uint32_t n, float h) {
  __shared__ PgsTiles ft;
  pgs_tiles(d, ft);
  const float inv_h = h > 0.f ? 1.0f / h : 0.f;
  const float hertz = fminf(p.contact_hertz, inv_h * 0.3333333333333333f);
  const uint32_t T = ft.first[BB_MAX_COLORS], over = ft.start[BB_MAX_COLORS], end = ft.start[BB_MAX_COLORS + 1];
  const uint32_t TO = T + (end - over + 31u) / 32u;
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u, nw = gridDim.x * (blockDim.x >> 5);
  for (uint32_t t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < TO; t += nw) {
    uint32_t k = BB_NONE;
    if (t < T) k = pgs_tile_item(ft, t);
    else if (over + (t - T) * 32u + lane < end) k = over + (t - T) * 32u + lane;
    const bool ov = t >= T;
    const uint32_t cc = k != BB_NONE ? d.pgs_cnt[k] : 0u, c0 = k != BB_NONE ? d.pgs_coff[k] : 0u;
    uint32_t off = __shfl_sync(0xFFFFFFFFu, c0, 0), slot = 0;
    float mcoef = 0.f;
    if (k != BB_NONE) {
      slot = d.pgs_slot[k];
      mcoef = pgs_soft_coef(d.pgs_frame[k].w, d.pgs_frame[size_t(d.pair_capacity) + k].w, h, hertz).mcoef;
    }
    for (uint32_t j0 = 0; __any_sync(0xFFFFFFFFu, cc > j0); j0 += BB_PGS_PF) {
      float4 L[BB_PGS_PF];
#pragma unroll
      for (uint32_t u = 0; u < BB_PGS_PF; ++u) {
        const uint32_t j = j0 + u, m = __ballot_sync(0xFFFFFFFFu, cc > j);
        if (cc > j) L[u] = d.pgs_lam[ov ? c0 + j : off + uint32_t(__popc(m & lt))];
        off += uint32_t(__popc(m));
      }
#pragma unroll
      for (uint32_t u = 0; u < BB_PGS_PF; ++u)
        if (cc > j0 + u)
          d.c_lam[cur][size_t(slot) * BB_MAX_CONTACTS + j0 + u] = make_float4(L[u].x, L[u].y, L[u].z, mcoef);
    }
  }
  const float4* vw = pgs_vw(d);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (!(d.flags[i] & BB_BODY_DYNAMIC)) continue;
    d.vel[i] = f4(f3(vw[2 * size_t(i)]), d.vel[i].w);
    d.omega[i] = f4(f3(vw[2 * size_t(i) + 1]), 0.f);
  }
}

// blocks of k_pgs_soft per SM (one unit of its grid) that are resident together
static int pgs_blocks_per_sm() {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)k_pgs_soft<true>, BB_PGS_THREADS, 0);
  int other = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&other, (const void*)k_pgs_soft<false>, BB_PGS_THREADS, 0);
  per_sm = std::min(per_sm, other);
  return std::max(1, std::min(per_sm, BB_PGS_PER_SM));
}

// Grid: as many SMs' worth of blocks as 256-thread groups fit the largest colour (about half the
// bodies), so a small world leaves the rest of the GPU to other streams.
int bb_pgs_soft_blocks(int sms, uint32_t max_bodies) {
  const uint64_t groups = (uint64_t(max_bodies) / 2 + 255) / 256;
  return int(std::max<uint64_t>(1, std::min<uint64_t>(uint64_t(sms), groups))) * pgs_blocks_per_sm();
}

void bb_solve_pgs_soft(cudaStream_t s, const DevState& d, const Params& p, uint32_t n, float h, int cur,
                       const StepScratch& sc, int coop_blocks, int sms) {
  if (n == 0) return;
  const int T = BB_THREADS;
  const uint32_t blocks = (n + T - 1) / T;
  k_pgs_bodies<<<blocks, T, 0, s>>>(d, n, p, true);
  k_pgs_count<<<sms * 8, T, 0, s>>>(d, cur);
  bb_launch_scan(s, d.pgs_cnt, d.pgs_coff, &d.bucket_start[BB_MAX_COLORS + 1], d.pair_capacity, &d.ctr->pgs_contacts,
                 sc.scan_status + 4 * size_t(sc.scan_tiles), sc.scan_tile_ctr + 4, d.ctr);
  k_pgs_build<<<sms * 8, T, 0, s>>>(d, p, cur, h);
  DevState dd = d;
  Params pp = p;
  uint32_t nn = n;
  float hh = h;
  void* args[] = {&dd, &pp, &nn, &hh};
  const uint32_t both = BB_SIM_ACCUM_IMPULSE | BB_SIM_FRICTION;
  bb_launch_coop((p.flags & both) == both ? (const void*)k_pgs_soft<true> : (const void*)k_pgs_soft<false>, coop_blocks,
                 BB_PGS_THREADS, args, s);
  k_pgs_finish<<<sms * 8, T, 0, s>>>(d, p, cur, n, h);
}

// ---------------------------------------------------------------------------------------
// Per-island path (USE_GRAPH_COLORING off, RBM:1390-1399; RB_sim.slang:1122-1406): one thread
// per contact island runs the island's manifolds serially, in manifold order -- PGS_SOFT's
// pre-step and solve sweeps, or the Baumgarte PGS of solvers.slang:3-136 -- then all bodies
// integrate, then (PGS_SOFT only) the relax sweeps run per island again.  Manifolds are grouped
// by island with a stable sort keyed by the island id of their dynamic body.

// PGS::pre_step (solvers.slang:3-66) of one manifold slot
__device__ void baum_pre_step_slot(const DevState& d, const Params& p, int cur, uint32_t slot, uint2 b, float inv_h) {
  const uint32_t fa = d.flags[b.x], fb = d.flags[b.y];
  if (!awake(fa) && !awake(fb)) return;
  const float ima = d.pos[b.x].w, imb = d.pos[b.y].w;
  const Sym3 IA = load_iw(d, b.x), IB = load_iw(d, b.y);
  float3 va = f3(d.vel[b.x]), wa = f3(d.omega[b.x]), vb = f3(d.vel[b.y]), wb = f3(d.omega[b.y]);
  const float3 n = f3(d.m_normal[cur][slot]);
  const float3 t0 = f3(d.m_t0[cur][slot]), t1 = f3(d.m_t1[cur][slot]);
  const float3 pa = f3(d.pos[b.x]), pb = f3(d.pos[b.y]);
  const int cc = d.m_keycc[cur][slot].y;
  const bool accum = p.flags & BB_SIM_ACCUM_IMPULSE, fric = p.flags & BB_SIM_FRICTION;
  for (int j = 0; j < cc; ++j) {
    const uint32_t ci = slot * BB_MAX_CONTACTS + j;
    const float4 pp = d.c_pos[cur][ci];
    const float3 r1 = xsub(f3(pp), pa), r2 = xsub(f3(pp), pb);
    const float nmass = xrow_mass(r1, r2, n, ima, imb, IA, IB);
    const float tm0 = xrow_mass(r1, r2, t0, ima, imb, IA, IB), tm1 = xrow_mass(r1, r2, t1, ima, imb, IA, IB);
    const float bias = -0.2f * inv_h * fminf(pp.w + 0.01f, 0.f);
    d.c_r1[ci] = f4(r1, nmass);
    d.c_r2[ci] = f4(r2, tm0);
    d.c_k[ci] = make_float4(tm1, bias, 0.f, 0.f);
    const float4 lam = d.c_lam[cur][ci];
    if (accum) pgs_contact_warm(r1, r2, lam, n, t0, t1, fric, ima, imb, IA, IB, va, wa, vb, wb);
  }
  if (fa & BB_BODY_DYNAMIC) {
    d.vel[b.x] = f4(va, d.vel[b.x].w);
    d.omega[b.x] = f4(wa, 0.f);
  }
  if (fb & BB_BODY_DYNAMIC) {
    d.vel[b.y] = f4(vb, d.vel[b.y].w);
    d.omega[b.y] = f4(wb, 0.f);
  }
}

// PGS::solve (solvers.slang:68-136) of one manifold slot
__device__ void baum_solve_slot(const DevState& d, const Params& p, int cur, uint32_t slot, uint2 b) {
  const uint32_t fa = d.flags[b.x], fb = d.flags[b.y];
  if (!awake(fa) && !awake(fb)) return;
  const float ima = d.pos[b.x].w, imb = d.pos[b.y].w;
  const Sym3 IA = load_iw(d, b.x), IB = load_iw(d, b.y);
  float4 va4 = d.vel[b.x], vb4 = d.vel[b.y];
  float3 va = f3(va4), wa = f3(d.omega[b.x]), vb = f3(vb4), wb = f3(d.omega[b.y]);
  const float mu = sqrtf(d.iinv[b.x].w * d.iinv[b.y].w);
  const float3 n = f3(d.m_normal[cur][slot]);
  const float3 t0 = f3(d.m_t0[cur][slot]), t1 = f3(d.m_t1[cur][slot]);
  const int cc = d.m_keycc[cur][slot].y;
  const bool accum = p.flags & BB_SIM_ACCUM_IMPULSE, fric = p.flags & BB_SIM_FRICTION;
  for (int j = 0; j < cc; ++j) {
    const uint32_t ci = slot * BB_MAX_CONTACTS + j;
    const float4 R1 = d.c_r1[ci], R2 = d.c_r2[ci], K = d.c_k[ci];
    float4 lam = d.c_lam[cur][ci];
    const float3 r1 = f3(R1), r2 = f3(R2);
    if (fric) {
      const float3 rv = xrel(r1, r2, va, wa, vb, wb);
      const float tmass[2] = {R2.w, K.x};
      float imp_t[2] = {lam.y, lam.z};
      const float maxf = mu * lam.x;
      for (int k = 0; k < 2; ++k) {
        const float3 t = k == 0 ? t0 : t1;
        float ti = tmass[k] * -xdot(rv, t);
        if (accum) {
          const float old = imp_t[k];
          imp_t[k] = fminf(fmaxf(old + ti, -maxf), maxf);
          ti = imp_t[k] - old;
        } else {
          ti = fminf(fmaxf(ti, -maxf), maxf);
        }
        xapply(xscale(t, ti), r1, r2, ima, imb, IA, IB, va, wa, vb, wb);
      }
      lam.y = imp_t[0];
      lam.z = imp_t[1];
    }
    float imp = R1.w * (K.y - xdot(xrel(r1, r2, va, wa, vb, wb), n));
    if (accum) {
      const float old = lam.x;
      lam.x = fmaxf(old + imp, 0.f);
      imp = lam.x - old;
    } else {
      imp = fmaxf(imp, 0.f);
    }
    xapply(xscale(n, imp), r1, r2, ima, imb, IA, IB, va, wa, vb, wb);
    d.c_lam[cur][ci] = lam;
  }
  if (fa & BB_BODY_DYNAMIC) {
    d.vel[b.x] = f4(va, va4.w);
    d.omega[b.x] = f4(wa, 0.f);
  }
  if (fb & BB_BODY_DYNAMIC) {
    d.vel[b.y] = f4(vb, vb4.w);
    d.omega[b.y] = f4(wb, 0.f);
  }
}

// key of every manifold: the island of its dynamic body
__global__ void k_island_keys(const DevState d, int cur) {
  const uint32_t M = d.ctr->manifold_count;
  for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < M; m += gridDim.x * blockDim.x) {
    const uint2 b = d.m_bodies[cur][d.man_slot[cur][m]];
    const uint32_t ia = d.island[b.x];
    d.bucket_keys[0][m] = ia != BB_NONE ? ia : d.island[b.y];
    d.bucket_vals[0][m] = m;
  }
}
// island_start[v] = first sorted position with key >= v, v = 0..island_count
__global__ void k_island_starts(const DevState d, uint32_t* starts, uint32_t n) {
  const uint32_t M = d.ctr->manifold_count, nb = d.ctr->island_count;
  const uint32_t* keys = d.bucket_keys[1];
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v <= nb && v <= n; v += gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = M;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (keys[mid] < v) lo = mid + 1;
      else hi = mid;
    }
    starts[v] = lo;
  }
}
// phase 0: pre-step + solve sweeps; phase 1: relax sweeps (PGS_SOFT)
__global__ void k_island_solve(const DevState d, Params p, int cur, const uint32_t* starts, float h, int phase) {
  const uint32_t nb = d.ctr->island_count;
  const uint32_t* list = d.bucket_vals[1];
  const float inv_h = h > 0.f ? 1.0f / h : 0.f;
  const float hertz = fminf(p.contact_hertz, inv_h * 0.3333333333333333f);
  const bool soft = p.solver == BB_SOLVER_PGS_SOFT;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nb; v += gridDim.x * blockDim.x) {
    const uint32_t s0 = starts[v], s1 = starts[v + 1];
    auto each = [&](auto&& fn) {
      for (uint32_t k = s0; k < s1; ++k) {
        const uint32_t slot = d.man_slot[cur][list[k]];
        fn(slot, d.m_bodies[cur][slot]);
      }
    };
    if (phase == 0) {
      each([&](uint32_t slot, uint2 b) {
        if (soft) pgs_pre_step_slot(d, p, cur, slot, b, h, hertz);
        else baum_pre_step_slot(d, p, cur, slot, b, inv_h);
      });
      for (uint32_t it = 0; it < p.iterations; ++it)
        each([&](uint32_t slot, uint2 b) {
          if (soft) pgs_solve_slot(d, p, cur, slot, b, true);
          else baum_solve_slot(d, p, cur, slot, b);
        });
    } else {
      for (uint32_t it = 0; it < p.relax_iterations; ++it)
        each([&](uint32_t slot, uint2 b) { pgs_solve_slot(d, p, cur, slot, b, false); });
    }
  }
}
__global__ void k_island_integrate(const DevState d, Params p, uint32_t n, float h) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && awake(d.flags[i])) pgs_integrate(d, i, h, p.quirks & BB_QUIRK_INERTIA_TRANSPOSE);
}

void bb_solve_islands(cudaStream_t s, const DevState& d, const Params& p, uint32_t n, float h, int cur,
                      const StepScratch& sc, int sms) {
  if (n == 0) return;
  const int T = BB_THREADS;
  const uint32_t blocks = (n + T - 1) / T;
  k_pgs_bodies<<<blocks, T, 0, s>>>(d, n, p, false);
  k_island_keys<<<sms * 8, T, 0, s>>>(d, cur);
  uint32_t* keys[2] = {d.bucket_keys[0], d.bucket_keys[1]};
  uint32_t* vals[2] = {d.bucket_vals[0], d.bucket_vals[1]};
  // 3 digits (islands < 2^24): histogram region 1 and status slots 6..8 (the colouring's, unused here)
  uint32_t* hist = sc.sort_hist + 1 * BB_HIST_REGION;
  bb_launch_sort(s, keys, vals, &d.ctr->manifold_count, d.pair_capacity, 3, 0, hist,
                 sc.sort_status + 6 * size_t(sc.sort_tiles) * 256, sc.sort_tile_ctr + 6, d.ctr, sms);
  k_island_starts<<<(n + 1 + T - 1) / T, T, 0, s>>>(d, d.island_start, n);
  k_island_solve<<<(n + 127) / 128, 128, 0, s>>>(d, p, cur, d.island_start, h, 0);
  if (p.flags & BB_SIM_ADVECTION) k_island_integrate<<<blocks, T, 0, s>>>(d, p, n, h);
  if (p.solver == BB_SOLVER_PGS_SOFT) k_island_solve<<<(n + 127) / 128, 128, 0, s>>>(d, p, cur, d.island_start, h, 1);
}

// ---------------------------------------------------------------------------------------
// AVBD
__device__ __forceinline__ uint32_t avbd_priority(uint32_t body, uint32_t round) {
  uint32_t x = body * 0x9e3779b9u + round * 0x85ebca6bu;
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return ((x & 0xFFFu) << 20) | (body & 0xFFFFFu);
}
__device__ __forceinline__ float3 small_angle_delta(Quatf now, Quatf start) {
  Quatf dq = q_mul(now, q_conj(start));
  float sg = dq.w < 0.f ? -1.f : 1.f;
  return make_float3(dq.x, dq.y, dq.z) * (2.0f * sg);
}
__device__ __forceinline__ float3 avbd_q_rotate(Quatf q, float3 u) {
  float3 qv = make_float3(q.x, q.y, q.z);
  return u + 2.0f * cross3(qv, cross3(qv, u) + u * q.w);
}

// Jones-Plassmann colouring with start-of-round semantics: body_color holds
// ((round + 1) << 8) | colour while the kernel runs, so a neighbour coloured in the current
// round still counts as uncoloured.
__global__ void __launch_bounds__(BB_COOP_THREADS, 1) k_avbd_color(const DevState d, Params p, int cur, uint32_t n) {
  DevCounters* c = d.ctr;
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  uint32_t* uncol = c->round_flags;
  uint32_t* sync = &c->sync_count[2];
  uint32_t ep = 0;
  for (uint32_t i = tid; i < n; i += stride) d.body_color[i] = BB_UNCOLORED;
  if (tid == 0) {
    uncol[0] = 0;
    uncol[1] = 0;
    c->avbd_colors = 0;
  }
  grid_sync(c, sync, ep);
  for (uint32_t rd = 0; rd < p.avbd_color_rounds; ++rd) {
    uint32_t left = 0;
    for (uint32_t i = tid; i < n; i += stride) {
      if (d.body_color[i] != BB_UNCOLORED || !(d.flags[i] & BB_BODY_DYNAMIC)) continue;
      const uint32_t mine = avbd_priority(local_id(d, i), rd);
      uint32_t used = 0;
      bool wait = false;
      const uint32_t s0 = d.csr_start[cur][i], s1 = d.csr_start[cur][i + 1];
      for (uint32_t e = s0; e < s1 && !wait; ++e) {
        const uint32_t q = d.csr_partner[cur][e];
        if (q == i || !(d.flags[q] & BB_BODY_DYNAMIC)) continue;
        uint32_t pc = *(volatile uint32_t*)&d.body_color[q];
        bool unc = pc == BB_UNCOLORED || (pc >> 8) == rd + 1u;
        if (unc) {
          if (avbd_priority(local_id(d, q), rd) > mine) wait = true;
        } else {
          used |= 1u << (pc & 255u);
        }
      }
      if (wait || used == 0xFFFFFFFFu) {
        ++left;
        continue;
      }
      uint32_t col = uint32_t(__ffs(~used) - 1);
      d.body_color[i] = ((rd + 1u) << 8) | col;
      atomicMax(&c->avbd_colors, col + 1u);
    }
    if (left) atomicAdd(&uncol[rd & 1], left);
    grid_sync(c, sync, ep);
    if (*(volatile uint32_t*)&uncol[rd & 1] == 0u) break;
    if (tid == 0) uncol[(rd + 1) & 1] = 0;
    grid_sync(c, sync, ep);
  }
  for (uint32_t i = tid; i < n; i += stride) {
    uint32_t v = d.body_color[i];
    d.body_color[i] = v == BB_UNCOLORED ? BB_UNCOLORED : (v & 255u);
    d.a_depth[i] = awake(d.flags[i]) ? BB_NONE : 0u;
  }
  // Support depth (avbd.slang:667-724): breadth-first from the bodies at rest, one pass over the
  // manifolds per shock layer, until a pass lowers no depth (the reference dispatches all passes;
  // the later ones change nothing).
  grid_sync(c, sync, ep);  // the colouring's last flags are read
  if (tid == 0) {
    uncol[0] = 0;
    uncol[1] = 0;
  }
  grid_sync(c, sync, ep);
  const uint32_t M = c->manifold_count;
  for (uint32_t k = 0; k < p.avbd_shock_layers; ++k) {
    bool lower = false;
    for (uint32_t m = tid; m < M; m += stride) {
      const uint32_t slot = d.man_slot[cur][m];
      if (d.m_keycc[cur][slot].y <= 0) continue;
      const uint2 b = d.m_bodies[cur][slot];
      const uint32_t d1 = *(volatile uint32_t*)&d.a_depth[b.x], d2 = *(volatile uint32_t*)&d.a_depth[b.y];
      if (d2 != BB_NONE && d2 + 1u < d1) {
        atomicMin(&d.a_depth[b.x], d2 + 1u);
        lower = true;
      }
      if (d1 != BB_NONE && d1 + 1u < d2) {
        atomicMin(&d.a_depth[b.y], d1 + 1u);
        lower = true;
      }
    }
    if (lower) atomicOr(&uncol[k & 1], 1u);
    grid_sync(c, sync, ep);
    if (*(volatile uint32_t*)&uncol[k & 1] == 0u) break;
    if (tid == 0) uncol[(k + 1) & 1] = 0;
    grid_sync(c, sync, ep);
  }
}

// displacement of body i since the step's start, linear and angular (the AVBD sweeps read a
// partner's 32 bytes here instead of its pose and start pose)
__device__ __forceinline__ void avbd_store_disp(const DevState& d, uint32_t i, float3 dp, float3 dth) {
  d.iw[2 * size_t(i)] = f4(dp, 0.f);
  d.iw[2 * size_t(i) + 1] = f4(dth, 0.f);
}

__global__ void k_avbd_prepare(const DevState d, Params p, uint32_t n, float dt) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t f = d.flags[i];
  if (!awake(f)) return;
  float3 w = f3(d.omega[i]);
  float om = len3(w);
  if (om > 50.0f) {
    w = w * (50.0f / om);
    d.omega[i] = f4(w, 0.f);
  }
  float grav = (f & BB_BODY_GRAVITY) ? p.gravity : 0.f;
  float4 ps = d.pos[i];
  float3 pos = f3(ps), v = f3(d.vel[i]);
  Quatf q = q_from(d.rot[i]);
  d.a_pos_start[i] = f4(pos, 0.f);
  d.a_rot_start[i] = q_to4(q);
  d.a_pos_tilde[i] = f4(pos + v * dt + make_float3(0.f, grav, 0.f) * (dt * dt), 0.f);
  Quatf qt = apply_angular_velocity(q, w, dt);
  d.a_rot_tilde[i] = q_to4(qt);
  float aw = 0.f;
  if (fabsf(grav) > 1e-6f) {
    float ay = (v.y - d.pvel[i].y) / dt;
    float sg = grav > 0.f ? 1.f : -1.f;
    aw = fminf(fmaxf(ay * sg / fabsf(grav), 0.f), 1.f);
  }
  const float3 pn = pos + v * dt + make_float3(0.f, grav, 0.f) * (aw * dt * dt);
  d.pos[i] = f4(pn, ps.w);
  d.rot[i] = q_to4(qt);
  avbd_store_disp(d, i, pn - pos, small_angle_delta(qt, q));
}

__global__ void k_avbd_warmstart(const DevState d, Params p, int cur) {
  const uint32_t M = d.ctr->manifold_count;
  const bool warm = p.flags & BB_SIM_WARM_STARTING;
  for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < M; m += gridDim.x * blockDim.x) {
    const uint32_t slot = d.man_slot[cur][m];
    const uint2 b = d.m_bodies[cur][slot];
    const uint32_t fa = d.flags[b.x], fb = d.flags[b.y];
    // a paused world's manifolds are carried unchanged (no penalty decay, no new anchors), so
    // the world resumes exactly as it stopped
    if ((fa | fb) & BB_BODY_PAUSED) continue;
    bool d1 = awake(fa), d2 = awake(fb);
    float3 c1 = d1 ? f3(d.a_pos_start[b.x]) : f3(d.pos[b.x]);
    float3 c2 = d2 ? f3(d.a_pos_start[b.y]) : f3(d.pos[b.y]);
    Quatf q1c = q_conj(d1 ? q_from(d.a_rot_start[b.x]) : q_from(d.rot[b.x]));
    Quatf q2c = q_conj(d2 ? q_from(d.a_rot_start[b.y]) : q_from(d.rot[b.y]));
    const int cc = d.m_keycc[cur][slot].y;
    const float3 td[2] = {f3(d.m_t0[cur][slot]), f3(d.m_t1[cur][slot])};
    const float mu = sqrtf(fmaxf(d.iinv[b.x].w, 0.f) * fmaxf(d.iinv[b.y].w, 0.f));
    const Quatf q1 = d1 ? q_from(d.a_rot_start[b.x]) : q_from(d.rot[b.x]);
    const Quatf q2 = d2 ? q_from(d.a_rot_start[b.y]) : q_from(d.rot[b.y]);
    uint32_t sticks = 0;
    for (int j = 0; j < cc; ++j) {
      const uint32_t ci = slot * BB_MAX_CONTACTS + j;
      float4 lam = d.c_lam[cur][ci];
      float4 kt = d.c_kt[cur][ci];
      uint32_t wcount = __float_as_uint(kt.w), stick = __float_as_uint(kt.z);
      bool matched = wcount != 0u && warm;
      if (!matched) {
        lam = make_float4(0.f, 0.f, 0.f, p.avbd_k_min);
        kt.x = kt.y = p.avbd_k_min;
        stick = 0;
      } else {
        lam.w = fminf(fmaxf(lam.w * p.avbd_gamma, p.avbd_k_min), p.avbd_k_max);
        lam.x = fminf(lam.x, 0.f);
        kt.x = fminf(fmaxf(kt.x * p.avbd_gamma, p.avbd_k_min), p.avbd_k_max);
        kt.y = fminf(fmaxf(kt.y * p.avbd_gamma, p.avbd_k_min), p.avbd_k_max);
      }
      bool sticking = matched && stick != 0u;
      const float4 cp = d.c_pos[cur][ci];
      float4 aa = d.c_anc_a[cur][ci], ab = d.c_anc_b[cur][ci];
      if (!sticking) {
        aa = f4(avbd_q_rotate(q1c, f3(cp) - c1), aa.w);
        ab = f4(avbd_q_rotate(q2c, f3(cp) - c2), 0.f);
        d.c_anc_a[cur][ci] = aa;
        d.c_anc_b[cur][ci] = ab;
      } else {
        ++sticks;
      }
      d.c_lam[cur][ci] = lam;
      d.c_kt[cur][ci] = make_float4(kt.x, kt.y, __uint_as_float(stick), kt.w);
      // rows: what the sweeps need of this contact that no sweep changes
      const float3 ar1 = avbd_q_rotate(q1, f3(aa)), ar2 = avbd_q_rotate(q2, f3(ab));
      const float3 sep = (c2 + ar2) - (c1 + ar1);
      d.c_r1[ci] = f4(f3(cp) - c1, cp.w + p.avbd_margin);
      d.c_r2[ci] = f4(f3(cp) - c2, dot3(td[0], sep));
      d.c_k[ci] = f4(ar1, dot3(td[1], sep));
      d.pgs_lam[ci] = f4(ar2, mu);
    }
    if (sticks) atomicAdd(&d.ctr->stick, sticks);
  }
}

// starts[v] = first sorted position with key >= v * scale, for v in [0, nb]
__global__ void k_lower_bounds(const uint32_t* keys, uint32_t n, uint32_t* starts, uint32_t nb, uint32_t scale) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v > nb) return;
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    if (keys[mid] < v * scale) lo = mid + 1;
    else hi = mid;
  }
  starts[v] = lo;
}

// One contact's rows, written once per substep by k_avbd_warmstart at the contact's slot index:
// R0 = lever arm on a and depth + margin, R1 = lever arm on b and the start separation along
// tangent 0, R2 = anchor arm on a and the separation along tangent 1, R3 = anchor arm on b and
// the pair's friction.  The sweeps visit a contact some 25 times per body and substep; forming
// these from positions, start poses and anchors on each visit took ~20 dependent gathers.
struct AvbdRow {
  float4 r0, r1, r2, r3;
};
__device__ __forceinline__ AvbdRow avbd_row(const DevState& d, uint32_t ci) {
  return AvbdRow{d.c_r1[ci], d.c_r2[ci], d.c_k[ci], d.pgs_lam[ci]};
}
// displacements of a manifold's two bodies since the step's start
struct AvbdDisp {
  float3 dp1, dth1, dp2, dth2;
};

__device__ __forceinline__ float avbd_contact_C(const AvbdRow& r, const AvbdDisp& u, bool d1, bool d2, float alpha, float3 n) {
  float C = r.r0.w * (1.0f - alpha);
  if (d1) C -= dot3(n, u.dp1 + cross3(u.dth1, f3(r.r0)));
  if (d2) C += dot3(n, u.dp2 + cross3(u.dth2, f3(r.r1)));
  return C;
}

__device__ __forceinline__ float avbd_dir_C(const AvbdRow& r, const AvbdDisp& u, float C0t, float slop, bool d1, bool d2,
                                            float alpha, float3 dir) {
  float sg = C0t > 0.f ? 1.f : (C0t < 0.f ? -1.f : 0.f);
  float c0e = sg * fmaxf(0.f, fabsf(C0t) - slop);
  float C = c0e * (1.0f - alpha);
  if (d1) C -= dot3(dir, u.dp1 + cross3(u.dth1, f3(r.r2)));
  if (d2) C += dot3(dir, u.dp2 + cross3(u.dth2, f3(r.r3)));
  return C;
}

// per entry of the bodies' manifold lists: x = partner | partner awake << 30 | this body is a << 31,
// y = slot | (contact count - 1) << 29
__device__ __forceinline__ uint2* avbd_entries(const DevState& d) { return reinterpret_cast<uint2*>(d.pgs_rec); }
__device__ __forceinline__ uint32_t* avbd_class(const DevState& d) { return d.flow_counter; }
// Also the body's work class, 0 for the most: by the contacts of its longest lane (lane l sums the
// manifolds l, l + AVBD_LANES, ... of the list).  The sweeps take a colour's bodies by class, so
// that the bodies of a warp are equally long and the long ones start first.
#define AVBD_LANES 8
#define AVBD_CLASSES 7u
__global__ void k_avbd_entries(const DevState d, uint32_t n, int cur) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !awake(d.flags[i])) return;
  uint32_t len[AVBD_LANES] = {}, l = 0, most = 0;
  for (uint32_t e = d.csr_start[cur][i]; e < d.csr_start[cur][i + 1]; ++e, l = (l + 1) % AVBD_LANES) {
    const uint32_t slot = d.csr_slot[cur][e], q = d.csr_partner[cur][e], cc = uint32_t(d.m_keycc[cur][slot].y);
    avbd_entries(d)[e] = make_uint2(q | (awake(d.flags[q]) ? 1u << 30 : 0u) | (d.m_bodies[cur][slot].x == i ? 1u << 31 : 0u),
                                    slot | (cc - 1u) << 29);
#pragma unroll
    for (int k = 0; k < AVBD_LANES; ++k)
      if (uint32_t(k) == l) {
        len[k] += cc;
        most = max(most, len[k]);
      }
  }
  avbd_class(d)[i] = most > 8u ? 0u : most > 6u ? 1u : most > 4u ? 2u : most > 3u ? 3u : most > 2u ? 4u : most > 1u ? 5u : 6u;
}

// bucket keys of awake coloured bodies: bucket * AVBD_CLASSES + work class, where the bucket is the
// colour (main and last sweeps) or min(depth, L-1) * 32 + colour (post-stabilisation cascade);
// others sort last
__global__ void k_avbd_keys(const DevState d, Params p, uint32_t n, int post) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t col = d.body_color[i];
  uint32_t key = 0xFFFFu;
  if (awake(d.flags[i]) && col < BB_MAX_COLORS) {
    if (post) {
      uint32_t layer = min(d.a_depth[i], p.avbd_shock_layers - 1u);
      key = layer * BB_MAX_COLORS + col;
    } else {
      key = col;
    }
    key = key * AVBD_CLASSES + avbd_class(d)[i];
  }
  (post ? d.bucket_keys[0] : d.a_bucket_keys[0])[i] = key;
  (post ? d.bucket_vals[0] : d.a_bucket_vals[0])[i] = i;
}
// entry_avbd_primal (avbd.slang:478-658): Gauss-Newton step of body i on its 6 DoF, in two
// parts: the sums over its contacts (avbd_gather) and the solve (avbd_move).
// A group of AVBD_LANES lanes per body.  Lane l of the group takes manifolds l, l + AVBD_LANES, ...
// of the body's list and sums their contacts' gradient and Hessian terms in order; a butterfly
// over the group adds the lanes' sums (a fixed order, so the result does not depend on
// scheduling or on which bodies share a warp; it differs from a serial sum in the last bits);
// one lane then adds the inertial terms, solves the 6x6 system and moves the body.
// Serially, a body's whole contact loop was one dependent chain per colour step (a box in a
// pile: 15-30 us); a warp per body cut the chain but left too few bodies in flight where a
// colour holds tens of thousands of them.  i == BB_NONE: the group only takes part in the
// shuffles (the trips over a colour's bodies are block-uniform).
// Bound: latency, the contacts of a colour's longest bodies one after the other, 100 to 250 dependent
// colour steps per substep.  Solve stage per substep, with poses and anchors gathered per visit
// and the solve on one lane in eight of 512-thread blocks -> now: 8.3 -> 3.3 ms on a 20k mixed
// pile (10 iterations), 6.9 -> 4.0 ms on 256 batched worlds (119k bodies, 4 iterations).  Tried and
// slower: the next contact's rows loaded, prefetched to L1 or staged by cp.async ahead of use.
// H is kept as its lower triangle, row-major: entry (a, b), b <= a, at a * (a + 1) / 2 + b.
#define AVBD_THREADS 128  // small blocks: a world of few bodies spreads over more SMs
#define AVBD_BODIES (AVBD_THREADS / AVBD_LANES)  // bodies of a block's trip
__device__ __forceinline__ int avbd_lt(int a, int b) { return a * (a + 1) / 2 + b; }
__device__ __forceinline__ void avbd_gather(const DevState& d, const Params& p, int cur, uint32_t i, float alpha, float* out) {
  const int lane = threadIdx.x & (AVBD_LANES - 1);
  float g[6], H[21];
#pragma unroll
  for (int a = 0; a < 6; ++a) g[a] = 0.f;
#pragma unroll
  for (int a = 0; a < 21; ++a) H[a] = 0.f;
  const uint32_t s0 = i == BB_NONE ? 0u : d.csr_start[cur][i], s1 = i == BB_NONE ? 0u : d.csr_start[cur][i + 1];
  float3 odp{}, odth{};
  if (i != BB_NONE) {
    odp = f3(d.iw[2 * size_t(i)]);
    odth = f3(d.iw[2 * size_t(i) + 1]);
  }
  for (uint32_t e = s0 + uint32_t(lane); e < s1; e += AVBD_LANES) {
    const uint2 en = avbd_entries(d)[e];
    const bool i1 = en.x >> 31, qa = (en.x >> 30) & 1u;
    const uint32_t q = en.x & 0x3FFFFFFFu, slot = en.y & 0x1FFFFFFFu;
    const int cc = int(en.y >> 29) + 1;
    const bool d1 = i1 || qa, d2 = !i1 || qa;
    const float3 n = f3(d.m_normal[cur][slot]);
    const float3 td[2] = {f3(d.m_t0[cur][slot]), f3(d.m_t1[cur][slot])};
    float3 qdp{}, qdth{};
    if (qa) {
      qdp = f3(d.iw[2 * size_t(q)]);
      qdth = f3(d.iw[2 * size_t(q) + 1]);
    }
    const AvbdDisp u = i1 ? AvbdDisp{odp, odth, qdp, qdth} : AvbdDisp{qdp, qdth, odp, odth};
    for (int j = 0; j < cc; ++j) {
      const uint32_t ci = slot * BB_MAX_CONTACTS + uint32_t(j);
      const AvbdRow r = avbd_row(d, ci);
      const float4 lam = d.c_lam[cur][ci];
      const float4 kt = d.c_kt[cur][ci];
      const float mu = r.r3.w;
      const float C = avbd_contact_C(r, u, d1, d2, alpha, n);
      const float f = fminf(lam.w * C + lam.x, 0.f);
      const float3 Jl = i1 ? -n : n;
      const float3 Ja = i1 ? -cross3(f3(r.r0), n) : cross3(f3(r.r1), n);
      const float J[6] = {Jl.x, Jl.y, Jl.z, Ja.x, Ja.y, Ja.z};
#pragma unroll
      for (int a = 0; a < 6; ++a) g[a] += f * J[a];
#pragma unroll
      for (int a = 0; a < 6; ++a)
#pragma unroll
        for (int bb = 0; bb <= a; ++bb) H[avbd_lt(a, bb)] += lam.w * J[a] * J[bb];
      const float bound = mu * fabsf(lam.x);
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const float Ct = avbd_dir_C(r, u, t == 0 ? r.r1.w : r.r2.w, p.avbd_stick_slop, d1, d2, alpha, td[t]);
        const float ktt = t == 0 ? kt.x : kt.y;
        const float lt = t == 0 ? lam.y : lam.z;
        const float ft = fminf(fmaxf(ktt * Ct + lt, -bound), bound);
        const float3 Jlt = i1 ? -td[t] : td[t];
        const float3 Jat = i1 ? -cross3(f3(r.r2), td[t]) : cross3(f3(r.r3), td[t]);
        const float Jt[6] = {Jlt.x, Jlt.y, Jlt.z, Jat.x, Jat.y, Jat.z};
#pragma unroll
        for (int a = 0; a < 6; ++a) g[a] += ft * Jt[a];
#pragma unroll
        for (int a = 0; a < 6; ++a)
#pragma unroll
          for (int bb = 0; bb <= a; ++bb) H[avbd_lt(a, bb)] += ktt * Jt[a] * Jt[bb];
      }
    }
  }
#pragma unroll
  for (int o = AVBD_LANES / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int a = 0; a < 6; ++a) g[a] += __shfl_xor_sync(0xFFFFFFFFu, g[a], o);
#pragma unroll
    for (int a = 0; a < 21; ++a) H[a] += __shfl_xor_sync(0xFFFFFFFFu, H[a], o);
  }
  if (lane != 0 || i == BB_NONE) return;
#pragma unroll
  for (int a = 0; a < 6; ++a) out[a * AVBD_BODIES] = g[a];
#pragma unroll
  for (int a = 0; a < 21; ++a) out[(6 + a) * AVBD_BODIES] = H[a];
}

// the step of body i from its summed gradient and Hessian: inertial terms, 6x6 solve, new pose
__device__ __forceinline__ void avbd_move(const DevState& d, const Params& p, uint32_t i, float dt, const float* sum) {
  float g[6], H[21];
#pragma unroll
  for (int a = 0; a < 6; ++a) g[a] = sum[a * AVBD_BODIES];
#pragma unroll
  for (int a = 0; a < 21; ++a) H[a] = sum[(6 + a) * AVBD_BODIES];
  const bool tq = p.quirks & BB_QUIRK_INERTIA_TRANSPOSE;
  const float inv_dt2 = dt > 0.f ? 1.0f / (dt * dt) : 0.f;
  const float m_lin = d.vel[i].w * inv_dt2;
  Quatf rot = q_from(d.rot[i]);
  Sym3 wi = body_world_inv_inertia(d.iinv, d.iinv_off, d.full_inertia != 0, i, rot, tq);
  // avbd_inverse3 (avbd.slang:309-326) of the symmetric world inverse inertia
  float3 c0 = make_float3(wi.xx, wi.xy, wi.xz), c1 = make_float3(wi.xy, wi.yy, wi.yz), c2 = make_float3(wi.xz, wi.yz, wi.zz);
  float3 r0 = cross3(c1, c2), r1 = cross3(c2, c0), r2 = cross3(c0, c1);
  float det = dot3(c0, r0);
  float inv = fabsf(det) > 1e-12f ? 1.0f / det : 0.f;
  r0 = r0 * inv;
  r1 = r1 * inv;
  r2 = r2 * inv;
  const float Iw[3][3] = {{r0.x, r0.y, r0.z}, {r1.x, r1.y, r1.z}, {r2.x, r2.y, r2.z}};
  H[avbd_lt(0, 0)] += m_lin;
  H[avbd_lt(1, 1)] += m_lin;
  H[avbd_lt(2, 2)] += m_lin;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int bb = 0; bb <= a; ++bb) H[avbd_lt(3 + a, 3 + bb)] += Iw[a][bb] * inv_dt2;
  const float3 dpos = f3(d.pos[i]) - f3(d.a_pos_tilde[i]);
  const float3 dth = small_angle_delta(rot, q_from(d.a_rot_tilde[i]));
  g[0] += m_lin * dpos.x;
  g[1] += m_lin * dpos.y;
  g[2] += m_lin * dpos.z;
  const float3 ga = make_float3(Iw[0][0] * dth.x + Iw[0][1] * dth.y + Iw[0][2] * dth.z,
                                Iw[1][0] * dth.x + Iw[1][1] * dth.y + Iw[1][2] * dth.z,
                                Iw[2][0] * dth.x + Iw[2][1] * dth.y + Iw[2][2] * dth.z) * inv_dt2;
  g[3] += ga.x;
  g[4] += ga.y;
  g[5] += ga.z;
  // avbd_solve6: in-place LDL^T, diagonal floor 1e-8
  float x[6], rhs[6];
#pragma unroll
  for (int a = 0; a < 6; ++a) rhs[a] = -g[a];
#pragma unroll
  for (int jj = 0; jj < 6; ++jj) {
    float dd = H[avbd_lt(jj, jj)];
#pragma unroll
    for (int kk = 0; kk < 6; ++kk)
      if (kk < jj) dd -= H[avbd_lt(jj, kk)] * H[avbd_lt(jj, kk)] * H[avbd_lt(kk, kk)];
    dd = fmaxf(dd, 1e-8f);
    H[avbd_lt(jj, jj)] = dd;
#pragma unroll
    for (int ii = 0; ii < 6; ++ii) {
      if (ii > jj) {
        float sm = H[avbd_lt(ii, jj)];
#pragma unroll
        for (int kk = 0; kk < 6; ++kk)
          if (kk < jj) sm -= H[avbd_lt(ii, kk)] * H[avbd_lt(jj, kk)] * H[avbd_lt(kk, kk)];
        H[avbd_lt(ii, jj)] = sm / dd;
      }
    }
  }
#pragma unroll
  for (int ii = 0; ii < 6; ++ii) {
    float sm = rhs[ii];
#pragma unroll
    for (int kk = 0; kk < 6; ++kk)
      if (kk < ii) sm -= H[avbd_lt(ii, kk)] * rhs[kk];
    rhs[ii] = sm;
  }
#pragma unroll
  for (int ii = 0; ii < 6; ++ii) rhs[ii] /= H[avbd_lt(ii, ii)];
#pragma unroll
  for (int ii = 5; ii >= 0; --ii) {
    float sm = rhs[ii];
#pragma unroll
    for (int kk = 0; kk < 6; ++kk)
      if (kk > ii) sm -= H[avbd_lt(kk, ii)] * x[kk];
    x[ii] = sm;
  }
  const float4 ps = d.pos[i];
  const float3 pn = make_float3(ps.x + x[0], ps.y + x[1], ps.z + x[2]);
  d.pos[i] = f4(pn, ps.w);
  Quatf dq{x[3] * 0.5f, x[4] * 0.5f, x[5] * 0.5f, 1.0f};
  const Quatf qn = q_normalize(q_mul(dq, rot));
  d.rot[i] = q_to4(qn);
  avbd_store_disp(d, i, pn - f3(d.a_pos_start[i]), small_angle_delta(qn, q_from(d.a_rot_start[i])));
}

// entry_avbd_dual (avbd.slang:728-808)
// lane l of a manifold's AVBD_DUAL_LANES lanes takes contacts l, l + AVBD_DUAL_LANES, ... (they are
// independent): neighbouring lanes read neighbouring 16 bytes of each plane
#define AVBD_DUAL_LANES 4
__device__ void avbd_dual(const DevState& d, const Params& p, int cur, uint32_t m, int lane) {
  const uint32_t slot = d.man_slot[cur][m];
  const uint2 b = d.m_bodies[cur][slot];
  const bool d1 = awake(d.flags[b.x]), d2 = awake(d.flags[b.y]);
  if (!d1 && !d2) return;
  const float3 n = f3(d.m_normal[cur][slot]);
  const float3 td[2] = {f3(d.m_t0[cur][slot]), f3(d.m_t1[cur][slot])};
  const int cc = d.m_keycc[cur][slot].y;
  AvbdDisp u{};
  if (d1) {
    u.dp1 = f3(d.iw[2 * size_t(b.x)]);
    u.dth1 = f3(d.iw[2 * size_t(b.x) + 1]);
  }
  if (d2) {
    u.dp2 = f3(d.iw[2 * size_t(b.y)]);
    u.dth2 = f3(d.iw[2 * size_t(b.y) + 1]);
  }
  for (int j = lane; j < cc; j += AVBD_DUAL_LANES) {
    const uint32_t ci = slot * BB_MAX_CONTACTS + j;
    const AvbdRow r = avbd_row(d, ci);
    const float mu = r.r3.w;
    const float C = avbd_contact_C(r, u, d1, d2, 1.0f, n);
    float4 lam = d.c_lam[cur][ci];
    float4 kt = d.c_kt[cur][ci];
    const float lam0 = lam.x, k = lam.w;
    float nl = fminf(k * C + lam0, 0.f);
    lam.x = nl;
    if (nl < 0.f) lam.w = fminf(k + p.avbd_beta * fabsf(C), p.avbd_k_max);
    const float bound = mu * fabsf(lam0);
    bool stick_ok = true;
    float drift2 = 0.f;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const float C0t = t == 0 ? r.r1.w : r.r2.w;
      const float Ct = avbd_dir_C(r, u, C0t, p.avbd_stick_slop, d1, d2, 1.0f, td[t]);
      float lt = t == 0 ? lam.y : lam.z;
      float ktt = t == 0 ? kt.x : kt.y;
      float nlt = fminf(fmaxf(ktt * Ct + lt, -bound), bound);
      if (t == 0) lam.y = nlt;
      else lam.z = nlt;
      if (nlt > -bound && nlt < bound) {
        float nk = fminf(ktt + p.avbd_beta * fabsf(Ct), p.avbd_k_max);
        if (t == 0) kt.x = nk;
        else kt.y = nk;
      } else {
        stick_ok = false;
      }
      drift2 += C0t * C0t;
    }
    uint32_t stick = (stick_ok && drift2 < p.avbd_stick_thresh * p.avbd_stick_thresh) ? 1u : 0u;
    d.c_lam[cur][ci] = lam;
    d.c_kt[cur][ci] = make_float4(kt.x, kt.y, __uint_as_float(stick), kt.w);
  }
}

// entry_avbd_finalize (avbd.slang:132-202)
__device__ void avbd_finalize(const DevState& d, int cur, uint32_t i, float dt) {
  const float inv_dt = dt > 0.f ? 1.0f / dt : 0.f;
  float4 v4 = d.vel[i];
  d.pvel[i] = v4;
  float3 v = (f3(d.pos[i]) - f3(d.a_pos_start[i])) * inv_dt;
  Quatf dq = q_mul(q_from(d.rot[i]), q_conj(q_from(d.a_rot_start[i])));
  float sg = dq.w < 0.f ? -1.f : 1.f;
  float3 w = make_float3(dq.x, dq.y, dq.z) * (2.0f * sg * inv_dt);
  if (dot3(v, v) < 0.09f && dot3(w, w) < 0.16f && d.csr_start[cur][i + 1] - d.csr_start[cur][i] >= 3u) {
    v = v * 0.9f;
    w = w * 0.9f;
  }
  d.vel[i] = f4(v, v4.w);
  d.omega[i] = f4(w, 0.f);
}

// One bucket of bodies, no two of which share a manifold: a block takes AVBD_BODIES of them per
// trip.  All lanes sum the contacts; then the block's first lanes solve one body each, so that
// the 6x6 solve (hundreds of instructions) is issued once per block and trip and not by every warp
// for its few bodies.  buf alternates, so a trip's sums are written while the last one's are solved.
__device__ __forceinline__ void avbd_bucket(const DevState& d, const Params& p, int cur, const uint32_t* list, uint32_t s0,
                                            uint32_t s1, float dt, float alpha, float* sums, uint32_t& trip) {
  for (uint32_t base = s0 + blockIdx.x * AVBD_BODIES; base < s1; base += gridDim.x * AVBD_BODIES, ++trip) {
    float* buf = sums + (trip & 1u) * 27 * AVBD_BODIES;
    const uint32_t k = base + threadIdx.x / AVBD_LANES;
    const bool mover = threadIdx.x < AVBD_BODIES && base + threadIdx.x < s1;
    const uint32_t mine = mover ? list[base + threadIdx.x] : 0u;
    avbd_gather(d, p, cur, k < s1 ? list[k] : BB_NONE, alpha, buf + threadIdx.x / AVBD_LANES);
    __syncthreads();
    if (mover) avbd_move(d, p, mine, dt, buf + threadIdx.x);
  }
}

// persistent solve: main iterations (colour sweeps + dual), finalize, post-stabilisation
__global__ void __launch_bounds__(AVBD_THREADS, 512 / AVBD_THREADS) k_avbd_solve(const DevState d, Params p, int cur,
                                                                                 uint32_t n, float dt, int phase) {
  __shared__ float sums[2 * 27 * AVBD_BODIES];
  __shared__ uint32_t bs[64 * BB_MAX_COLORS + 1];  // starts of the buckets that hold bodies, and their end
  __shared__ uint32_t s_nb;
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  uint32_t* sync = &d.ctr->sync_count[3 + phase];
  uint32_t ep = 0, trip = 0;
  const uint32_t keys = phase == 1 ? p.avbd_shock_layers * BB_MAX_COLORS : min(d.ctr->avbd_colors, uint32_t(BB_MAX_COLORS));
  const uint32_t* list = phase == 1 ? d.bucket_vals[0] : d.a_bucket_vals[1];
  const uint32_t* starts = phase == 1 ? d.a_bucket_start : d.bucket_start;
  if (threadIdx.x < 32u) {
    uint32_t c = 0;
    for (uint32_t k0 = 0; k0 < keys; k0 += 32u) {
      const uint32_t k = k0 + threadIdx.x;
      const uint32_t a = k < keys ? starts[k] : 0u;
      const bool full = k < keys && starts[k + 1] != a;
      const uint32_t m = __ballot_sync(0xFFFFFFFFu, full);
      if (full) bs[c + uint32_t(__popc(m & ((1u << threadIdx.x) - 1u)))] = a;
      c += uint32_t(__popc(m));
    }
    if (threadIdx.x == 0) {
      bs[c] = keys ? starts[keys] : 0u;
      s_nb = c;
    }
  }
  __syncthreads();
  const uint32_t nb = s_nb;
  // sweeps over the buckets, a barrier after each; after each of the main iterations the dual step
  const uint32_t sweeps = phase == 0 ? p.avbd_iterations : phase == 1 ? 1u : p.avbd_post_stab_sweeps - 1u;
  const float alpha = phase == 0 ? 1.0f : 0.0f;
  const uint32_t M = d.ctr->manifold_count;
  for (uint32_t sw = 0; sw < sweeps; ++sw) {
    for (uint32_t b = 0; b < nb; ++b) {
      avbd_bucket(d, p, cur, list, bs[b], bs[b + 1], dt, alpha, sums, trip);
      grid_sync(d.ctr, sync, ep);
    }
    if (phase == 0) {
      for (uint32_t m = tid / AVBD_DUAL_LANES; m < M; m += stride / AVBD_DUAL_LANES)
        avbd_dual(d, p, cur, m, int(threadIdx.x % AVBD_DUAL_LANES));
      grid_sync(d.ctr, sync, ep);
    }
  }
  if (phase == 0)
    for (uint32_t i = tid; i < n; i += stride)
      if (awake(d.flags[i])) avbd_finalize(d, cur, i, dt);
}

// The body lists of the colour sweeps (post = 0: a_bucket_vals[1], starts in bucket_start) and of the
// sweep over the support layers (post = 1: bucket_vals[0], starts in a_bucket_start).  Both stay
// until the solve ends: the last sweeps walk the colour lists again.  bucket_* are the edge
// colouring's arrays, which AVBD does not read after it.  Scratch: histogram region 2 or 3, status
// and tile-counter slots 7 or 8 and 9 (every one is zeroed once per substep and used once).
static void avbd_buckets(cudaStream_t s, const DevState& d, const Params& p, uint32_t n, const StepScratch& sc, int sms,
                         int post) {
  const int T = BB_THREADS;
  uint32_t blocks = (n + T - 1) / T;
  k_avbd_keys<<<blocks, T, 0, s>>>(d, p, n, post);
  uint32_t* keys[2] = {post ? d.bucket_keys[0] : d.a_bucket_keys[0], post ? d.bucket_keys[1] : d.a_bucket_keys[1]};
  uint32_t* vals[2] = {post ? d.bucket_vals[0] : d.a_bucket_vals[0], post ? d.bucket_vals[1] : d.a_bucket_vals[1]};
  const int slot = post ? 8 : 7;
  // colour keys fit one 8-bit digit (result in buffer 1), layer keys two (buffer 0)
  bb_launch_sort(s, keys, vals, nullptr, n, post ? 2 : 1, 0, sc.sort_hist + size_t(post ? 3 : 2) * BB_HIST_REGION,
                 sc.sort_status + size_t(slot) * sc.sort_tiles * 256, sc.sort_tile_ctr + slot, d.ctr, sms);
  const uint32_t nb = post ? p.avbd_shock_layers * BB_MAX_COLORS : BB_MAX_COLORS;
  k_lower_bounds<<<(nb + 1 + 127) / 128, 128, 0, s>>>(keys[post ? 0 : 1], n, post ? d.a_bucket_start : d.bucket_start, nb,
                                                      AVBD_CLASSES);
}

int bb_avbd_color_blocks(int sms) { return bb_coop_blocks((const void*)k_avbd_color, BB_COOP_THREADS, sms); }
// Blocks of k_avbd_solve: AVBD_THREADS threads, 512 per SM in all; for a world of n bodies as many
// as hold one thread per body (8 lanes for each body of the largest colour, about an eighth)
int bb_avbd_blocks(int sms, uint32_t max_bodies) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)k_avbd_solve, AVBD_THREADS, 0);
  per_sm = std::max(1, std::min(per_sm, 512 / AVBD_THREADS));
  const uint64_t want = (uint64_t(max_bodies) + AVBD_THREADS - 1) / AVBD_THREADS;
  return int(std::max<uint64_t>(1, std::min<uint64_t>(uint64_t(sms) * per_sm, want)));
}

void bb_solve_avbd(cudaStream_t s, const DevState& d, const Params& p, uint32_t n, float h, const StepScratch& sc,
                   int sms, int cur, int coop_blocks, int color_blocks) {
  if (n == 0) return;
  const int T = BB_THREADS;
  uint32_t blocks = (n + T - 1) / T;
  {
    DevState dd = d;
    Params pp = p;
    int cc = cur;
    uint32_t nn = n;
    void* args[] = {&dd, &pp, &cc, &nn};
    bb_launch_coop((const void*)k_avbd_color, color_blocks, BB_COOP_THREADS, args, s);
  }
  k_avbd_prepare<<<blocks, T, 0, s>>>(d, p, n, h);
  k_avbd_warmstart<<<sms * 8, T, 0, s>>>(d, p, cur);
  k_avbd_entries<<<blocks, T, 0, s>>>(d, n, cur);
  DevState dd = d;
  Params pp = p;
  int cc = cur;
  uint32_t nn = n;
  float hh = h;
  int phase = 0;
  void* args[] = {&dd, &pp, &cc, &nn, &hh, &phase};
  avbd_buckets(s, d, p, n, sc, sms, 0);
  bb_launch_coop((const void*)k_avbd_solve, coop_blocks, AVBD_THREADS, args, s);
  avbd_buckets(s, d, p, n, sc, sms, 1);
  int phase1 = 1;
  void* args1[] = {&dd, &pp, &cc, &nn, &hh, &phase1};
  bb_launch_coop((const void*)k_avbd_solve, coop_blocks, AVBD_THREADS, args1, s);
  if (p.avbd_post_stab_sweeps > 1) {
    int phase2 = 2;
    void* args2[] = {&dd, &pp, &cc, &nn, &hh, &phase2};
    bb_launch_coop((const void*)k_avbd_solve, coop_blocks, AVBD_THREADS, args2, s);
  }
}
