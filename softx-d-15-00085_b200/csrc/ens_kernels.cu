// ens_kernels.cu -- kernels of the ensemble path (see ens_kernels.cuh).
//
//   k_ens_hash     system-prefixed cell key per particle
//   [counting sort by cell and cell table, cell_sort.cu]
//   k_ens_reorder  move state, pid and wall history into sorted order
//   k_ens_nlist    27-cell Verlet list inside the particle's own system, carrying
//                  the tangential history of every surviving contact by partner pid
//   k_ens_step     pair law + walls + symplectic Euler, fused, gather only
//
// The contact model (per pair, with m* = ma mb / (ma + mb), R* = ra rb / (ra + rb),
// overlap d, unit normal n from b to a, v_n = (va - vb) . n):
//   linear        f_n = kn d - c_n v_n,  c_n = 2 beta sqrt(m* kn);  k_t = kt,
//                 c_t = 2 beta sqrt(m* kt)
//   Hertz-Mindlin S_n = 2 E* sqrt(R* d), f_n = 2/3 S_n d - c_n v_n,
//                 c_n = 2 sqrt(5/6) beta sqrt(S_n m*);  k_t = 8 G* sqrt(R* d),
//                 c_t = 2 sqrt(5/6) beta sqrt(k_t m*)
//   with beta = -ln e / sqrt(ln^2 e + pi^2); f_n is not clamped (the damping
//   may pull at the end of a contact, so the linear law rebounds with e).
//   Tangential: the history xi is turned into the tangent plane (length
//   kept), advanced by v_t dt, f_t = -k_t xi - c_t v_t, capped at
//   mu max(f_n, 0) (xi then set back to the spring length that gives the
//   capped force).  Rolling friction: a torque -mu_r max(f_n, 0) R* w_rel / |w_rel|.
//   Walls use the same law with R* = r, m* = m.
#include "ens_kernels.cuh"
#include "ens_device.cuh"
#include "dem_laws.cuh"

#include <algorithm>

namespace blaze {
namespace {

constexpr int kThreads = 256;

// ------------------------------------------------------------------- hash
__global__ void __launch_bounds__(kSortThreads)
k_ens_hash(EnsGeom g, StateBuf s0, StateBuf s1, const int* at, int n, CellSort cs, StepCtl* ctl,
           const int* gate) {
  if (gate && *gate == 0) return;
  const bool second = at && *at != 0;
  const float4* __restrict__ pos = second ? s1.pos : s0.pos;
  const float4* __restrict__ vel = second ? s1.vel : s0.vel;
  const int i = blockIdx.x * kSortThreads + threadIdx.x;
  const bool valid = i < n;
  uint32_t st = 0, key = 0;
  if (valid) {
    const uint32_t sys = __float_as_uint(vel[i].w) & kSysMask;
    const EnsSysDev& S = g.sys[sys];
    const int3 c = ens_cell(S, xyz(pos[i]));
    if (ens_in(S, c)) {
      key = ens_key(S, c);
    } else {
      key = g.ncell_tab;
      st = kStatusOutOfGrid;
    }
  }
  cell_count(cs, i, valid, key);
  ens_flag(ctl, st);
}

// ---------------------------------------------------------------- reorder
// (the place pass before it has already counted the re-sort: the old lists
// are those of the other parity)
__global__ void __launch_bounds__(kSortThreads)
k_ens_reorder(StateBuf s0, StateBuf s1, const int* at, StateBuf dst, EnsBufs b, int n, CellSort cs,
              const StepCtl* ctl, const int* gate) {
  if (gate && *gate == 0) return;
  const StateBuf src = at && *at != 0 ? s1 : s0;
  const int j = blockIdx.x * kSortThreads + threadIdx.x;
  const bool valid = j < n;
  const int i = cell_dest(cs, j, valid);
  if (!valid) return;
  const int e = (ctl->epoch & 1) ^ 1;
  const float4 x = src.pos[j];
  dst.pos[i] = x;
  const float4 v = src.vel[j];
  dst.vel[i] = v;
  float4 w = src.angv[j];
  if (x.w < 0.0f) {   // a polyhedron: angv.w is its id; its path restarts per id
    const int pq = __float_as_int(w.w);
    b.pat[pq] = i;
    b.ppath[pq] = 0.0f;
  } else {
    w.w = 0.0f;
  }
  dst.angv[i] = w;
  b.pid[e ^ 1][i] = b.pid[e][j];
  if ((__float_as_uint(v.w) >> kSysBits) != 0u) {
#pragma unroll
    for (int q = 0; q < kWallSlots; ++q)
      b.wh[e ^ 1][(size_t)q * b.stride + i] = b.wh[e][(size_t)q * b.stride + j];
  }
}

// ------------------------------------------------------------------ nlist
// Pairs with |xi - xj|^2 < (ri + rj + skin)^2 from the 27 surrounding cells
// of the particle's own system (z, y, x order; j ascending inside a cell).
// The history of a slot of the old list moves to the new slot of the same
// partner (matched by pid).  Rows of three cells are ranges of the cell
// table, walked as one sequence of candidates with the next position loaded
// ahead; rows and end cells out of reach are left out (see k_nlist): a
// partner's radius is at most (cell - skin) / 2 (blaze_ens_set_state), so the
// reach is ra + (cell + skin) / 2.
constexpr int kNlistThreads = 128;
__global__ void __launch_bounds__(kNlistThreads)
k_ens_nlist(EnsGeom g, EnsBufs b, const float4* __restrict__ pos, const float4* __restrict__ vel,
            int n, const int32_t* __restrict__ perm, const uint32_t* __restrict__ start,
            StepCtl* ctl, const int* gate) {
  if (gate && *gate == 0) return;
  __shared__ uint2 row[9][kNlistThreads];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int e = (ctl->epoch & 1) ^ 1;
  const EnsList Lo = b.L[e], Ln = b.L[e ^ 1];
  const int* pid_old = b.pid[e];
  const int* pid_new = b.pid[e ^ 1];
  const size_t stride = (size_t)b.stride;
  const float4 pa4 = pos[i];
  if (pa4.w < 0.0f) {   // a polyhedron: its neighbours are listed by k_mix_plist
    Ln.cnt[i] = 0;
    Ln.mask[i] = 0;
    return;
  }
  const float3 pa = xyz(pa4);
  const float ra = pa4.w;
  const uint32_t sys = __float_as_uint(vel[i].w) & kSysMask;
  const EnsSysDev& S = g.sys[sys];
  const int3 c = ens_cell(S, pa);
  const int io = perm[i];
  const uint32_t cnt_o = Lo.cnt[io];
  const uint32_t mask_o = Lo.mask[io];
  uint32_t cnt = 0, mask = 0, st = 0;
  int rows = 0;
  if (ens_in(S, c)) {
    const float reach = (ra + 0.5f * (S.cell + g.skin)) * (1.0f + 1e-5f);
    const float lim = reach * reach;
    const float2 dx = cell_gap(pa.x, S.origin.x, S.cell, c.x, S.nc.x);
    const float2 dy = cell_gap(pa.y, S.origin.y, S.cell, c.y, S.nc.y);
    const float2 dz = cell_gap(pa.z, S.origin.z, S.cell, c.z, S.nc.z);
#pragma unroll
    for (int z = -1; z <= 1; ++z) {
      const float gz = z < 0 ? dz.x : (z > 0 ? dz.y : 0.0f);
      if (c.z + z < 0 || c.z + z >= S.nc.z || gz * gz > lim) continue;
#pragma unroll
      for (int y = -1; y <= 1; ++y) {
        const float gy = y < 0 ? dy.x : (y > 0 ? dy.y : 0.0f);
        const float yz = gy * gy + gz * gz;
        if (c.y + y < 0 || c.y + y >= S.nc.y || yz > lim) continue;
        const int x0 = c.x == 0 || yz + dx.x * dx.x > lim ? c.x : c.x - 1;
        const int x1 = c.x == S.nc.x - 1 || yz + dx.y * dx.y > lim ? c.x : c.x + 1;
        const uint32_t h = S.cell_off + (uint32_t)(S.nc.x * (c.y + y + S.nc.y * (c.z + z)));
        const uint32_t s0 = __ldg(start + h + (uint32_t)x0);
        const uint32_t s1 = __ldg(start + h + (uint32_t)x1 + 1u);
        if (s0 < s1) row[rows++][threadIdx.x] = make_uint2(s0, s1);
      }
    }
  } else {
    st |= kStatusOutOfGrid;
  }
  if (rows > 0) {
    uint2 q = row[0][threadIdx.x];
    int r = 1;
    uint32_t jn = q.x;
    float4 pn = __ldg(pos + jn);
    for (bool more = true; more;) {
      const uint32_t j = jn;
      const float4 pb = pn;
      if (++jn == q.y) {
        more = r < rows;
        if (more) {
          q = row[r++][threadIdx.x];
          jn = q.x;
        }
      }
      if (more) pn = __ldg(pos + jn);
      if ((int)j == i) continue;
      const float3 rel = pa - xyz(pb);
      const float lim = (ra + fabsf(pb.w)) + g.skin;   // a polyhedron: its bounding radius
      if (!(dot3(rel, rel) < lim * lim)) continue;
      if (cnt < (uint32_t)b.cap) {
        Ln.idx[cnt * stride + i] = j;
        uint8_t from = 0xffu;
        uint32_t mo = mask_o;
        if (mo) {
          const int pj = pid_new[j];
          while (mo) {
            const int ko = __ffs(mo) - 1;
            mo &= mo - 1u;
            if ((uint32_t)ko >= cnt_o) break;
            const size_t so = (size_t)ko * stride + io;
            if (pid_old[Lo.idx[so]] == pj) {
              const size_t sn = (size_t)cnt * stride + i;
              Ln.hx[sn] = Lo.hx[so];
              Ln.hy[sn] = Lo.hy[so];
              Ln.hz[sn] = Lo.hz[so];
              mask |= 1u << cnt;
              from = (uint8_t)ko;
              break;
            }
          }
        }
        if (Ln.src) Ln.src[cnt * stride + i] = from;
      } else {
        st |= kStatusListOverflow;
      }
      ++cnt;
    }
  }
  Ln.cnt[i] = cnt < (uint32_t)b.cap ? cnt : (uint32_t)b.cap;
  Ln.mask[i] = mask;
  ens_flag(ctl, st);
}

// ------------------------------------------------------------------- step
// candidate slots tested per batch of independent loads in the contact pass
constexpr uint32_t kEnsMaskBatch = 4;
// A neighbour's state: through the read-only cache (kNc) when the state
// cannot change during the kernel, else a plain load (the persistent kernel
// reads, after a grid barrier, what other blocks wrote in the same launch).
template <bool kNc>
__device__ __forceinline__ float4 ld_state(const float4* p) {
  if constexpr (kNc) return __ldg(p);
  else return *p;
}

// ----------------------------------------------------- reference law (3)
// The reference's sphere step, per particle, with the parameters its
// parser derives for a particle object formed here from the particle's own
// radius and the system's constants:
//   mass     m = (4/3 pi density) r^3 in double, rounded once
//            (KSimulationData.cpp:1096); 1/I = 1 / (0.4 r r m) in float
//            (main.cpp:622-626)
//   pairs    Kn = kn, Cn = (ref_a sqrt(Kn m*)) / ref_b in double with
//            m* = 1 / (1/ma + 1/mb) (KSimulationData.cpp:955-1016), kinetic
//            friction mu
//   planes   Kn = kn, Cn the same with m* = m (KSimulationData.cpp:1019-1047),
//            static friction mu_wall
// The contact test and penetration (|d| - (ra + rb), plus 1e-5), the laws
// (Collision_Response.cuh:374-494 and 4-109) and the integration
// (Integrate_Euler_NonSymmetry, Integration.cuh:6-184, rolling resistance
// mu_roll) are the sphere path's own functions; a plane is tested as the
// reference tests a face (Collision_Detection_Spheres.cuh:6-100) against
// its point d n.  The law keeps no history.
__device__ __forceinline__ float ref_mass(const EnsSysDev& S, float r) {
  const double r3 = ((double)r * (double)r) * (double)r;
  return (float)(S.ref_m * r3);
}

__device__ __forceinline__ float ref_damping(const EnsSysDev& S, double m) {
  return S.ref_b > 0.0 ? (float)((S.ref_a * sqrt((double)S.kn * m)) / S.ref_b) : 0.0f;
}

template <bool kCapture, bool kNc>
__device__ __forceinline__ float ens_particle_step_ref(const EnsGeom& g, const EnsBufs& b,
                                                       const StateBuf& in, const StateBuf& out,
                                                       int i, const EnsList& L,
                                                       const EnsCapture& cap, uint32_t& st) {
  const size_t stride = (size_t)b.stride;
  const float dt = g.dt;
  const float4 pa4 = in.pos[i], va4 = in.vel[i], wa4 = in.angv[i];
  const float3 pa = xyz(pa4), va = xyz(va4), wa = xyz(wa4);
  const float ra = pa4.w;
  const uint32_t sys = __float_as_uint(va4.w) & kSysMask;
  const EnsSysDev& S = g.sys[sys];
  const float ma = ref_mass(S, ra);
  SimParams P;   // the two fields the reference's laws read
  P.dt = dt;
  P.rotation = 1;

  // particle-particle (Kernel_ParticleInteraction_Spheres_NonSymmetry)
  float3 f = S.gravity * ma;
  float3 tl = f3(0.0f, 0.0f, 0.0f);
  const uint32_t cnt = L.cnt[i];
  for (uint32_t k = 0; k < cnt; ++k) {
    const uint32_t j = L.idx[(size_t)k * stride + i];
    const float4 pb4 = ld_state<kNc>(in.pos + j);
    const float3 rel = pa - xyz(pb4);
    const float rb = pb4.w;
    if (!touches(rel, ra + rb)) continue;
    const float dist = len3(rel);
    const float dis = fabsf(dist - (ra + rb)) + 0.000010f;
    const float3 nrm = div3_rn(rel, dist);
    const float4 vb4 = ld_state<kNc>(in.vel + j), wb4 = ld_state<kNc>(in.angv + j);
    const float mb = ref_mass(S, rb);
    PP_Parms pp;
    pp.Kn = S.kn;
    pp.Cn = ref_damping(S, 1.0 / ((1.0 / (double)ma) + (1.0 / (double)mb)));
    pp.Fric_static = S.mu;
    pp.Fric_kinetic = S.mu;
    const Forces F = law_pp<true>(P, va - xyz(vb4), nrm, dis, (-1.0f * nrm) * ra, nrm * rb, wa,
                                  xyz(wb4), pp, va, xyz(vb4), ma, mb);
    f = f + F.trans;
    tl = tl + F.torque;
  }

  // plane walls (WorldObject_InteractionParticle, face and plane contacts)
  float3 fw = f3(0.0f, 0.0f, 0.0f), tw = f3(0.0f, 0.0f, 0.0f);
  TypeParams T;
  T.mass = ma;
  T.s_kn = S.kn;
  T.s_cn = ref_damping(S, (double)ma);
  T.s_mus = S.mu_w;
  for (int w = S.wall0; w < S.wall0 + S.nwall; ++w) {
    const EnsWallDev& W = g.walls[w];
    const float3 n = W.a;
    const float3 c = n * W.r;
    const float3 pt = pa - ra * n;
    float dis = dot3(n, pt - c);
    if (!(dis < 0.000000f && dis > -ra)) continue;
    dis = fabsf(dis);
    const Forces F = law_static_surface(P, va, n, dis, pt - pa, wa, T);
    fw = fw + F.trans;
    tw = tw + F.torque;
  }

  // Integrate_Euler_NonSymmetry (Integration.cuh:6-184), spheres
  float3 acc = fw + f;
  acc = acc * (1.0f / ma);
  const float3 v = va + acc * dt;
  const float3 p = pa + v * dt;
  const float3 tq = tl + tw;
  float3 w = wa;
  if (dot3(tq, tq) > 0.0f) {
    const float iinv = 1.0f / (((0.4f * ra) * ra) * ma);
    const float3 aa = iinv * tq;
    w = w + aa * dt;
    w = w - w * S.mu_r;
  }
  const float path = wa4.w + len3(v) * dt;
  out.pos[i] = make_float4(p.x, p.y, p.z, ra);
  out.vel[i] = make_float4(v.x, v.y, v.z, __uint_as_float(sys));
  out.angv[i] = make_float4(w.x, w.y, w.z, path);
  if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z))) st |= kStatusNonFinite;
  if (kCapture) {
    const float3 fc = (f - S.gravity * ma) + fw;
    cap.f[i] = make_float4(fc.x, fc.y, fc.z, 0.0f);
    cap.t[i] = make_float4(tq.x, tq.y, tq.z, 0.0f);
  }
  return path;
}


// ------------------------------------------------ contacts shared by a warp
// A warp's 32 particles have 0 to a dozen contacts each, and the law is some
// 400 instructions: with every lane walking its own contacts the warp ran as
// long as its busiest particle with 16 of 32 lanes at work (60 % issue).  So
// the lanes first find their contacts, then the warp takes all of them 32 at
// a time, whoever they belong to, and each particle adds up its own in slot
// order, which gives the same sums.  The contacts are taken by rank (every
// particle's first, every particle's second, ...), so that lanes side by
// side mostly read and write the history of the same slot.  Wall contacts
// (a few particles of a warp, for one wall after the other) go the same way.
// Per 32 steps: hopper of 400,000 spheres 3.56 -> 2.66 ms, settled boxes of
// 2,000,000 14.0 -> 11.5 ms, mixed charge of 21,000 1.67 -> 1.49 ms.
constexpr int kPairChunk = 96;     // pair contacts in shared memory at a time
constexpr int kWallChunk = 64;     // wall contacts
constexpr int kContactWords = 624; // shared words per warp
static_assert(6 * kPairChunk + kPairChunk / 2 <= kContactWords && 9 * kWallChunk <= kContactWords,
              "contact buffer");
constexpr size_t contact_bytes(int threads) {
  return (size_t)(threads / 32) * kContactWords * sizeof(uint32_t);
}
constexpr unsigned kAll = 0xffffffffu;

// The step of particle i (every lane of a warp calls it, the lanes of valid
// particles first and with consecutive i): its contacts in list order (tangential histories updated in
// place, the particle's own slots only), its walls, symplectic Euler from
// `in` into `out`.  Raises status bits in st; returns the path
// the particle has moved since the last re-sort.  kRecord: also writes what
// the step reads into the tape view (histories to hrec when it is not null).
// kMix: the system holds polyhedra (linear law): a polyhedron's own entry is
// skipped (k_mix_poly_step steps it); a polyhedron neighbour's contact force
// and torque are the ones k_mix_poly_step left for this sphere (MixView),
// added in slot order.  sh: kContactWords of shared memory of this warp.
template <int kLaw, bool kCapture, bool kRecord, bool kCurved, bool kNc = true, bool kRot = false,
          bool kMix = false>
__device__ __forceinline__ float ens_particle_step(const EnsGeom& g, const EnsBufs& b,
                                                   const StateBuf& in, const StateBuf& out,
                                                   int i, bool valid, int e, const EnsList& L,
                                                   TapeView tv, float* hrec,
                                                   const EnsCapture& cap, uint32_t& st,
                                                   uint32_t* sh) {
  if constexpr (kLaw == kLawReference) {
    return valid ? ens_particle_step_ref<kCapture, kNc>(g, b, in, out, i, L, cap, st) : 0.0f;
  } else {
  const size_t stride = (size_t)b.stride;
  const float dt = g.dt;
  const int lane = threadIdx.x & 31;
  const int iw = i - lane;              // the warp's first particle
  const unsigned below = (1u << lane) - 1u;
  float4 pa4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), va4 = pa4, wa4 = pa4;
  if (valid) {
    pa4 = in.pos[i];
    va4 = in.vel[i];
    if constexpr (kRecord) wa4 = in.angv[i];
  }
  if constexpr (kMix) valid = valid && !(pa4.w < 0.0f);
  const float3 pa = xyz(pa4);
  const float ra = pa4.w;
  const uint32_t bits = __float_as_uint(va4.w);
  const uint32_t sys = bits & kSysMask;
  const uint32_t wmask_o = valid ? bits >> kSysBits : 0u;
  const EnsSysDev& S = g.sys[sys];

  // particle-particle contacts: the candidates in batches (all index loads
  // of a batch, then all position gathers, then the tests)
  float3 f = f3(0.0f, 0.0f, 0.0f), t = f3(0.0f, 0.0f, 0.0f);
  const uint32_t cnt = valid ? L.cnt[i] : 0u;
  const uint32_t mask_o = valid ? L.mask[i] : 0u;
  if constexpr (kRecord) {
    if (valid) {
      tv.pos[i] = pa4;
      tv.vel[i] = va4;
      tv.angv[i] = wa4;
      tv.mask[i] = mask_o;
    }
  }
  uint32_t mask = 0;
  uint32_t cmask = 0;
  for (uint32_t k0 = 0; k0 < cnt; k0 += kEnsMaskBatch) {
    uint32_t jj[kEnsMaskBatch];
#pragma unroll
    for (uint32_t u = 0; u < kEnsMaskBatch; ++u)
      jj[u] = k0 + u < cnt ? __ldg(L.idx + (size_t)(k0 + u) * stride + i) : 0u;
    float4 pb[kEnsMaskBatch];
#pragma unroll
    for (uint32_t u = 0; u < kEnsMaskBatch; ++u)
      pb[u] = k0 + u < cnt ? ld_state<kNc>(in.pos + jj[u]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (uint32_t u = 0; u < kEnsMaskBatch; ++u) {
      const float3 rel = pa - xyz(pb[u]);
      const float sr = ra + (kMix ? fabsf(pb[u].w) : pb[u].w);
      const float d2 = dot3(rel, rel);
      if (k0 + u < cnt && d2 < sr * sr && d2 > 0.0f) cmask |= 1u << (k0 + u);
    }
  }
  const int mine = __popc(cmask);
  const int total = __reduce_add_sync(kAll, mine);
  float* shf = reinterpret_cast<float*>(sh);
  uint16_t* con = reinterpret_cast<uint16_t*>(sh + 6 * kPairChunk);   // lane | slot << 5 | polyhedron << 14 | contact << 15
  // the law of slot k of the warp's particle o, by one lane
  auto pair = [&](int o, uint32_t k, uint32_t mo, float* ho, float3& F, float3& T) -> uint32_t {
    const int io = iw + o;
    const size_t sk = (size_t)k * stride + io;
    const uint32_t j = L.idx[sk];
    const float4 xo = ld_state<kNc>(in.pos + io), xj = ld_state<kNc>(in.pos + j);
    const float4 wj = ld_state<kNc>(in.angv + j);
    if constexpr (kMix) {
      if (xj.w < 0.0f) {
        const uint32_t tw = g.mix.twin[sk];
        if (tw == 0xffu) return 0u;
        const size_t sq = (size_t)tw * (size_t)g.mix.npoly + (size_t)__float_as_int(wj.w);
        const float4 F4 = g.mix.sf[sq];
        if (F4.w == 0.0f) return 0u;
        F = xyz(F4);
        T = xyz(g.mix.st[sq]);
        return 0xc000u;
      }
    }
    const float4 vo = ld_state<kNc>(in.vel + io), wo = ld_state<kNc>(in.angv + io);
    const float4 vj = ld_state<kNc>(in.vel + j);
    const float ro = xo.w, rj = xj.w;
    const float3 rel = xyz(xo) - xyz(xj);
    const float3 nrm = rel * (1.0f / sqrtf(dot3(rel, rel)));
    // the contact is decided by the overlap itself: the FP32 test above can
    // pass a pair whose FP64-formed overlap is not positive
    const float delta = overlap_pair(ro, rj, xyz(xo), xyz(xj));
    if (!(delta > 0.0f)) return 0u;
    float3 xi = f3(0.0f, 0.0f, 0.0f);
    if ((mo >> k) & 1u) {
      xi = f3(L.hx[sk], L.hy[sk], L.hz[sk]);
      if constexpr (kRecord) {
        if (ho) {
          float* h = ho + 3 * __popc(mo & ((1u << k) - 1u));
          h[0] = xi.x;
          h[1] = xi.y;
          h[2] = xi.z;
        }
      }
    }
    const EnsSysDev& So = g.sys[__float_as_uint(vo.w) & kSysMask];
    const float mp = sphere_mass(So, ro), mq = sphere_mass(So, rj);
    const float rs = (ro * rj) / (ro + rj);
    const float ms = (mp * mq) / (mp + mq);
    const float3 vcpa = xyz(vo) + cross3(xyz(wo), nrm * (-ro));
    const float3 vcpb = xyz(vj) + cross3(xyz(wj), nrm * rj);
    contact_law<kLaw>(So, So.mu, nrm, delta, rs, ms, xyz(vo) - xyz(vj), vcpa - vcpb,
                      xyz(wo) - xyz(wj), ro, dt, xi, F, T);
    L.hx[sk] = xi.x;
    L.hy[sk] = xi.y;
    L.hz[sk] = xi.z;
    return 0x8000u;
  };
  // row m: every particle's contact of rank m; m0 the first row that reaches
  // into the chunk, which starts at contact row0
  int m0 = 0, row0 = 0;
  for (int c0 = 0; c0 < total; c0 += kPairChunk) {
    const int nc = min(kPairChunk, total - c0);
    int m1 = m0, row1 = row0;
    uint32_t cm = cmask;   // this lane's contacts from row m on
    uint32_t cm1 = cm;
    for (int m = m0, row = row0 - c0; row < nc; ++m) {
      const unsigned bal = __ballot_sync(kAll, mine > m);
      if (mine > m) {
        const int c = row + __popc(bal & below);
        if (c >= 0 && c < nc) con[c] = (uint16_t)(lane | (__ffs(cm) - 1) << 5);
        cm &= cm - 1u;
      }
      row += __popc(bal);
      if (row <= nc) {
        m1 = m + 1;
        row1 = row + c0;
        cm1 = cm;
      }
    }
    cmask = cm1;
    __syncwarp();
    for (int r0 = 0; r0 < nc; r0 += 32) {
      const int r = r0 + lane;
      const uint32_t v = r < nc ? con[r] : (uint32_t)lane;
      const uint32_t mo = __shfl_sync(kAll, mask_o, (int)(v & 31u));
      float* ho = nullptr;
      if constexpr (kRecord)
        ho = reinterpret_cast<float*>(
            __shfl_sync(kAll, reinterpret_cast<unsigned long long>(hrec), (int)(v & 31u)));
      if (r < nc) {
        float3 F, T;
        const uint32_t hit = pair((int)(v & 31u), v >> 5, mo, ho, F, T);
        if (hit) {
          shf[r] = F.x;
          shf[kPairChunk + r] = F.y;
          shf[2 * kPairChunk + r] = F.z;
          shf[3 * kPairChunk + r] = T.x;
          shf[4 * kPairChunk + r] = T.y;
          shf[5 * kPairChunk + r] = T.z;
          con[r] = (uint16_t)(v | hit);
        }
      }
    }
    __syncwarp();
    for (int m = m0, row = row0 - c0; row < nc; ++m) {
      const unsigned bal = __ballot_sync(kAll, mine > m);
      const int c = row + __popc(bal & below);
      if (mine > m && c >= 0 && c < nc) {
        const uint32_t v = con[c];
        if (v & 0x8000u) {
          f = f + f3(shf[c], shf[kPairChunk + c], shf[2 * kPairChunk + c]);
          t = t + f3(shf[3 * kPairChunk + c], shf[4 * kPairChunk + c], shf[5 * kPairChunk + c]);
          if (!kMix || !(v & 0x4000u)) mask |= 1u << (v >> 5 & 31u);
        }
      }
      row += __popc(bal);
    }
    __syncwarp();
    m0 = m1;
    row0 = row1;
  }
  if (mask != mask_o) L.mask[i] = mask;
  if constexpr (kRecord) {
    if (valid) tv.cmask[i] = mask;
  }

  // walls: old history slots (by wall id) held in registers; new slots are
  // written in processing order straight over the old ones
  float4 oh[kWallSlots];
#pragma unroll
  for (int q = 0; q < kWallSlots; ++q) oh[q] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
  if (wmask_o) {
#pragma unroll
    for (int q = 0; q < kWallSlots; ++q)
      if ((wmask_o >> q) & 1u) oh[q] = b.wh[e][(size_t)q * stride + i];
    if constexpr (kRecord) {
      if (hrec) {
        float* h = hrec + 3 * __popc(mask_o);
#pragma unroll
        for (int q = 0; q < kWallSlots; ++q)
          if ((wmask_o >> q) & 1u) {
            float* hq = h + 4 * __popc(wmask_o & ((1u << q) - 1u));
            hq[0] = oh[q].x;
            hq[1] = oh[q].y;
            hq[2] = oh[q].z;
            hq[3] = oh[q].w;
          }
      }
    }
  }
  int nw = 0;       // this particle's wall contacts
  int held = 0;     // the warp's wall contacts in shared memory
  // a turning drum (kCurved only): its triangles are tested in the drum's
  // frame, where they stand still, and the normals turned back; triangles
  // and cylinders move with the turn
  bool rot = false;
  float rc = 1.0f, rsn = 0.0f;
  if constexpr (kCurved && kRot) {
    if (S.rot) {
      rot = true;
      const float2 cs = g.rot[sys];
      rc = cs.x;
      rsn = cs.y;
    }
  }
  // words of a held contact, kWallChunk apart: normal, overlap, history, wall
  // id, lane | history slot << 8 | moving << 16; the law leaves force and
  // torque in the first six
  auto wall_flush = [&]() {
    __syncwarp();
    for (int r = lane; r < held; r += 32) {
      const float3 nrm = f3(shf[r], shf[kWallChunk + r], shf[2 * kWallChunk + r]);
      const float delta = shf[3 * kWallChunk + r];
      float3 xi = f3(shf[4 * kWallChunk + r], shf[5 * kWallChunk + r], shf[6 * kWallChunk + r]);
      const uint32_t id = sh[7 * kWallChunk + r], meta = sh[8 * kWallChunk + r];
      const int io = iw + (int)(meta & 31u);
      const uint32_t slot = (meta >> 8) & 0xffu;
      const float4 xo = ld_state<kNc>(in.pos + io), vo = ld_state<kNc>(in.vel + io);
      const float4 wo = ld_state<kNc>(in.angv + io);
      const EnsSysDev& So = g.sys[__float_as_uint(vo.w) & kSysMask];
      const float ro = xo.w, mp = sphere_mass(So, ro);
      const float3 vcpa = xyz(vo) + cross3(xyz(wo), nrm * (-ro));
      float3 vr = xyz(vo), vc = vcpa, wr = xyz(wo);
      if (meta >> 16) {
        // the wall's velocity at the contact point, and its spin
        const float3 vw = cross3(So.rot_a, (xyz(xo) - nrm * ro) - So.rot_o) * So.rot_w;
        vr = vr - vw;
        vc = vcpa - vw;
        wr = wr - So.rot_a * So.rot_w;
      }
      float3 F, T;
      contact_law<kLaw>(So, So.mu_w, nrm, delta, ro, mp, vr, vc, wr, ro, dt, xi, F, T);
      if (slot < (uint32_t)kWallSlots)
        b.wh[e][(size_t)slot * stride + io] = make_float4(xi.x, xi.y, xi.z, __uint_as_float(id));
      shf[r] = F.x;
      shf[kWallChunk + r] = F.y;
      shf[2 * kWallChunk + r] = F.z;
      shf[3 * kWallChunk + r] = T.x;
      shf[4 * kWallChunk + r] = T.y;
      shf[5 * kWallChunk + r] = T.z;
    }
    __syncwarp();
    for (int r = 0; r < held; ++r)
      if ((int)(sh[8 * kWallChunk + r] & 31u) == lane) {
        f = f + f3(shf[r], shf[kWallChunk + r], shf[2 * kWallChunk + r]);
        t = t + f3(shf[3 * kWallChunk + r], shf[4 * kWallChunk + r], shf[5 * kWallChunk + r]);
      }
    __syncwarp();
    held = 0;
  };
  auto wall_contact = [&](bool hit, int id, float3 nrm, float delta, bool moving) {
    const unsigned bal = __ballot_sync(kAll, hit);
    if (!bal) return;
    if (held + __popc(bal) > kWallChunk) wall_flush();
    if (hit) {
      const int r = held + __popc(bal & below);
      float3 xi = f3(0.0f, 0.0f, 0.0f);
#pragma unroll
      for (int q = 0; q < kWallSlots; ++q)
        if (__float_as_int(oh[q].w) == id) xi = f3(oh[q].x, oh[q].y, oh[q].z);
      shf[r] = nrm.x;
      shf[kWallChunk + r] = nrm.y;
      shf[2 * kWallChunk + r] = nrm.z;
      shf[3 * kWallChunk + r] = delta;
      shf[4 * kWallChunk + r] = xi.x;
      shf[5 * kWallChunk + r] = xi.y;
      shf[6 * kWallChunk + r] = xi.z;
      sh[7 * kWallChunk + r] = (uint32_t)id;
      sh[8 * kWallChunk + r] = (uint32_t)lane | (uint32_t)min(nw, 255) << 8 | (moving ? 1u << 16 : 0u);
      if (nw < kWallSlots) ++nw;
      else st |= kStatusListOverflow;
    }
    held += __popc(bal);
  };
  // Planes only: most warps are near no wall, so every lane first takes its
  // walls' conservative test alone, and only walls that some lane is near are
  // met by the warp.  With the vote and the full test at every wall a loose bed
  // of 400,000 took 17.3 us a step instead of 15.2, one of 2,000,000 74 instead
  // of 67, and 512 beds of 7.4 million settling from rest 343 instead of 259.
  // With a mesh, where most walls are triangles (below), it costs more than it
  // gives: hopper of 400,000, 82 against 79 us.
  const int nwall = valid ? S.nwall : 0;
  const int nwall_most = __reduce_max_sync(kAll, nwall);
  if constexpr (kCurved) {
    for (int w = 0; w < nwall_most; ++w) {
      float3 nrm = f3(0.0f, 0.0f, 0.0f);
      float delta = 0.0f;
      int region;
      bool hit = false, moving = false;
      if (w < nwall) {
        const EnsWallDev& W = g.walls[S.wall0 + w];
        hit = wall_touch<kCurved>(W, pa, ra, nrm, delta, region);
        moving = rot && W.turning;
      }
      wall_contact(hit, S.wall0 + w, nrm, delta, moving);
    }
  } else {
    for (int w0 = 0; w0 < nwall_most; w0 += 32) {
      const int first = S.wall0 + w0, wn = min(32, nwall - w0);
      uint32_t near = 0u;
      for (int w = 0; w < wn; ++w)
        if (plane_near(g.walls[first + w], pa, ra)) near |= 1u << w;
      for (uint32_t any = __reduce_or_sync(kAll, near); any; any &= any - 1u) {
        const int w = __ffs(any) - 1;
        float3 nrm = f3(0.0f, 0.0f, 0.0f);
        float delta = 0.0f;
        int region;
        const bool hit = (near >> w & 1u) != 0u &&
                         wall_touch<kCurved>(g.walls[first + w], pa, ra, nrm, delta, region);
        wall_contact(hit, first + w, nrm, delta, false);   // only curved builds turn
      }
    }
  }
  if (kCurved && g.tri_off) {
    const float3 pd = rot ? S.rot_o + rot_about(S.rot_a, rc, -rsn, pa - S.rot_o) : pa;
    uint32_t o0 = 0, o1 = 0;
    if (valid) {
      const int3 c = ens_scell(S, pd);
      if (ens_sin(S, c)) {
        const uint32_t h = ens_skey(S, c);
        o0 = __ldg(g.stri_off + h);
        o1 = __ldg(g.stri_off + h + 1);
      }
    }
    // face contacts all count; without one, only the deepest edge/vertex
    // contact does (a sphere over a shared edge or vertex touches it once).
    // keep: the candidates (of the first 32) that touch on their face
    uint32_t keep = 0;
    int best = -1;
    float best_d = 0.0f;
    bool face = false;
    // most of a cell's triangles are out of reach: a sphere around each (tri_bound)
    // tells.  Its radius is rounded up by the coordinates' size, the sum by 1e-6:
    // the FP32 distance and square are off by 2e-7 of the sum, which a large
    // sphere at a small mesh near the origin would see.
    auto touches_tri = [&](uint32_t q, float3 pp, float rp, float& delta, int& region) -> bool {
      const float4 bs = __ldg(g.stri_b + q);
      const float3 dc = pp - xyz(bs);
      const float reach = (bs.w + rp) * (1.0f + 1e-6f);
      float3 nrm;
      return !(dot3(dc, dc) > reach * reach) &&
             wall_touch<kCurved>(g.walls[__ldg(g.stri_ids + q)], pp, rp, nrm, delta, region);
    };
    // the warp's 32 tests at candidates q0 .. of particle src, whose list begins at c0
    auto take = [&](int src, uint32_t q0, uint32_t c0, bool hit, int region, float delta) {
      const unsigned on_face = __ballot_sync(kAll, hit && region == 0);
      // overlaps are positive: their bits sort as they do; the first of equals
      const uint32_t depth = hit && region != 0 ? __float_as_uint(delta) : 0u;
      const uint32_t most = __reduce_max_sync(kAll, depth);
      const int first = __ffs(__ballot_sync(kAll, depth == most)) - 1;
      if (lane == src) {
        if (on_face) face = true;
        if (q0 == c0) keep = on_face;
        if (most && (best < 0 || __uint_as_float(most) > best_d)) {
          best = (int)(q0 - c0) + first;
          best_d = __uint_as_float(most);
        }
      }
    };
    // A particle's candidates are tested by the whole warp, one per lane: few of
    // a warp's particles are near the mesh, and with each tested by its own lane
    // the others wait for a chain of dependent loads: mixed charge of 21,000, 32
    // steps, 1.41 -> 1.25-1.30 ms (alone 3.04 -> 2.66); 100,000 spheres in a drum
    // of 16,384 triangles 23.0 -> 19.3 us a step.  Where a warp lies on the mesh and
    // that takes more turns than the longest list, every lane tests its own: such
    // warps are the last to end (hopper of 400,000, one alone, 148 -> 122 us a step,
    // of 150,000 85 -> 77).  Not in a turning drum or among polyhedra, whose builds
    // it only slows (drum 12.8 -> 13.5 us, mixed charge 67.7 -> 68.7).
    unsigned near = __ballot_sync(kAll, o1 > o0);
    if constexpr (kRot || kMix) {
      for (; near; near &= near - 1u) {
        const int src = __ffs(near) - 1;
        const uint32_t c0 = __shfl_sync(kAll, o0, src), c1 = __shfl_sync(kAll, o1, src);
        const float rp = __shfl_sync(kAll, ra, src);
        const float3 pp = f3(__shfl_sync(kAll, pd.x, src), __shfl_sync(kAll, pd.y, src),
                             __shfl_sync(kAll, pd.z, src));
        for (uint32_t q0 = c0; q0 < c1; q0 += 32u) {
          const uint32_t q = q0 + (uint32_t)lane;
          int region = 0;
          float delta = 0.0f;
          const bool hit = q < c1 && touches_tri(q, pp, rp, delta, region);
          take(src, q0, c0, hit, region, delta);
        }
      }
    } else {
      const bool own = __reduce_max_sync(kAll, o1 - o0) <=
                       __reduce_add_sync(kAll, (o1 - o0 + 31u) / 32u);
      int src = lane;
      uint32_t q0 = o0, c0 = o0, c1 = own ? o1 : o0;
      float rp = ra;
      float3 pp = pd;
      for (;;) {
        if (own) {
          if (!__any_sync(kAll, q0 < c1)) break;
        } else if (q0 >= c1) {   // the same in every lane
          if (!near) break;
          src = __ffs(near) - 1;
          near &= near - 1u;
          q0 = c0 = __shfl_sync(kAll, o0, src);
          c1 = __shfl_sync(kAll, o1, src);
          rp = __shfl_sync(kAll, ra, src);
          pp = f3(__shfl_sync(kAll, pd.x, src), __shfl_sync(kAll, pd.y, src),
                  __shfl_sync(kAll, pd.z, src));
        }
        const uint32_t q = own ? q0 : q0 + (uint32_t)lane;
        int region = 0;
        float delta = 0.0f;
        const bool hit = q < c1 && touches_tri(q, pp, rp, delta, region);
        if (own) {
          if (hit && region == 0) {
            face = true;
            if (q - o0 < 32u) keep |= 1u << (q - o0);
          } else if (hit && (best < 0 || delta > best_d)) {
            best = (int)(q - o0);
            best_d = delta;
          }
          ++q0;
        } else {
          take(src, q0, c0, hit, region, delta);
          q0 += 32u;
        }
      }
    }
    // the lanes' next kept candidates, ascending: of the first 32 by the mask,
    // the others (long lists) tested again
    uint32_t next = 0;
    const uint32_t len = o1 - o0;
    for (;;) {
      int at = -1;
      float3 nrm = f3(0.0f, 0.0f, 0.0f);
      float delta = 0.0f;
      int region;
      if (face) {
        if (keep) {
          at = __ffs(keep) - 1;
          keep &= keep - 1u;
          wall_touch<kCurved>(g.walls[__ldg(g.stri_ids + o0 + at)], pd, ra, nrm, delta, region);
        } else {
          for (next = max(next, 32u); next < len && at < 0; ++next)
            if (wall_touch<kCurved>(g.walls[__ldg(g.stri_ids + o0 + next)], pd, ra, nrm, delta,
                                    region) && region == 0)
              at = (int)next;
        }
      } else if (best >= 0) {
        at = best;
        best = -1;
        wall_touch<kCurved>(g.walls[__ldg(g.stri_ids + o0 + at)], pd, ra, nrm, delta, region);
      }
      if (!__any_sync(kAll, at >= 0)) break;
      const int id = at >= 0 ? (int)__ldg(g.stri_ids + o0 + at) : -1;
      if (at >= 0 && rot) nrm = rot_about(S.rot_a, rc, rsn, nrm);
      wall_contact(at >= 0, id, nrm, delta, rot);
    }
  }
  if (held) wall_flush();
  const uint32_t wmask = nw >= kWallSlots ? (1u << kWallSlots) - 1u : (1u << nw) - 1u;

  if (!valid) return 0.0f;
  // symplectic Euler (the velocities read again rather than held in registers
  // through the contacts)
  va4 = in.vel[i];
  wa4 = in.angv[i];
  const float3 va = xyz(va4), wa = xyz(wa4);
  const float ma = sphere_mass(S, ra);
  const float inv_m = 1.0f / ma;
  const float3 acc = f * inv_m + S.gravity;
  const float3 v = va + acc * dt;
  const float3 p = pa + v * dt;
  const float inertia = (0.4f * ma) * (ra * ra);
  const float3 w = wa + (t * (1.0f / inertia)) * dt;
  const float path = wa4.w + len3(v) * dt;
  out.pos[i] = make_float4(p.x, p.y, p.z, ra);
  out.vel[i] = make_float4(v.x, v.y, v.z, __uint_as_float(sys | (wmask << kSysBits)));
  out.angv[i] = make_float4(w.x, w.y, w.z, path);
  if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z))) st |= kStatusNonFinite;
  if (kCapture) {
    cap.f[i] = make_float4(f.x, f.y, f.z, 0.0f);
    cap.t[i] = make_float4(t.x, t.y, t.z, 0.0f);
  }
  return path;
  }
}

// kRecord: also write what the step reads into tape slot tp.ctl->slot (the
// history words are reserved first, by every thread of the block).
template <int kLaw, bool kCapture, bool kRecord, bool kCurved, bool kRot, bool kMix>
__device__ __forceinline__ void ens_step_body(const EnsGeom& g, const EnsBufs& b,
                                              const StateBuf& in_plain, const StateBuf& in_sorted,
                                              const StateBuf& out, int n, int wp, StepCtl* ctl,
                                              const StepLink& link, const EnsCapture& cap,
                                              const EnsTape& tp) {
  extern __shared__ uint32_t contact_sh[];
  if constexpr (!kRecord) {
    if (!round_runs(link.round)) return;
  }
  const bool rebuilt = step_rebuilt(link);
  const StateBuf in = rebuilt ? in_sorted : in_plain;
  // wp particles per warp (ens_warp_particles)
  const int lane = threadIdx.x & 31;
  const int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * wp + lane;
  const bool valid = lane < wp && i < n;
  const int e = ctl->epoch & 1;
  const EnsList L = b.L[e];
  TapeView tv{};
  float* hrec = nullptr;
  if constexpr (kRecord) {
    const TapeStep ts = tp.steps[tp.ctl->slot];
    tv = tape_view(tp, ts.block, n);
    uint32_t words = 0;
    if (valid)
      words = 3u * (uint32_t)__popc(L.mask[i]) +
              4u * (uint32_t)__popc(__float_as_uint(in.vel[i].w) >> kSysBits);
    bool ok;
    const uint32_t off =
        tape_reserve(words, &tp.ctl->cur, tp.ctl->lim, ts.hbase, &tp.ctl->overflow, ok);
    if (valid) {
      tv.hoff[i] = off;
      if (ok) hrec = reinterpret_cast<float*>(tp.arena + ts.hbase + off);
    }
  }
  uint32_t st = 0;
  const float path = ens_particle_step<kLaw, kCapture, kRecord, kCurved, true, kRot, kMix>(
      g, b, in, out, i, valid, e, L, tv, hrec, cap, st,
      contact_sh + (threadIdx.x >> 5) * kContactWords);
  {
    const unsigned m = __activemask();
    const unsigned req = __ballot_sync(m, path > 0.5f * g.skin);
    if (req && (threadIdx.x & 31) == (__ffs(m) - 1)) request_resort(link, ctl);
  }
  ens_flag(ctl, st);
}

// Registers: 64 (four blocks of 256 per SM, with some spills) where the grid
// has more blocks than the GPU holds, since the law's dependent chains need the
// warps; 80 where it has fewer (kEnsOneWave particles at most).  Per pass at 64, 80 and 96: settled boxes of
// 2,000,000 spheres, 32 steps, 13.9, 14.7, 17.4 ms; hopper of 400,000, 32 steps,
// 2.85, 2.90, 3.26 ms; mixed charge of 21,000, 32 steps, 1.53, 1.49, 1.50 ms; a
// box of 6,000, 16 steps, 181, 168, 166 us.
constexpr int kStepRegs = 64, kStepRegsSmall = 80;
template <int kLaw, bool kCapture, bool kCurved, bool kRot, bool kMix, bool kSmall>
__global__ void __maxnreg__(kSmall ? kStepRegsSmall : kStepRegs)
k_ens_step(EnsGeom g, EnsBufs b, StateBuf in_plain, StateBuf in_sorted, StateBuf out, int n,
           int wp, StepCtl* ctl, StepLink link, EnsCapture cap) {
  ens_step_body<kLaw, kCapture, false, kCurved, kRot, kMix>(g, b, in_plain, in_sorted, out, n, wp,
                                                           ctl, link, cap, EnsTape{});
}

// The recording step (reverse mode, linear law, plane walls) held to the
// plain step's 80 registers: at the 88 it takes by itself a block of 256
// fits twice per SM instead of three times.
constexpr int kRecordRegs = 80;
__global__ void __maxnreg__(kRecordRegs)
k_ens_step_rec(EnsGeom g, EnsBufs b, StateBuf in_plain, StateBuf in_sorted, StateBuf out, int n,
               int wp, StepCtl* ctl, StepLink link, EnsTape tp) {
  ens_step_body<kLawLinear, false, true, false, false, false>(
      g, b, in_plain, in_sorted, out, n, wp, ctl, link, EnsCapture{nullptr, nullptr}, tp);
}

// ------------------------------------------------------------ drum turn
__global__ void k_ens_rot_tick(const EnsSysDev* __restrict__ sys, float2* rot, int nsys,
                               RoundLink round) {
  if (!round_runs(round)) return;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsys || !sys[s].rot) return;
  const float2 r = rot[s];
  const float c1 = r.x * sys[s].rot_cd - r.y * sys[s].rot_sd;
  const float s1 = r.y * sys[s].rot_cd + r.x * sys[s].rot_sd;
  const float m = sqrtf(c1 * c1 + s1 * s1);
  rot[s] = make_float2(c1 / m, s1 / m);
}

// ---------------------------------------------------------------- rounds
__global__ void k_round_init(EnsRound r, int steps, int at) {
  *r.left = steps;
  *r.at = at;
  *r.want = at ^ (steps & 1);
}

__global__ void k_round_gate(StepCtl* ctl, EnsRound r, int* rb, int steps, int few,
                             cudaGraphConditionalHandle switch_h) {
  const int req = ctl->rebuild_req;
  ctl->rebuild_req = 0;
  *rb = 0;
  *r.stop = 0x7fffffff;
  const bool hot = req && *r.last > 0 && *r.last <= few;
  *r.len = hot ? few : steps;
  if (req) *r.since = 0;
  cudaGraphSetConditional(switch_h, req ? (hot ? 2u : 1u) : 0u);
}

__global__ void k_round_end(StepCtl* ctl, EnsRound r, int home,
                            cudaGraphConditionalHandle loop_h) {
  int ran = min(*r.len, *r.left);
  const bool stopped = *r.stop < ran;
  if (stopped) {
    ran = *r.stop + 1;
    ctl->rebuild_req = 1;
  }
  *r.since += ran;
  if (stopped) *r.last = *r.since;
  const int left = *r.left - ran;
  *r.left = left;
  *r.at = home ^ (ran & 1);
  cudaGraphSetConditional(loop_h, left > 0 ? 1u : 0u);
}

__global__ void __launch_bounds__(kThreads)
k_round_last(StateBuf s0, StateBuf s1, EnsRound r, int n) {
  const int at = *r.at;
  if (at == *r.want) return;
  const StateBuf src = at ? s1 : s0, dst = at ? s0 : s1;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  dst.pos[i] = src.pos[i];
  dst.vel[i] = src.vel[i];
  dst.angv[i] = src.angv[i];
}

// ------------------------------------------------------- persistent steps
// One launch runs up to *left steps with a grid barrier between them, so a
// stretch of steps without a re-sort costs one launch instead of one launch
// and one conditional node per step.  Every block is resident (cooperative
// launch, grid from the occupancy), the particles are strided over the grid.
// Buffers: step 0 reads the sorted copy after a re-sort, else `home`; steps
// then alternate home -> other -> home, and an odd count ends with a copy
// back, so each launch leaves the state in `home`.  A step whose particles
// ask for a re-sort is the launch's last: requests record the step index
// (atomicMin), and after barrier k every block reads the same answer to
// "was one made at step <= k" (a block already in step k + 1 can only write
// k + 1).  Barrier waits are bounded by the global timer; a block that gives
// up raises kStatusTimeout and the abort word, and every block returns.
constexpr unsigned long long kBarrierLimitNs = 2000000000ull;   // 2 s

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Arrival counter bar[0], generation bar[1], abort word bar[2].  Returns
// false when the barrier was aborted (by this block or another).
__device__ __forceinline__ bool grid_barrier(unsigned int* bar, unsigned int nblocks,
                                             StepCtl* ctl) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned int* vb = bar;
    int ok = vb[2] == 0u;
    if (ok) {
      const unsigned int gen = vb[1];
      __threadfence();
      if (atomicAdd(bar, 1u) == nblocks - 1u) {
        atomicExch(bar, 0u);
        __threadfence();
        atomicAdd(bar + 1, 1u);
      } else {
        const unsigned long long t0 = global_ns();
        while (vb[1] == gen) {
          if (vb[2] != 0u) { ok = 0; break; }
          if (global_ns() - t0 > kBarrierLimitNs) {
            atomicExch(bar + 2, 1u);
            atomicOr(&ctl->status, kStatusTimeout);
            ok = 0;
            break;
          }
          __nanosleep(100);
        }
      }
      __threadfence();
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// Registers as the small step's: kEnsOneWave particles are one per resident
// lane.  A box of 113,000 settling from rest at 64 and 80: 11.0 and 9.8 us a step.
constexpr int kPersistRegs = kStepRegsSmall;
// Particles per warp of the persistent step: spread over at most a third of the
// resident warps.  A grid that fills the GPU makes ensembles stepped side by
// side wait for one another: three boxes of 16,000 at 4, 16 and 32 per warp
// 11.8, 6.2 and 6.4 us a step.
inline int persist_warp_particles(int law, int n) {
  return law == kLawReference ? 32 : warp_particles(n, kEnsOneWave / 32 / 3);
}

// Self-check of the barrier's bounded wait: the barrier is told of one
// block more than the launch has, so nothing completes it; every block must
// give up after the limit, raise kStatusTimeout and return.
__global__ void k_barrier_check(unsigned int* bar, StepCtl* ctl) {
  grid_barrier(bar, gridDim.x + 1u, ctl);
}

template <int kLaw, bool kCurved>
__global__ void __maxnreg__(kPersistRegs)
k_ens_persist(EnsGeom g, EnsBufs b, StateBuf home, StateBuf other, StateBuf sorted, int n, int wp,
              StepCtl* ctl, const int* rebuilt, EnsPersist p) {
  extern __shared__ uint32_t contact_sh[];
  const int e = ctl->epoch & 1;
  const EnsList L = b.L[e];
  const int budget = *p.left;
  const bool rb = *rebuilt != 0;
  const int lane = threadIdx.x & 31;
  const int gstride = (int)(gridDim.x * (blockDim.x >> 5)) * wp;
  const int i0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * wp + lane;
  int done = 0;
  bool stop = false, aborted = false;
  for (int k = 0; k < budget && !stop; ++k) {
    const StateBuf in = k == 0 ? (rb ? sorted : home) : ((k & 1) ? other : home);
    const StateBuf out = (k & 1) ? home : other;
    uint32_t st = 0;
    bool req = false;
    for (int i = i0; i - lane < n; i += gstride) {   // whole warps
      const float path = ens_particle_step<kLaw, false, false, kCurved, false>(
          g, b, in, out, i, lane < wp && i < n, e, L, TapeView{}, nullptr, EnsCapture{nullptr, nullptr}, st,
          contact_sh + (threadIdx.x >> 5) * kContactWords);
      req |= path > 0.5f * g.skin;
    }
    if (__syncthreads_or(req ? 1 : 0) && threadIdx.x == 0) atomicMin(p.req_step, k);
    if (st) atomicOr(&ctl->status, st);
    if (!grid_barrier(p.bar, gridDim.x, ctl)) { aborted = true; break; }
    done = k + 1;
    stop = *(volatile int*)p.req_step <= k;
  }
  if (!aborted && (done & 1)) {
    for (int i = (int)(blockIdx.x * blockDim.x + threadIdx.x); i < n;
         i += (int)(gridDim.x * blockDim.x)) {
      home.pos[i] = other.pos[i];
      home.vel[i] = other.vel[i];
      home.angv[i] = other.angv[i];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    int left = aborted ? 0 : budget - done;
    if (stop) ctl->rebuild_req = 1;
    if (aborted) left = 0;
    *p.left = left;
    *p.done += done;
    cudaGraphSetConditional(p.loop_h, left > 0 ? 1u : 0u);
  }
}

// Start of a round of the WHILE loop: take the pending re-sort request into
// the IF node, clear the round's words.
__global__ void k_ens_persist_gate(StepCtl* ctl, EnsPersist p, int* rb,
                                   cudaGraphConditionalHandle if_h) {
  const int r = ctl->rebuild_req;
  ctl->rebuild_req = 0;
  *rb = 0;
  *p.req_step = 0x7fffffff;
  p.bar[0] = 0u;
  p.bar[1] = 0u;
  p.bar[2] = 0u;
  cudaGraphSetConditional(if_h, r ? 1u : 0u);
}

__global__ void k_ens_persist_init(EnsPersist p, int steps) {
  *p.left = steps;
}

// ---------------------------------------------------------------- staging
__global__ void __launch_bounds__(kThreads)
k_ens_pack(const float* __restrict__ pos3, const float* __restrict__ rad,
           const float* __restrict__ vel3, const float* __restrict__ avel3,
           const int* __restrict__ sys_of, StateBuf s, int* __restrict__ pid, EnsList L0,
           EnsList L1, int n, int* flags) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float r = rad[i];
  s.pos[i] = make_float4(pos3[3 * i], pos3[3 * i + 1], pos3[3 * i + 2], r);
  const float sb = __uint_as_float((uint32_t)sys_of[i] & kSysMask);
  s.vel[i] = vel3 ? make_float4(vel3[3 * i], vel3[3 * i + 1], vel3[3 * i + 2], sb)
                  : make_float4(0.0f, 0.0f, 0.0f, sb);
  s.angv[i] = avel3 ? make_float4(avel3[3 * i], avel3[3 * i + 1], avel3[3 * i + 2], 0.0f)
                    : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  pid[i] = i;
  L0.cnt[i] = 0; L0.mask[i] = 0;
  L1.cnt[i] = 0; L1.mask[i] = 0;
  if (!(r > 0.0f) || !isfinite(r)) atomicOr(flags, 1);
}

__global__ void __launch_bounds__(kThreads)
k_ens_unpack(StateBuf s, const int* __restrict__ pid_src, int n, float* pos3, float* rad,
             float* vel3, float* avel3, int* sys, int* pid) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 p = s.pos[i], v = s.vel[i], w = s.angv[i];
  pos3[3 * i] = p.x; pos3[3 * i + 1] = p.y; pos3[3 * i + 2] = p.z;
  rad[i] = fabsf(p.w);   // a polyhedron: its bounding radius
  vel3[3 * i] = v.x; vel3[3 * i + 1] = v.y; vel3[3 * i + 2] = v.z;
  avel3[3 * i] = w.x; avel3[3 * i + 1] = w.y; avel3[3 * i + 2] = w.z;
  sys[i] = (int)(__float_as_uint(v.w) & kSysMask);
  pid[i] = pid_src[i];
}

inline int nblk(int n) { return (n + kThreads - 1) / kThreads; }

}  // namespace

void ens_launch_hash(const EnsGeom& g, const EnsBufs& b, int cur, const int* at, int n,
                     const CellSort& cs, StepCtl* ctl, const int* gate, cudaStream_t st) {
  k_ens_hash<<<sort_blocks(n), kSortThreads, 0, st>>>(g, b.S[at ? 0 : cur], b.S[1], at, n, cs,
                                                      ctl, gate);
}

void ens_launch_reorder(const EnsBufs& b, int cur, const int* at, int n, const CellSort& cs,
                        StepCtl* ctl, const int* gate, cudaStream_t st) {
  k_ens_reorder<<<sort_blocks(n), kSortThreads, 0, st>>>(b.S[at ? 0 : cur], b.S[1], at, b.S[2],
                                                         b, n, cs, ctl, gate);
}

void ens_launch_nlist(const EnsGeom& g, const EnsBufs& b, int n, const CellSort& cs, StepCtl* ctl,
                      const int* gate, cudaStream_t st) {
  k_ens_nlist<<<(n + kNlistThreads - 1) / kNlistThreads, kNlistThreads, 0, st>>>(
      g, b, b.S[2].pos, b.S[2].vel, n, cs.perm, cs.start, ctl, gate);
}

void ens_launch_step(const EnsGeom& g, const EnsBufs& b, int cur, int n, StepCtl* ctl,
                     StepLink link, const EnsCapture* cap, int block, cudaStream_t st) {
  const EnsCapture c = cap ? *cap : EnsCapture{nullptr, nullptr};
  const int bs = block >= 64 && block <= kMaxStepBlock && block % 32 == 0 ? block : kThreads;
  const int wp = g.launch.warp_particles;
  const int gs = warp_blocks(n, wp, bs);
#define ENS_ARGS g, b, b.S[cur], b.S[2], b.S[cur ^ 1], n, wp, ctl, link, c
#define ENS_LAUNCH(...)                                                             \
  do {                                                                              \
    if (g.launch.resident)                                                          \
      k_ens_step<__VA_ARGS__, true><<<gs, bs, contact_bytes(bs), st>>>(ENS_ARGS);   \
    else                                                                            \
      k_ens_step<__VA_ARGS__, false><<<gs, bs, contact_bytes(bs), st>>>(ENS_ARGS);  \
  } while (0)
#define ENS_STEP(L, C, K) ENS_LAUNCH(L, C, K, false, false)
#define ENS_STEP_ROT(L, C) ENS_LAUNCH(L, C, true, true, false)
#define ENS_STEP_MIX(C, K, R) ENS_LAUNCH(kLawLinear, C, K, R, true)
  if (g.mix.npoly > 0) {   // polyhedra among the spheres (linear law)
    if (g.curved && g.any_rot) {
      if (cap) ENS_STEP_MIX(true, true, true);
      else ENS_STEP_MIX(false, true, true);
    } else if (g.curved) {
      if (cap) ENS_STEP_MIX(true, true, false);
      else ENS_STEP_MIX(false, true, false);
    } else {
      if (cap) ENS_STEP_MIX(true, false, false);
      else ENS_STEP_MIX(false, false, false);
    }
  } else if (g.curved && g.any_rot) {   // a turning drum
    if (g.law == kLawHertz) {
      if (cap) ENS_STEP_ROT(kLawHertz, true);
      else ENS_STEP_ROT(kLawHertz, false);
    } else {
      if (cap) ENS_STEP_ROT(kLawLinear, true);
      else ENS_STEP_ROT(kLawLinear, false);
    }
  } else if (g.curved) {
    if (g.law == kLawHertz) {
      if (cap) ENS_STEP(kLawHertz, true, true);
      else ENS_STEP(kLawHertz, false, true);
    } else {
      if (cap) ENS_STEP(kLawLinear, true, true);
      else ENS_STEP(kLawLinear, false, true);
    }
  } else {
    if (g.law == kLawReference) {   // plane walls only
      if (cap) ENS_STEP(kLawReference, true, false);
      else ENS_STEP(kLawReference, false, false);
    } else if (g.law == kLawHertz) {
      if (cap) ENS_STEP(kLawHertz, true, false);
      else ENS_STEP(kLawHertz, false, false);
    } else {
      if (cap) ENS_STEP(kLawLinear, true, false);
      else ENS_STEP(kLawLinear, false, false);
    }
  }
#undef ENS_STEP_MIX
#undef ENS_STEP_ROT
#undef ENS_STEP
#undef ENS_LAUNCH
#undef ENS_ARGS
}

void ens_launch_step_record(const EnsGeom& g, const EnsBufs& b, int cur, int n, StepCtl* ctl,
                            StepLink link, const EnsTape& tape, int block, cudaStream_t st) {
  const int bs = block >= 64 && block <= kMaxStepBlock && block % 32 == 0 ? block : kThreads;
  const int wp = g.launch.warp_particles;
  const int gs = warp_blocks(n, wp, bs);
  // reverse mode accepts plane walls only (blaze_ens_adj_create)
  k_ens_step_rec<<<gs, bs, contact_bytes(bs), st>>>(g, b, b.S[cur], b.S[2], b.S[cur ^ 1], n, wp, ctl, link, tape);
}

int ens_persist_grid(const EnsGeom& g, int block, int n) {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  cudaError_t err;
  if (g.law == kLawReference)
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ens_persist<kLawReference, false>, block, contact_bytes(block));
  else if (g.curved)
    err = g.law == kLawHertz
              ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ens_persist<kLawHertz, true>, block, contact_bytes(block))
              : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ens_persist<kLawLinear, true>, block, contact_bytes(block));
  else
    err = g.law == kLawHertz
              ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ens_persist<kLawHertz, false>, block, contact_bytes(block))
              : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ens_persist<kLawLinear, false>, block, contact_bytes(block));
  if (err != cudaSuccess || per_sm < 1) return 0;
  const int need = warp_blocks(n, persist_warp_particles(g.law, n), block);
  return std::max(1, std::min(need, per_sm * sms));
}

cudaError_t ens_launch_persist(const EnsGeom& g, const EnsBufs& b, int home, int n, StepCtl* ctl,
                               const int* rebuilt, const EnsPersist& p, int block, int grid,
                               bool coop, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = contact_bytes(block);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = coop ? 1 : 0;
  const StateBuf sh = b.S[home], so = b.S[home ^ 1], ss = b.S[2];
  const int wp = persist_warp_particles(g.law, n);
  if (g.law == kLawReference)
    return cudaLaunchKernelEx(&cfg, k_ens_persist<kLawReference, false>, g, b, sh, so, ss, n, wp, ctl, rebuilt, p);
  if (g.curved) {
    if (g.law == kLawHertz)
      return cudaLaunchKernelEx(&cfg, k_ens_persist<kLawHertz, true>, g, b, sh, so, ss, n, wp, ctl, rebuilt, p);
    return cudaLaunchKernelEx(&cfg, k_ens_persist<kLawLinear, true>, g, b, sh, so, ss, n, wp, ctl, rebuilt, p);
  }
  if (g.law == kLawHertz)
    return cudaLaunchKernelEx(&cfg, k_ens_persist<kLawHertz, false>, g, b, sh, so, ss, n, wp, ctl, rebuilt, p);
  return cudaLaunchKernelEx(&cfg, k_ens_persist<kLawLinear, false>, g, b, sh, so, ss, n, wp, ctl, rebuilt, p);
}

void ens_launch_rot_tick(const EnsGeom& g, int nsys, const RoundLink& round, cudaStream_t st) {
  k_ens_rot_tick<<<(nsys + kThreads - 1) / kThreads, kThreads, 0, st>>>(g.sys, g.rot, nsys, round);
}

void ens_launch_round_init(const EnsRound& r, int steps, int at, cudaStream_t st) {
  k_round_init<<<1, 1, 0, st>>>(r, steps, at);
}

void ens_launch_round_gate(StepCtl* ctl, const EnsRound& r, int* rb, int steps, int few,
                           cudaGraphConditionalHandle switch_h, cudaStream_t st) {
  k_round_gate<<<1, 1, 0, st>>>(ctl, r, rb, steps, few, switch_h);
}

void ens_launch_round_end(StepCtl* ctl, const EnsRound& r, int home,
                          cudaGraphConditionalHandle loop_h, cudaStream_t st) {
  k_round_end<<<1, 1, 0, st>>>(ctl, r, home, loop_h);
}

void ens_launch_round_last(const EnsBufs& b, const EnsRound& r, int n, cudaStream_t st) {
  k_round_last<<<nblk(n), kThreads, 0, st>>>(b.S[0], b.S[1], r, n);
}

void ens_launch_barrier_check(unsigned int* bar, StepCtl* ctl, cudaStream_t st) {
  k_barrier_check<<<2, 64, 0, st>>>(bar, ctl);
}

void ens_launch_persist_gate(StepCtl* ctl, const EnsPersist& p, int* rb,
                             cudaGraphConditionalHandle if_h, cudaStream_t st) {
  k_ens_persist_gate<<<1, 1, 0, st>>>(ctl, p, rb, if_h);
}

void ens_launch_persist_init(const EnsPersist& p, int steps, cudaStream_t st) {
  k_ens_persist_init<<<1, 1, 0, st>>>(p, steps);
}

void ens_launch_pack(const float* pos3, const float* rad, const float* vel3, const float* avel3,
                     const int* sys_of, const EnsBufs& b, int cur, int* pid_dst, int n,
                     int* flags, cudaStream_t st) {
  k_ens_pack<<<nblk(n), kThreads, 0, st>>>(pos3, rad, vel3, avel3, sys_of, b.S[cur], pid_dst,
                                           b.L[0], b.L[1], n, flags);
}

void ens_launch_unpack(const EnsBufs& b, int cur, int n, const int* pid_src, float* pos3,
                       float* rad, float* vel3, float* avel3, int* sys, int* pid,
                       cudaStream_t st) {
  k_ens_unpack<<<nblk(n), kThreads, 0, st>>>(b.S[cur], pid_src, n, pos3, rad, vel3, avel3, sys,
                                             pid);
}

}  // namespace blaze
