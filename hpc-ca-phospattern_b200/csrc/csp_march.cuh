// csp_march.cuh -- the step kernel: any number of time steps in one launch.
//
// The CTAs of a launch (at most one per SM, launched cooperatively) form teams; a team takes
// its realisations one after the other and advances each by all the steps of the call, with
// a barrier between the CTAs of the team after every step.  How many realisations are in
// flight at once (the number of teams) is chosen so that their fields -- both buffers of
// every species -- stay in the L2 cache while they are stepped: HBM is read and written once
// per call instead of once per step, and no launch, and no drain of the GPU at its end, lies
// between two steps.  (One launch per step streams every realisation through HBM: 41 bytes
// per voxel and step.)
//
// Within a step a warp takes units (realisation, column of 128 plane positions, x segment):
// each lane owns 4 consecutive positions of one row (rows are padded to a multiple of 4) and
// marches along x with the planes x-1, x, x+1 of every species that diffuses this step in
// registers, the plane x+2 on its way; the y-neighbour rows and the two outer z-neighbours
// come from L1 / L2 (the warps of a CTA hold adjacent columns).  Species that only react are
// read one plane ahead, 128 bits at a time.  The arithmetic rounds like voxel_update
// (csp_kernels.cuh), which the direct kernel runs, so both give bitwise equal fields.
//
// A group code per 4 voxels (RealDesc::gcode) names the domain when the group and its whole
// neighbourhood lie in it and no voxel of it receives boundary flux, or a pattern (regular
// groups along domain sheets: coefficients per direction, SERCA flux from the values at hand).
// A warp whose groups are all uniform takes the leaner of two forms of the loop body.  The
// voxels of irregular groups and those with channels are the boundary work, in tiles of 32
// (mixed_voxel); a batch with many irregular voxels has them in tiles of 32 groups (mixed_group).
//
// The barrier's wait is bounded in time (MarchArgs::wait_ns).  A CTA that gives up sets ERR_TIMEOUT in the
// device error word, which the other waits see too, and every CTA leaves the launch; the fields
// are undefined then (the host reports CSP_EDEVICE).  Nothing is in flight when a CTA leaves
// but its own plain loads and stores.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "csp_kernels.cuh"
#include "csp_ptx.cuh"

namespace csp {

constexpr int MARCH_T = 512;              // threads per CTA
constexpr int MARCH_COL = 128;            // plane positions per unit: 4 per lane
constexpr unsigned long long INJECT_WAIT_NS = 1000000ull;   // limit of a wait with the test hook: 1 ms

// What a launch does with the step of a realisation.
enum : unsigned {
  MARCH_UNITS = 1u,      // the groups
  MARCH_VOXELS = 2u,     // the boundary work without channels
  MARCH_CHANNELS = 4u,   // the voxels with channels (gating)
  MARCH_ADVANCE = 8u,    // then go on: step counter, abort rule
  MARCH_STEP = 15u,
  MARCH_REPEAT = 16u     // the same step again, with the barriers (csp_autotune)
};

// A realisation's part of a launch: its units and its boundary work.
struct MarchReal {
  int r;
  int ncol, nseg;                    // columns, x segments
  int cut0;                          // segment s: planes [cuts[cut0 + s], cuts[cut0 + s + 1])
  int chan0, nchan, vox0, nvox, grp0, ngrp;
};
// Irregular voxels of a batch from which they are taken as groups (MixGroup): with fewer, a
// voxel per lane fills the GPU and its chain is shorter (us per step of random 2^3 blocks of
// domains, by voxel and by group: one grid of 40x40x36 6.8 and 12.1, one of 100x100x50 34.7 and
// 23.4, 24 of those 845 and 423; 8^3 blocks, 24 grids: 344 and 247).  Realisations count where
// they are at least a share of the voxels: the sheets of a dyad leave 1 %, and their kernel
// (MARCH_KNOWN) is the faster for having no code for groups (64 grids of 100x100x50 278 us per
// step, with that code and their 1 % as groups 345).
constexpr size_t MIX_GROUPS_MIN = 262144;
constexpr double MIX_GROUPS_SHARE = 1.0 / 8;
// Share of uniform groups below which the units of such a realisation would read its planes for
// next to nothing: all of its groups are boundary work (24 grids of 2^3 blocks: 423 -> 374 us).
constexpr double MIX_DENSE = 1.0 / 16;
constexpr int MARCH_CUTS = 1024;          // segments of a realisation (at most), plus one

struct MarchArgs {
  const RealDesc* descs;
  const VoxDesc* vdescs;
  RealCtl* ctl;
  StepRec* rec;
  const MarchReal* real;             // by team
  const int* cuts;
  const int* first;                  // [teams + 1]: the entries of team t are real[first[t] ... first[t + 1])
  int size;                          // CTAs per team
  long long nsteps;
  unsigned what;                     // MARCH_*
  MixArgs mix;
  unsigned* arrived;                 // [teams * 32]: CTAs arrived at the team's barriers, 0 before the launch
  int* flags;                        // nullable [nsteps][flag_stride]: stop flag of realisation r at [r]
  int flag_stride;
  int* err;
  unsigned long long wait_ns;        // limit of a wait
  int inject;                        // test hook (csp_test_wait_timeout)
};

// The running step of the CTA's realisation.
struct MarchStep {
  unsigned cur, updated, pre, sub, flags;
  int go;                            // 0: no further step; -1: leave the launch
  long long k;                       // steps taken before it
  const float* uo[NS];               // current and next buffer of every species
  float* un[NS];
};
struct MarchShared {
  alignas(16) VoxDesc desc;
  MarchStep step;
  int next;                          // items of the step that a warp has taken beyond its first
  int next_group;                    // tiles of irregular groups taken
  // the same on every step: the segments, and the entries of the CTA's first boundary tiles
  int cut[MARCH_CUTS];
  alignas(16) int4 tile[MARCH_T][2];
};

__device__ __forceinline__ const float* field(const float* p) {
  __builtin_assume(__isGlobal(p));
  return p;
}
__device__ __forceinline__ float* field(float* p) {
  __builtin_assume(__isGlobal(p));
  return p;
}

// rx_classify on the four voxels of a group in one domain d, in two-lane FP32 with the
// same rounding (ca0 / ca1: Ca of voxels 0,1 / 2,3; G0 / G1: their sums of the increments
// dJ_s in slot order, accumulated by the reaction loop that applies them): the class of
// voxel j in byte j.
template <int MS>
__device__ __forceinline__ unsigned rx_classify4(const VoxDesc& D, int d, F2 ca0, F2 ca1, const float (&val)[MS][4],
                                                 F2 G0, F2 G1) {
  const unsigned kind = D.sur_kind[d];
  if (kind != RX_ELIGIBLE) return kind == RX_STIFF ? RX_CLASS_PLAIN * 0x01010101u : 0u;
  const unsigned rm = D.rmask[d];
  const F2 dca0 = f2(val[0][0], val[0][1]), dca1 = f2(val[0][2], val[0][3]);
  const F2 aG0 = f2_abs(G0), aG1 = f2_abs(G1);
  unsigned long long neg0 = 0, neg1 = 0;   // sign bits of the margins, OR-ed over the slots
#pragma unroll
  for (int s = 1; s < MS; s++) {
    if (!(rm >> s & 1u)) continue;
    const F2 nkon = {D.rk2[d][s][0]}, nkoff = {D.rk2[d][s][1]}, a = {D.rk2[d][s][2]}, j0 = {D.rk2[d][s][3]};
    const F2 cs = f2(D.sur_cs[d][s], D.sur_cs[d][s]), thr = f2(D.sur_thr2[d][s], D.sur_thr2[d][s]);
    const F2 db0 = f2(val[s][0], val[s][1]), db1 = f2(val[s][2], val[s][3]);
    const F2 in0 = f2_fma(nkon, ca0, nkoff), in1 = f2_fma(nkon, ca1, nkoff);
    const F2 dj0 = f2_fma(db0, in0, f2_fma(a, dca0, j0)), dj1 = f2_fma(db1, in1, f2_fma(a, dca1, j0));
    neg0 |= f2_fma(in0, f2_abs(dj0), f2_fma(f2_mul(nkon, f2_sub(cs, db0)), aG0, thr)).v;
    neg1 |= f2_fma(in1, f2_abs(dj1), f2_fma(f2_mul(nkon, f2_sub(cs, db1)), aG1, thr)).v;
  }
  const unsigned e = RX_CLASS_EXPLICIT, nt = RX_CLASS_NETWORK;
  return ((neg0 >> 31 & 1u) ? nt : e) | ((neg0 >> 63) ? nt : e) << 8 | ((neg1 >> 31 & 1u) ? nt : e) << 16 |
         ((neg1 >> 63) ? nt : e) << 24;
}

// General reactions (react_general) of a group in domain d, the four voxels of a species
// together (models whose buffers do not all bind species 0): local arrays indexed by the
// buffers' species, so that the fast path's registers stay registers.  24 grids of 100x100x50
// with such a buffer: 616 us per step with a voxel at a time and the masks at run time, now 249.
template <int MS>
__device__ __noinline__ void react_group(const RealDesc& D, int d, const float4* val, float4* out, unsigned pre,
                                         unsigned fq) {
  for (int bi = 0; bi < D.nbuf; bi++) {
    const int t = bi * D.nd + d;
    const int s0 = D.bsp0[t], s1 = D.bsp1[t];
    const float nkon = -D.kon_dt[t], nkoff = -D.koff_dt[t], a = D.a_dt[t], j0 = D.j0_dt[t], base = D.fbase[d][s1];
    const float4 b0 = val[s0], b1 = val[s1];
    auto dj = [&](float x0, float x1) { return buffer_dj(nkon, nkoff, a, j0, x0, x1, __fadd_rn(base, x1)); };
    const float4 J = make_float4(dj(b0.x, b1.x), dj(b0.y, b1.y), dj(b0.z, b1.z), dj(b0.w, b1.w));
    float4 r = (pre >> s0 & 1u) ? out[s0] : b0;
    if ((fq & ~pre) >> s0 & 1u) r = J;
    else r = make_float4(__fadd_rn(r.x, J.x), __fadd_rn(r.y, J.y), __fadd_rn(r.z, J.z), __fadd_rn(r.w, J.w));
    out[s0] = r;
    r = (pre >> s1 & 1u) ? out[s1] : b1;
    out[s1] = make_float4(__fsub_rn(r.x, J.x), __fsub_rn(r.y, J.y), __fsub_rn(r.z, J.z), __fsub_rn(r.w, J.w));
  }
}

// What a kernel's bodies know at compile time: every mask of the step (MARCH_KNOWN, for batches
// of the reference model's shape, see march_masks_known), or the species that diffuse
// (MARCH_MASKS, any other model of up to five species; masks it has no body for run on one with
// run-time masks), or nothing (MARCH_RUNTIME, up to eight species).  us per step of 24 grids of
// 100x100x50 with run-time masks and on MARCH_MASKS: Dirichlet faces 256 -> 126, two
// fixed-point species 261 -> 116, three species 161 -> 90; the reference model on MARCH_KNOWN
// 104.  The bodies are kernels of their own: in one kernel the run-time body's registers and
// spills (1,008 bytes of loads) became everyone's.
enum : int { MARCH_KNOWN = 0, MARCH_MASKS = 1, MARCH_RUNTIME = 2 };
// A body's reactions: none, fast (STEP_REACT_FAST), general, or as the step says.
enum : int { REACT_NONE = 0, REACT_FAST = 1, REACT_GENERAL = 2, REACT_ANY = 3 };

// Whether every step of a realisation runs on the variants with compile-time masks (see
// march_dispatch): the reference model's shape.
inline bool march_masks_known(const RealDesc& D) {
  if (D.ns != 5 || D.fixq != 1u << 4 || D.dirichlet || !D.react_fast || D.nbuf == 0) return false;
  for (int d = 0; d < ND; d++)
    if (D.fixed_mask[d]) return false;
  const int k = D.dsi_of[0];
  return k >= 0 && D.substeps[k] == 1 && (D.reaction_flag_mask & 0x1Fu) == 0x1Fu;
}

// What a lane knows of its unit's groups: the place in the row and the offsets of their
// neighbours (out of the box: the voxel itself, so the values need no selection afterwards).
struct GroupPlace {
  int z0, lastj;            // first position, last voxel inside the box (>= 3: all four)
  int dym, dyp, dzm, dzp;
};

// One unit.  PRE >= 0: the species of PRE diffuse and the reactions are REACT, known at compile
// time, so the loop has no test of them and three planes of registers for the species of PRE
// alone.  EXACT: so is the rest -- with reactions every species is updated, FQ are exactly the
// fixed-point species and nothing is fixed.  PRE < 0: all at run time, any model.
template <int MS, unsigned FQ, bool SUR, int PRE, int REACT, bool EXACT>
__device__ __forceinline__ void march_unit(const RealDesc* __restrict__ descs, int r_, int col, int x0, int x1) {
  constexpr bool DYN = PRE < 0;
  // from the shared array itself, not by argument: the compiler then knows the address space
  extern __shared__ __align__(128) unsigned char smem[];
  const MarchShared& S = *reinterpret_cast<const MarchShared*>(smem);
  const VoxDesc& D = S.desc;
  const MarchStep& U = S.step;
  const unsigned pre = DYN ? U.pre : (unsigned)PRE;
  const unsigned lmask = DYN                   ? U.updated
                         : REACT == REACT_NONE ? (unsigned)PRE
                         : EXACT               ? (1u << MS) - 1u
                                               : U.updated | (unsigned)PRE;
  const bool react = DYN ? (U.flags & STEP_REACT) != 0u : REACT != REACT_NONE;
  const bool react_fast = DYN ? (U.flags & STEP_REACT_FAST) != 0u : REACT == REACT_FAST;
  // fixed-point species (never diffusing ones)
  const unsigned fq = EXACT ? FQ & lmask : FQ & D.fixq & lmask & ~pre;
  const int nz = D.nz;
  const int p0 = col * MARCH_COL + 4 * (int)(threadIdx.x & 31u);
  const unsigned lanes = __ballot_sync(0xffffffffu, p0 < D.plane);
  if (p0 >= D.plane) return;
  GroupPlace G;
  {
    const int y = p0 / nz;
    G.z0 = p0 - y * nz;
    G.lastj = D.nzv - 1 - G.z0;
    G.dym = y > 0 ? -nz : 0;
    G.dyp = y < D.ny - 1 ? nz : 0;
    G.dzm = G.z0 > 0 ? -1 : 0;
    G.dzp = G.lastj >= 4 ? 4 : 3;
  }
  const int cut = D.nzv != nz && G.lastj < 3 ? G.lastj : 4;     // the row ends inside the group, after voxel cut
  const int nx = D.nx, P = D.P;
  unsigned off = (unsigned)x0 * P + p0;          // the lane's position (padded fields hold < 2^32)
  // planes x-1, x, x+1 (cur: also the species that only react)
  float4 prv[MS], cur[MS], nxt[MS];
#pragma unroll
  for (int s = 0; s < MS; s++) {
    prv[s] = cur[s] = nxt[s] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!(lmask >> s & 1u)) continue;
    const float* u = field(U.uo[s]) + off;
    cur[s] = *reinterpret_cast<const float4*>(u);
    if (!(pre >> s & 1u)) continue;
    prv[s] = *reinterpret_cast<const float4*>(u - (x0 > 0 ? P : 0));
    nxt[s] = *reinterpret_cast<const float4*>(u + (x0 + 1 < nx ? P : 0));
  }
  unsigned code_next = __ldg(D.gcode + (off >> 2));
  for (int x = x0; x < x1; x++) {
    const unsigned code = code_next;
    const bool more = x + 1 < x1;
    float4 fut[MS];                              // plane x+2
#pragma unroll
    for (int s = 0; s < MS; s++) {
      fut[s] = nxt[s];
      if ((pre >> s & 1u) && more && x + 2 < nx)
        fut[s] = *reinterpret_cast<const float4*>(field(U.uo[s]) + (off + 2u * P));
    }
    if (more) code_next = __ldg(D.gcode + ((off + P) >> 2));
    // every neighbour before the first store: a load that follows a store to another buffer
    // waits for it in program order, one L2 latency per species
    float4 ym[MS], yp[MS];
    float zm[MS], zp[MS];
#pragma unroll
    for (int s = 0; s < MS; s++) {
      ym[s] = yp[s] = make_float4(0.f, 0.f, 0.f, 0.f);
      zm[s] = zp[s] = 0.f;
      if (!(pre >> s & 1u)) continue;
      const float* u = field(U.uo[s]) + off;
      ym[s] = *reinterpret_cast<const float4*>(u + G.dym);
      yp[s] = *reinterpret_cast<const float4*>(u + G.dyp);
      zm[s] = u[G.dzm];
      zp[s] = u[G.dzp];
    }
    // the next plane's values of a species that only reacts, into the registers its values of
    // this plane leave
    auto fetch_next = [&](int s) {
      if (more && ((lmask & ~pre) >> s & 1u))
        cur[s] = *reinterpret_cast<const float4*>(field(U.uo[s]) + (off + P));
    };
    // ---- the group: one species at a time from load to store (Ca first, stored last), voxel
    // pairs (0,1) and (2,3) in two-lane FP32.  REG: the warp has regular groups ----
    auto group = [&](auto reg) {
      constexpr bool REG = decltype(reg)::value;
      GroupPattern pt{code * 0x49249u, PAT_NONE};              // a uniform group: its domain seven times
      if (REG && code >= (unsigned)ND) pt = D.pat[code - ND];
      const int d0 = REG ? (int)(pt.code & 7u) : (int)code;
      auto dn = [&](int kk) -> int { return (int)(pt.code >> (3 + 3 * kk)) & 7; };
      const bool allyx = !REG || ((pt.code >> 9) & 0xfffu) == (unsigned)d0 * 0x249u;
      const bool uni0 = allyx && dn(0) == d0, uni3 = allyx && dn(1) == d0;
      const unsigned fixed = EXACT ? 0u : D.fixed_mask[d0];
      // value and diffusion of species s: v = the stored values (fixed point: converted),
      // o2 = diffused value (fixed point: the increment so far, 0)
      auto load_diffuse = [&](int s, float4& v, F2 (&o2)[2]) {
        v = cur[s];
        if (fq >> s & 1u) {
          const float qu = D.qunit[d0][s];
          v = make_float4(q_value(v.x, qu), q_value(v.y, qu), q_value(v.z, qu), q_value(v.w, qu));
          o2[0] = o2[1] = f2(0.f, 0.f);
          return;
        }
        o2[0] = f2(v.x, v.y);
        o2[1] = f2(v.z, v.w);
        if (!(pre >> s & 1u)) return;
        const float cdd = D.cdiag[d0][s];
        const float4 vp = prv[s], vn = nxt[s];
        const float4 qm = ym[s], qp = yp[s];
        float r0 = v.y, r1 = v.z, r2 = v.w;
        if (cut < 3) {
          r0 = cut == 0 ? v.x : r0;
          r1 = cut == 1 ? v.y : r1;
          r2 = cut == 2 ? v.z : r2;
        }
        const F2 m2 = f2(-2.f, -2.f), c2 = f2(cdd, cdd);
        const F2 zs0 = f2(__fadd_rn(zm[s], r0), __fadd_rn(v.x, r1));
        const F2 zs1 = f2(__fadd_rn(v.y, r2), __fadd_rn(v.z, zp[s]));
        const F2 ys0 = f2_add(f2(qm.x, qm.y), f2(qp.x, qp.y)), ys1 = f2_add(f2(qm.z, qm.w), f2(qp.z, qp.w));
        const F2 xs0 = f2_add(f2(vp.x, vp.y), f2(vn.x, vn.y)), xs1 = f2_add(f2(vp.z, vp.w), f2(vn.z, vn.w));
        const F2 u0 = o2[0], u1 = o2[1];
        o2[0] = diffuse_uniform2(c2, m2, u0, zs0, ys0, xs0);
        o2[1] = diffuse_uniform2(c2, m2, u1, zs1, ys1, xs1);
        if constexpr (REG) {
          // the per-neighbour-coefficient form (diffuse_coef6), taken by the voxels that have a
          // neighbour in another domain
          const float* c = D.coef[s] + d0 * ND;
          const float cz0 = c[dn(0)], cz1 = c[dn(1)];
          F2 a0 = f2_fma(f2(cz0, cdd), f2_sub(f2(zm[s], v.x), u0), f2(0.f, 0.f));
          F2 a1 = f2_fma(c2, f2_sub(f2(v.y, v.z), u1), f2(0.f, 0.f));
          a0 = f2_fma(c2, f2_sub(f2(r0, r1), u0), a0);
          a1 = f2_fma(f2(cdd, cz1), f2_sub(f2(r2, zp[s]), u1), a1);
          auto side = [&](float ck, const float4& q) {
            const F2 k2 = f2(ck, ck);
            a0 = f2_fma(k2, f2_sub(f2(q.x, q.y), u0), a0);
            a1 = f2_fma(k2, f2_sub(f2(q.z, q.w), u1), a1);
          };
          side(c[dn(2)], qm);
          side(c[dn(3)], qp);
          side(c[dn(4)], vp);
          side(c[dn(5)], vn);
          float g0, g1, g2, g3, n0, n1, n2, n3;
          f2_split(f2_add(u0, a0), g0, g1);
          f2_split(f2_add(u1, a1), g2, g3);
          f2_split(o2[0], n0, n1);
          f2_split(o2[1], n2, n3);
          o2[0] = f2(uni0 ? n0 : g0, allyx ? n1 : g1);
          o2[1] = f2(allyx ? n2 : g2, uni3 ? n3 : g3);
        }
      };
      // stored form of species s (st: its stored values) after the step
      auto store = [&](int s, float4 st, const F2 (&o2)[2]) {
        float4 r;
        f2_split(o2[0], r.x, r.y);
        f2_split(o2[1], r.z, r.w);
        if (!EXACT && (fixed >> s & 1u)) {
          float iv = D.dinit[d0][s];
          if (fq >> s & 1u) iv = q_set(iv, D.qinv[d0][s]);
          r = make_float4(iv, iv, iv, iv);
        } else if (fq >> s & 1u) {                  // the stored integers plus the increments
          const float qi = D.qinv[d0][s];
          r = make_float4(q_add(st.x, r.x, qi), q_add(st.y, r.y, qi), q_add(st.z, r.z, qi), q_add(st.w, r.w, qi));
        }
        if (!EXACT && s == 0 && D.dirichlet) {
          const bool face = x == 0 || x + 1 == nx || G.dym == 0 || G.dyp == 0;
          const float iv = D.dinit[d0][0];
          if (face || G.z0 == 0) r.x = iv;
          if (face || G.lastj == 0) r.x = iv;
          if (face || G.lastj == 1) r.y = iv;
          if (face || G.lastj == 2) r.z = iv;
          if (face || G.lastj == 3) r.w = iv;
        }
        if (REG && s == 0 && pt.flux != PAT_NONE && (!DYN || (pre & 1u))) {
          // SERCA across one face (boundaryfluxes.c:60-84) on the steps on which Ca diffuses, from
          // the old Ca of its two sides
          const int kk = (int)(pt.flux & 7u);
          const float4 q = kk == 2 ? ym[0] : kk == 3 ? yp[0] : kk == 4 ? prv[0] : nxt[0];
          const double bs = D.base0[d0], bo = D.base0[dn(kk)], scale = D.serca;
          const bool to = pt.flux & PAT_TO;
          auto add = [&](float& z, float self, float other, int j) {
            const double us = (double)self + bs, uo = (double)other + bo;
            const double J = serca_flux_fast(to ? uo : us, to ? us : uo, scale);
            if (pt.flux >> (4 + j) & 1u) z = (float)((double)z + (to ? J : -J));
          };
          add(r.x, cur[0].x, q.x, 0); add(r.y, cur[0].y, q.y, 1); add(r.z, cur[0].z, q.z, 2); add(r.w, cur[0].w, q.w, 3);
        }
        *reinterpret_cast<float4*>(field(U.un[s]) + off) = r;
      };
      if (react && !react_fast) {
        float4 tv[MS], to[MS];
#pragma unroll
        for (int s = 0; s < MS; s++) {
          F2 o2[2];
          load_diffuse(s, tv[s], o2);
          f2_split(o2[0], to[s].x, to[s].y);
          f2_split(o2[1], to[s].z, to[s].w);
        }
        react_group<MS>(descs[r_], d0, tv, to, pre, fq);
#pragma unroll
        for (int s = 0; s < MS; s++) {
          const F2 o2[2] = {f2(to[s].x, to[s].y), f2(to[s].z, to[s].w)};
          if (lmask >> s & 1u) store(s, cur[s], o2);
          fetch_next(s);
        }
      } else {
        float4 ca;                               // Ca's deviations, then Ca itself in c0, c1
        F2 o0[2], c0, c1, G0 = f2(0.f, 0.f), G1 = G0;
        float val[SUR ? MS : 1][4];              // SUR: the classification reads every species again
        load_diffuse(0, ca, o0);
        const F2 dc0 = f2(ca.x, ca.y), dc1 = f2(ca.z, ca.w);
        if (react_fast) {
          const float cb = D.fbase0[d0];
          c0 = f2_add(f2(cb, cb), dc0);
          c1 = f2_add(f2(cb, cb), dc1);
        }
        if (SUR) { val[0][0] = ca.x; val[0][1] = ca.y; val[0][2] = ca.z; val[0][3] = ca.w; }
#pragma unroll
        for (int s = 1; s < MS; s++) {
          if (!(lmask >> s & 1u)) continue;
          const float4 st = cur[s];
          float4 v;
          F2 o2[2];
          load_diffuse(s, v, o2);
          if (react_fast) {
            // a domain without a buffer for s has zero constants, which add an exact zero
            const ulonglong2 k0 = *reinterpret_cast<const ulonglong2*>(&D.rk2[d0][s][0]);
            const ulonglong2 k1 = *reinterpret_cast<const ulonglong2*>(&D.rk2[d0][s][2]);
            const F2 nkon = {k0.x}, nkoff = {k0.y}, a = {k1.x}, j0 = {k1.y};
            const F2 dj0 = buffer_dj2(nkon, nkoff, a, j0, f2(v.x, v.y), dc0, c0);
            const F2 dj1 = buffer_dj2(nkon, nkoff, a, j0, f2(v.z, v.w), dc1, c1);
            o2[0] = f2_add(o2[0], dj0);
            o2[1] = f2_add(o2[1], dj1);
            o0[0] = f2_sub(o0[0], dj0);
            o0[1] = f2_sub(o0[1], dj1);
            if (SUR) {
              G0 = f2_add(G0, dj0);
              G1 = f2_add(G1, dj1);
            }
          }
          if (SUR) { val[s][0] = v.x; val[s][1] = v.y; val[s][2] = v.z; val[s][3] = v.w; }
          store(s, st, o2);
          fetch_next(s);
        }
        if (lmask & 1u) store(0, cur[0], o0);
        fetch_next(0);
        if constexpr (SUR) {
          if (react_fast && D.sur) {
            unsigned cls = rx_classify4<MS>(D, d0, c0, c1, val, G0, G1);
            if (G.lastj < 3) cls &= (1u << (8 * (G.lastj + 1))) - 1u;   // the row's padding has no class
            *reinterpret_cast<unsigned*>(D.rx_class + off) = cls;
          }
        }
      }
    };
    const bool mine = code != CODE_MIXED;
    if (__all_sync(lanes, code < (unsigned)ND || code == CODE_MIXED)) {
      if (mine) group(std::false_type{});
    } else {
      if (mine) group(std::true_type{});
    }
    if (!mine) {
#pragma unroll
      for (int s = 0; s < MS; s++) fetch_next(s);
    }
#pragma unroll
    for (int s = 0; s < MS; s++) {
      if (!(pre >> s & 1u)) continue;
      prv[s] = cur[s];
      cur[s] = nxt[s];
      nxt[s] = fut[s];
    }
    off += P;
  }
}

// The body of a step: Ca and any of the species 1-3 diffusing; everything else at run time.
template <int MS, unsigned FQ, bool SUR, int BODY>
__device__ __forceinline__ void march_dispatch(const MarchShared& S, const RealDesc* __restrict__ descs, int r, int col,
                                               int x0, int x1) {
  const MarchStep& U = S.step;
  if constexpr (BODY != MARCH_RUNTIME) {
    constexpr bool EXACT = BODY == MARCH_KNOWN;
    const bool none = !(U.flags & STEP_REACT), fast = U.flags & STEP_REACT_FAST;
#define CSP_UNIT(p)                                                                                     \
  case p:                                                                                               \
    if (fast) march_unit<MS, FQ, SUR, p, REACT_FAST, EXACT>(descs, r, col, x0, x1);                     \
    else if (EXACT || none) march_unit<MS, FQ, SUR, p, REACT_NONE, EXACT>(descs, r, col, x0, x1);       \
    else if constexpr (!EXACT) march_unit<MS, FQ, SUR, p, REACT_GENERAL, EXACT>(descs, r, col, x0, x1); \
    return;
    switch (U.pre) {
      CSP_UNIT(0x1) CSP_UNIT(0x3) CSP_UNIT(0x5) CSP_UNIT(0x7)
      CSP_UNIT(0x9) CSP_UNIT(0xB) CSP_UNIT(0xD) CSP_UNIT(0xF)
      default: break;
    }
#undef CSP_UNIT
  }
  if constexpr (BODY != MARCH_KNOWN) march_unit<MS, FQ, SUR, -1, REACT_ANY, false>(descs, r, col, x0, x1);
}

// The step counters of a realisation, on the lanes of a warp: lane l < 30 holds the step index
// modulo the substep of diffusive index l, lane 30 modulo the gating's,
// lane 31 modulo the reaction's.  next() goes to the
// following step and gives its masks (step_masks, step_info) to every lane: a few
// instructions between two steps, where the divisions and the loads of the descriptor they
// replace took 8 us.
struct MarchCount {
  int rem, sub, species;             // sub 0: the lane has no counter
  unsigned reaction_flags;
  bool react_fast;
  __device__ __forceinline__ void init(const RealDesc& D, long long k, int lane) {
    sub = lane < D.ndiff && lane < NS ? D.substeps[lane] : lane == 31 && D.nbuf > 0 ? D.reaction_substep
          : lane == 30                      ? D.stochastic_substep : 0;
    species = lane < D.ndiff && lane < NS ? D.diff_species[lane] : 0;
    rem = sub > 0 ? (int)(k % sub) : 0;
    reaction_flags = D.reaction_flag_mask;
    react_fast = D.react_fast;
  }
  __device__ __forceinline__ void next(int lane, unsigned& pre, unsigned& updated, unsigned& dsi, unsigned& flags) {
    rem = rem + 1 >= sub ? 0 : rem + 1;
    const unsigned due = __ballot_sync(0xffffffffu, sub > 0 && rem == 0);
    dsi = due & 0x3fffffffu;
    pre = __reduce_or_sync(0xffffffffu, lane < 30 && (due >> lane & 1u) ? 1u << species : 0u);
    const bool react = due >> 31;
    updated = pre | (react ? reaction_flags : 0u);
    flags = (react ? (react_fast && (pre & 1u) ? STEP_REACT | STEP_REACT_FAST : STEP_REACT) : 0u) |
            (due >> 30 & 1u ? STEP_GATE : 0u);
  }
};

// Barrier of a team in two halves, for one thread of every CTA after __syncthreads: what the
// CTA wrote is released with its arrival, what the others wrote is acquired after the wait
// (false: given up).
__device__ __forceinline__ void march_arrive(unsigned* arrived) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
}
__device__ __forceinline__ bool march_wait(const unsigned* arrived, unsigned target, unsigned long long limit_ns, int* err) {
  auto count = [&]() {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrived) : "memory");
    return v;
  };
  if (count() >= target) return true;
  const unsigned long long t0 = global_ns();
  while (count() < target) {
    if (*(volatile int*)err & ERR_TIMEOUT) return false;
    if (global_ns() - t0 > limit_ns) {
      atomicOr(err, ERR_TIMEOUT);
      return false;
    }
  }
  return true;
}

// Flux of an item of any law: the channel's gating, then its flux.
__device__ __noinline__ bool mix_pair_flux(const RealDesc& D, RealCtl* C, const MixItem& it, const FluxPair& pr,
                                           const FluxParams& fp, const float* uold, const float* ca,
                                           unsigned char* states, int nch, long long k, double& J) {
  return pair_step<true>(D, C, pr.species, pr.kind, pr.dsi, pr.channel, pr.local_channel, pr.boundary,
                         (it.meta & MIX_OWNER) ? 1 : 0, pr.v0, pr.v1, pr.doms, fp, uold, ca, states, nch, k,
                         ((k + 1) % D.stochastic_substep) == 0, J);
}

// One voxel of an irregular group: everything a step does to it -- diffusion with its
// neighbours' coefficients, reactions, fixed values (the arithmetic of voxel_update), then the
// fluxes of its boundary pairs in pair order, summed in FP64 and added with one rounding
// (Species_step_boundary_fluxes, species.c:1704-1907; channels gated first,
// boundaryfluxes.c:295-359).  Bound: the latency of its chain of loads, so the entry (in hand)
// carries what its loads need and the tables are in shared memory: entry, then every value
// and the flux partner together.
template <int MS, bool SUR>
__device__ __forceinline__ void mixed_voxel(const VoxDesc& D, const MarchStep& U, const RealDesc& R, RealCtl& C,
                                            const MixArgs& A, const int4& e0, const int4& e1) {
  const unsigned v = (unsigned)e0.x;
  const unsigned code = (unsigned)e0.y, valid = (code >> 21) & 63u;
  const unsigned pre = U.pre, updated = U.updated;
  const int d = (int)(code & 7u);
  const int off[6] = {(valid & 1u) ? -1 : 0, (valid & 2u) ? 1 : 0, (valid & 4u) ? -D.nz : 0, (valid & 8u) ? D.nz : 0,
                      (valid & 16u) ? -D.P : 0, (valid & 32u) ? D.P : 0};
  int dn[6];
  bool uniform = true;
#pragma unroll
  for (int q = 0; q < 6; q++) {
    dn[q] = (int)(code >> (3 + 3 * q)) & 7;
    uniform = uniform && dn[q] == d;
  }
  // every value first (out-of-box neighbours: the voxel itself), the first flux's too
  const unsigned m0 = (unsigned)e1.y;
  const int sp0 = (int)(m0 >> 8) & 0xff;
  float part = 0.f, self = 0.f;
  int ch_old = 0;
  if (!(m0 & MIX_NONE)) {
    const float* u = field(U.uo[sp0]);
    part = u[(unsigned)e1.x];
    self = u[v];
    if (m0 & MIX_CHANNEL) ch_old = A.states[(U.k & 1) * (long long)A.nch + e0.w];
  }
  float raw[MS], un[MS][6];
#pragma unroll
  for (int s = 0; s < MS; s++) {
    raw[s] = 0.f;
    if (!(updated >> s & 1u)) continue;
    const float* u = field(U.uo[s]) + v;
    raw[s] = u[0];
    if (!(pre >> s & 1u)) continue;
#pragma unroll
    for (int q = 0; q < 6; q++) un[s][q] = u[off[q]];
  }
  // fluxes of the item's species: the items of one species follow one another
  MixItem it{(unsigned)e1.x, m0, e1.z, e1.w};
  auto base = [&](unsigned dd, int s) -> double { return s == 0 ? D.base0[dd] : R.base[dd][s]; };
  auto fluxes = [&](int& sp, bool& apply, double& acc, bool& left, bool first) -> bool {
    bool any = false;
    sp = (int)(it.meta >> 8) & 0xff;
    acc = 0.0;
    while (true) {
      const unsigned meta = it.meta;
      if ((int)(meta >> 8 & 0xffu) != sp) return any;          // the next species' items
      apply = meta & MIX_APPLY;
      const bool to = meta & MIX_TO;
      double J = 0.0;
      bool on;
      if (meta & (MIX_SERCA | MIX_CHANNEL)) {
        on = U.sub >> ((meta >> 16) & 0xffu) & 1u;
        const unsigned ds = (meta >> 24) & 7u, dq = (meta >> 27) & 7u;
        if (!first) {
          const float* u = field(U.uo[sp]);
          part = u[it.vo];
          self = u[v];
        }
        const double us = (double)self + base(ds, sp), uo = (double)part + base(dq, sp);
        const double u0 = to ? uo : us, u1 = to ? us : uo;
        if (meta & MIX_SERCA) {
          if (on) J = serca_flux_fast(u0, u1, D.serca);
        } else {
          // the channel: gated on the Ca of its "to" voxel (species 0), then its flux
          const FluxParams& fp = D.gate[(meta & MIX_PRYR) ? 1 : 0];
          int s = ch_old;
          if (U.flags & STEP_GATE) {
            double c0 = u1;
            if (sp != 0) {
              const unsigned dt_ = to ? ds : dq;
              c0 = (double)field(U.uo[0])[to ? v : it.vo] + base(dt_, 0);
            }
            s = gate(fp, ch_old, c0, (double)(U.k + 1) * D.dt, D.dts, D.seed, D.stream, (unsigned)e0.z & 0xffffffu,
                     (unsigned)e0.z >> 24, U.k + 1);
          }
          if (meta & MIX_OWNER) {
            A.states[((U.k + 1) & 1) * (long long)A.nch + e0.w] = (unsigned char)s;
            if (s == 1) atomicAdd(&C.open_count[(U.k + 1) % 3], 1);
          }
          on = on && s == 1;
          if (on) J = ryr_flux(u0, u1, fp.k1);
        }
      } else {
        const FluxPair& pr = A.pairs[it.pair];
        on = mix_pair_flux(R, &C, it, pr, A.params[pr.param], U.uo[sp], U.uo[0], A.states, A.nch, U.k, J);
      }
      first = false;
      if (on) {
        acc += to ? J : -J;
        any = true;
      }
      if (meta & MIX_LAST) {
        left = false;
        return any;
      }
      const int4 q = __ldg(reinterpret_cast<const int4*>(A.items + it.more));
      it = MixItem{(unsigned)q.x, (unsigned)q.y, q.z, q.w};
    }
  };
  int sp = -1;
  bool apply = false, any = false, left = !(it.meta & MIX_NONE);
  double acc = 0.0;
  if (left) any = fluxes(sp, apply, acc, left, true);
  const bool react = U.flags & STEP_REACT, react_fast = U.flags & STEP_REACT_FAST;
  const unsigned fq = D.fixq & updated;           // fixed-point species: out[] holds the increment
  float val[MS], out[MS];
#pragma unroll
  for (int s = 0; s < MS; s++) {
    val[s] = (fq >> s & 1u) ? q_value(raw[s], D.qunit[d][s]) : raw[s];
    out[s] = (fq >> s & 1u) ? 0.f : val[s];
    if (!(pre >> s & 1u)) continue;
    const float* c = D.coef[s] + d * ND;
    out[s] = uniform ? diffuse_uniform(c[d], val[s], un[s]) : diffuse_general(c, dn, val[s], un[s]);
  }
  unsigned cls = RX_CLASS_NONE;
  if (react_fast) {
    const float dca = val[0], ca = __fadd_rn(D.fbase0[d], dca);
    if (SUR && D.sur) cls = rx_classify<MS>(R, d, ca, val);
    const unsigned rm = D.rmask[d];
#pragma unroll
    for (int s = 1; s < MS; s++) {
      if (!(rm >> s & 1u)) continue;
      const float4 ka = *reinterpret_cast<const float4*>(&D.rk2[d][s][0]);   // -kon, -kon, -koff, -koff
      const float4 kb = *reinterpret_cast<const float4*>(&D.rk2[d][s][2]);   // a, a, j0, j0
      const float dJ = buffer_dj(ka.x, ka.z, kb.x, kb.z, val[s], dca, ca);
      out[s] = __fadd_rn(out[s], dJ);
      out[0] = __fsub_rn(out[0], dJ);
    }
  } else if (react) {
    react_general<MS>(R, d, val, out, pre, fq);
  }
  const unsigned fm = D.fixed_mask[d];
#pragma unroll
  for (int s = 0; s < MS; s++) {
    if (fm >> s & 1u) out[s] = D.dinit[d][s];
    if (fq >> s & 1u) out[s] = (fm >> s & 1u) ? q_set(out[s], D.qinv[d][s]) : q_add(raw[s], out[s], D.qinv[d][s]);
  }
  if (D.dirichlet && valid != 63u) out[0] = D.dinit[d][0];
  while (sp >= 0) {
    if (any && apply && (updated >> sp & 1u)) put(out, sp, (float)((double)sel(out, sp) + acc));
    if (!left) break;
    any = fluxes(sp, apply, acc, left, false);
  }
#pragma unroll
  for (int s = 0; s < MS; s++)
    if (updated >> s & 1u) field(U.un[s])[v] = out[s];
  if (SUR && D.sur && react_fast) D.rx_class[v] = (unsigned char)cls;
}

__device__ __forceinline__ float part(const float4& q, int j) { return j == 0 ? q.x : j == 1 ? q.y : j == 2 ? q.z : q.w; }

// The four voxels of an irregular group (MixGroup) as mixed_voxel takes one: the same
// arithmetic per voxel, from values read 128 bits at a time.  A lane's chain is longer than a
// voxel's, so only batches with many irregular voxels have such entries (MIX_GROUPS_MIN).
// Bound by issue: 2,000 instructions per tile, half of the slots used by the 16 warps that 128
// registers allow, 0.06 of the DRAM bandwidth.
template <int MS, unsigned FQ, bool SUR>
__device__ __forceinline__ void mixed_group(const VoxDesc& D, const MarchStep& U, const RealDesc& R, const int4& e0,
                                            const int4& e1) {
  const unsigned v = (unsigned)e0.x;
  const unsigned flux = (unsigned)e0.y, order = (unsigned)e0.z;
  const unsigned code[4] = {(unsigned)e1.x, (unsigned)e1.y, (unsigned)e1.z, (unsigned)e1.w};
  const int nv = (int)(order >> 18);
  const unsigned pre = U.pre, updated = U.updated;
  const unsigned fq = FQ & D.fixq & updated;           // fixed-point species: out[] holds the increment
  const bool react = U.flags & STEP_REACT_FAST;   // (realisations with other reactions have no such entries)
  const int dym = (code[0] >> 23 & 1u) ? -D.nz : 0, dyp = (code[0] >> 24 & 1u) ? D.nz : 0;
  const int dxm = (code[0] >> 25 & 1u) ? -D.P : 0, dxp = (code[0] >> 26 & 1u) ? D.P : 0;
  const int dzm = (code[0] >> 21 & 1u) ? -1 : 0, dzp = (code[3] >> 22 & 1u) ? 4 : 3;
  float4 raw[MS];
#pragma unroll
  for (int s = 0; s < MS; s++)
    raw[s] = (updated >> s & 1u) ? *reinterpret_cast<const float4*>(field(U.uo[s]) + v) : make_float4(0.f, 0.f, 0.f, 0.f);
  float out[MS][4];
#pragma unroll
  for (int s = 0; s < MS; s++) {
#pragma unroll
    for (int j = 0; j < 4; j++) out[s][j] = (fq >> s & 1u) ? 0.f : part(raw[s], j);
    if (!(pre >> s & 1u)) continue;
    const float* u = field(U.uo[s]) + v;
    const float4 ym = *reinterpret_cast<const float4*>(u + dym), yp = *reinterpret_cast<const float4*>(u + dyp);
    const float4 xm = *reinterpret_cast<const float4*>(u + dxm), xp = *reinterpret_cast<const float4*>(u + dxp);
    const float zm = u[dzm], zp = u[dzp];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const unsigned c = code[j];
      const int d = (int)(c & 7u);
      const float self = part(raw[s], j);
      const float un[6] = {j == 0 ? zm : part(raw[s], j > 0 ? j - 1 : 0),
                           !(c >> 22 & 1u) ? self : j == 3 ? zp : part(raw[s], j < 3 ? j + 1 : 3),
                           part(ym, j), part(yp, j), part(xm, j), part(xp, j)};
      int dn[6];
#pragma unroll
      for (int q = 0; q < 6; q++) dn[q] = (int)(c >> (3 + 3 * q)) & 7;
      const bool uniform = (c >> 3 & 0x3ffffu) == (unsigned)d * 0x9249u;
      const float* co = D.coef[s] + d * ND;
      const float across = diffuse_general(co, dn, self, un), inside = diffuse_uniform(co[d], self, un);
      out[s][j] = uniform ? inside : across;         // (both, no branch: the lanes differ)
    }
  }
  // SERCA (boundaryfluxes.c:60-84) across the faces of all four voxels in one loop, so that a
  // warp takes as many turns as its lane with the most (random 2^3 blocks of domains: 8, where a
  // loop per voxel and face takes 24: 527 -> 471 us); the partner's value once more, from L1.
  // (Two fluxes per turn 512 us, the warp's fluxes dealt to its lanes the same.)
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  if (pre & 1u) {
    const float* u = field(U.uo[0]) + v;
    for (unsigned m = flux & 0x3f3f3f3fu; m; m &= m - 1u) {
      const int b = __ffs(m) - 1, j = b >> 3, k = (int)(order >> (3 * (b & 7))) & 7;
      const unsigned c = j == 0 ? code[0] : j == 1 ? code[1] : j == 2 ? code[2] : code[3];
      const int off = k == 0 ? -1 : k == 1 ? 1 : k == 2 ? dym : k == 3 ? dyp : k == 4 ? dxm : dxp;
      const double us = (double)u[j] + D.base0[c & 7u], uo = (double)u[j + off] + D.base0[(c >> (3 + 3 * k)) & 7u];
      const bool to = flux >> (8 * j) & MIXG_TO;
      const double J = serca_flux_fast(to ? uo : us, to ? us : uo, D.serca);
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (q == j) acc[q] += to ? J : -J;
    }
  }
  unsigned cls = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const unsigned c = code[j];
    const int d = (int)(c & 7u);
    float val[MS];
#pragma unroll
    for (int s = 0; s < MS; s++) val[s] = (fq >> s & 1u) ? q_value(part(raw[s], j), D.qunit[d][s]) : part(raw[s], j);
    if (react) {
      const float dca = val[0], ca = __fadd_rn(D.fbase0[d], dca);
      if (SUR && D.sur && j < nv) cls |= rx_classify<MS>(R, d, ca, val) << (8 * j);
      const unsigned rm = D.rmask[d];
#pragma unroll
      for (int s = 1; s < MS; s++) {
        const float4 ka = *reinterpret_cast<const float4*>(&D.rk2[d][s][0]);   // -kon, -kon, -koff, -koff
        const float4 kb = *reinterpret_cast<const float4*>(&D.rk2[d][s][2]);   // a, a, j0, j0
        const float dJ = buffer_dj(ka.x, ka.z, kb.x, kb.z, val[s], dca, ca);
        const bool on = rm >> s & 1u;              // (no branch: the lanes' domains differ)
        out[s][j] = on ? __fadd_rn(out[s][j], dJ) : out[s][j];
        out[0][j] = on ? __fsub_rn(out[0][j], dJ) : out[0][j];
      }
    }
    const unsigned fm = D.any_fixed ? D.fixed_mask[d] : 0u;
#pragma unroll
    for (int s = 0; s < MS; s++) {
      float& o = out[s][j];
      if (fm >> s & 1u) o = D.dinit[d][s];
      if (fq >> s & 1u) o = (fm >> s & 1u) ? q_set(o, D.qinv[d][s]) : q_add(part(raw[s], j), o, D.qinv[d][s]);
    }
    if (D.dirichlet && (c >> 21 & 63u) != 63u) out[0][j] = D.dinit[d][0];
    const unsigned f = flux >> (8 * j);
    if ((pre & 1u) && (f & 63u) && (f & MIXG_APPLY)) out[0][j] = (float)((double)out[0][j] + acc[j]);
  }
#pragma unroll
  for (int s = 0; s < MS; s++)
    if (updated >> s & 1u)
      *reinterpret_cast<float4*>(field(U.un[s]) + v) = make_float4(out[s][0], out[s][1], out[s][2], out[s][3]);
  if (SUR && D.sur && react) *reinterpret_cast<unsigned*>(D.rx_class + v) = cls;
}

// A CTA's share of a realisation's step: units [u0, u1) and boundary tiles [t0, t1) (of 32
// voxels, those with channels first), taken by its warps as they come free, units first.  Contiguous
// units share their columns' rows in L1; the tiles, whose lanes touch a line each, are spread
// evenly over the CTAs (16 of them on one SM took twice the time of one).
struct MarchShare {
  int u0, u1, t0, t1, tc, nc, nv;
  __device__ __forceinline__ MarchShare(const MarchReal& R, unsigned what, int rank, int size) {
    const long long units = (what & MARCH_UNITS) ? R.ncol * (long long)R.nseg : 0;
    nc = (what & MARCH_CHANNELS) ? R.nchan : 0;
    nv = (what & MARCH_VOXELS) ? R.nvox : 0;
    tc = (nc + 31) / 32;
    const long long tiles = tc + (nv + 31) / 32;
    u0 = (int)(units * rank / size);
    u1 = (int)(units * (rank + 1) / size);
    // the CTAs with one unit less get the odd tiles
    t0 = (int)(tiles * (size - 1 - rank) / size);
    t1 = (int)(tiles * (size - rank) / size);
  }
};

// The lane's entry of tile t; false: none.
__device__ __forceinline__ bool march_entry(const MarchArgs& A, const MarchReal& R, const MarchShare& H, int t, int4& e0,
                                            int4& e1) {
  const bool c = t < H.tc;
  const int i = (c ? t : t - H.tc) * 32 + (int)(threadIdx.x & 31u);
  if (t >= H.t1 || i >= (c ? H.nc : H.nv)) return false;
  const int4* e = reinterpret_cast<const int4*>((c ? A.mix.chan + R.chan0 : A.mix.vox + R.vox0) + i);
  e0 = __ldg(e);
  e1 = __ldg(e + 1);
  return true;
}
static_assert(sizeof(MixVoxel) == 32 && sizeof(MixGroup) == 32, "two 16-byte loads");

// A warp's next item of the step: the CTA's units, then its boundary tiles, are taken as warps
// come free.  Dealt in turn, the warps with a unit also got the later tiles while those that
// began with a tile were idle (us per step: 64 grids of 36x36x32 43.4 -> 41.9, 16 of 2.9 M
// voxels 309 -> 290, 40 of 100x100x50 185 -> 183, one of 100x100x50 7.5 -> 7.3).
__device__ __forceinline__ int march_next(MarchShared& S, int items) {
  int i = 0;
  if (items <= MARCH_T / 32) return items;
  if ((threadIdx.x & 31u) == 0) i = atomicAdd(&S.next, 1);
  return __shfl_sync(0xffffffffu, i, 0) + MARCH_T / 32;
}

// Boundary tiles (from tile k of the CTA on, then those the warp takes next; nu: the CTA's units).
template <int MS, bool SUR>
__device__ __noinline__ void march_mixed(const MarchArgs& A, const MarchReal& R, const MarchShare& H, int nu, int k) {
  extern __shared__ __align__(128) unsigned char smem[];
  MarchShared& S = *reinterpret_cast<MarchShared*>(smem);
  const int items = nu + H.t1 - H.t0;
  for (; k < items - nu; k = march_next(S, items) - nu) {
    int4 e0, e1;
    bool have;
    if (k < MARCH_T / 32) {
      const int i = k * 32 + (int)(threadIdx.x & 31u);
      e0 = S.tile[i][0];
      e1 = S.tile[i][1];
      have = e0.x != -1;
    } else {
      have = march_entry(A, R, H, H.t0 + k, e0, e1);
    }
    if (have) mixed_voxel<MS, SUR>(S.desc, S.step, A.descs[R.r], A.ctl[R.r], A.mix, e0, e1);
    __syncwarp();
  }
}

// The CTA's share of the irregular groups (entry e of the team), in tiles of 32 that its warps
// take as they come free.  A function and a counter of their own, not in MARCH_KNOWN.
template <int MS, unsigned FQ, bool SUR>
__device__ __noinline__ void march_groups(const MarchArgs& A, int e, int rank) {
  extern __shared__ __align__(128) unsigned char smem[];
  MarchShared& S = *reinterpret_cast<MarchShared*>(smem);
  const int r = A.real[e].r, n = A.real[e].ngrp, lane = (int)(threadIdx.x & 31u);
  const MixGroup* entries = A.mix.grp + A.real[e].grp0;
  const long long tiles = (n + 31) / 32;
  const int t0 = (int)(tiles * rank / A.size), t1 = (int)(tiles * (rank + 1) / A.size);
  while (true) {
    int t = 0;
    if (lane == 0) t = t0 + atomicAdd(&S.next_group, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= t1) break;
    if (t * 32 + lane < n) {
      const int4* g = reinterpret_cast<const int4*>(entries + t * 32 + lane);
      const int4 e0 = __ldg(g), e1 = __ldg(g + 1);
      mixed_group<MS, FQ, SUR>(S.desc, S.step, A.descs[r], e0, e1);
    }
    __syncwarp();
  }
}

template <int MS, unsigned FQ, bool SUR, int BODY>
__global__ void __launch_bounds__(MARCH_T, 1) k_march(const __grid_constant__ MarchArgs A) {
  extern __shared__ __align__(128) unsigned char smem[];
  MarchShared& S = *reinterpret_cast<MarchShared*>(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int team = blockIdx.x / A.size, rank = blockIdx.x - team * A.size;
  unsigned target = 0;                   // arrivals after which the team's next barrier opens
  if (A.inject && blockIdx.x == 0) {
    // test hook: this CTA leaves without arriving, so that the waits of its team run out.  Where
    // no CTA will wait for it, one thread waits for an arrival that nothing makes.
    bool waited_for = false;
    if (A.size > 1 && A.nsteps > 0 && (A.what & (MARCH_ADVANCE | MARCH_REPEAT)))
      for (int e = A.first[0]; e < A.first[1]; e++) waited_for = waited_for || !A.ctl[A.real[e].r].stopped;
    if (!waited_for && tid == 37) march_wait(A.arrived + 31, 1u, A.wait_ns, A.err);
    return;
  }
  for (int e = A.first[team]; e < A.first[team + 1]; e++) {
    const MarchReal R = A.real[e];
    const RealDesc& D = A.descs[R.r];
    RealCtl& C = A.ctl[R.r];
    {
      const int4* src = reinterpret_cast<const int4*>(&A.vdescs[R.r]);
      int4* dst = reinterpret_cast<int4*>(&S.desc);
      for (int i = tid; i < (int)(sizeof(VoxDesc) / 16); i += MARCH_T) dst[i] = __ldg(src + i);
    }
    const MarchShare H(R, A.what, rank, A.size);
    const int nu = H.u1 - H.u0, items = nu + H.t1 - H.t0;
    for (int c = tid; c <= R.nseg; c += MARCH_T) S.cut[c] = __ldg(A.cuts + R.cut0 + c);
    {
      int4 e0 = make_int4(-1, 0, 0, 0), e1 = e0;
      if (!march_entry(A, R, H, H.t0 + warp, e0, e1)) e0.x = -1;
      S.tile[tid][0] = e0;
      S.tile[tid][1] = e1;
    }
    // warp 0 keeps the step counters, its lane 0 the abort rule's bookkeeping
    MarchCount count{};
    double last_closed = 0.0, dt = 0.0, tabort = 0.0;
    long long total = 0;
    int stopped = 0;
    if (tid == 0) {
      S.next = 0;
      if (BODY != MARCH_KNOWN) S.next_group = 0;
    }
    if (warp == 0) {
      const long long k = C.step;
      const unsigned cur = C.cur_mask[k & 1];
      stopped = C.stopped;
      last_closed = C.last_closed;
      dt = D.dt;
      tabort = D.has_channels ? D.tabort : 0.0;
      total = D.total_steps;
      count.init(D, k, lane);
      unsigned pre, updated, dsi, flags;
      count.next(lane, pre, updated, dsi, flags);
      if (lane < NS) {
        S.step.uo[lane] = D.u[(cur >> lane) & 1u][lane];
        S.step.un[lane] = D.u[((cur >> lane) & 1u) ^ 1u][lane];
      }
      if (lane == 0) {
        S.step.k = k;
        S.step.cur = cur;
        S.step.pre = pre; S.step.updated = updated; S.step.sub = dsi; S.step.flags = flags;
        S.step.go = stopped ? 0 : 1;
      }
    }
    __syncthreads();
    long long i = 0;
    for (; i < A.nsteps && S.step.go > 0; i++) {
      if (S.step.updated) {
        int item = warp;
        for (; item < nu; item = march_next(S, items)) {
          const int u = H.u0 + item, seg = u / R.ncol, col = u - seg * R.ncol;
          march_dispatch<MS, FQ, SUR, BODY>(S, A.descs, R.r, col, S.cut[seg], S.cut[seg + 1]);
          __syncwarp();
        }
        if (item < items) march_mixed<MS, SUR>(A, R, H, nu, item - nu);
        if constexpr (BODY != MARCH_KNOWN) {
          if (R.ngrp > 0 && (A.what & MARCH_VOXELS)) march_groups<MS, FQ, SUR>(A, e, rank);
        }
      }
      if (!(A.what & (MARCH_ADVANCE | MARCH_REPEAT))) break;
      __syncthreads();
      if (warp == 0) {
        target += (unsigned)A.size;
        if (A.size > 1 && lane == 0) march_arrive(A.arrived + team * 32);
        const bool adv = A.what & MARCH_ADVANCE;
        const long long ti = S.step.k + 1;
        const unsigned done = S.step.updated;
        unsigned pre = 0, updated = 0, dsi = 0, flags = 0;
        if (adv) count.next(lane, pre, updated, dsi, flags);
        bool ok = true;
        if (A.size > 1 && lane == 0) ok = march_wait(A.arrived + team * 32, target, A.wait_ns, A.err);
        // every lane has read the step's masks (votes and reductions are no memory barriers)
        __syncwarp();
        // the step is taken: every CTA of the team follows the same rules (see k_epilogue)
        if (adv && lane == 0) {
          if (tabort != 0) {
            const double tt = (double)ti * dt;
            if (__ldcg(&C.open_count[ti % 3])) {
              last_closed = -1.0;
            } else if (tabort >= 0) {
              if (last_closed < 0) last_closed = tt;
              if (tt - last_closed >= tabort) stopped = 1;
            }
          }
          if (ti >= total) stopped = 1;
          if (rank == 0) {
            C.open_count[(ti + 2) % 3] = 0;      // read after the previous barrier, counted next in two steps
            if (A.flags) A.flags[i * A.flag_stride + R.r] = stopped;
          }
          S.step.k = ti;
          S.step.cur ^= done;
          S.step.pre = pre; S.step.updated = updated; S.step.sub = dsi; S.step.flags = flags;
        }
        if (lane == 0) {
          S.next = 0;
          if (BODY != MARCH_KNOWN) S.next_group = 0;
          S.step.go = !ok ? -1 : stopped ? 0 : 1;
        }
        if (adv && lane < NS && (done >> lane & 1u)) {
          const float* o = S.step.uo[lane];
          S.step.uo[lane] = S.step.un[lane];
          S.step.un[lane] = const_cast<float*>(o);
        }
      }
      __syncthreads();
    }
    if (S.step.go < 0) return;
    if (tid == 0 && rank == 0 && (A.what & MARCH_ADVANCE)) {
      C.step = S.step.k;
      C.cur_mask[S.step.k & 1] = S.step.cur;
      C.last_closed = last_closed;
      C.stopped = stopped;
      write_steprec(D, C, A.rec[R.r]);
      if (A.flags)
        for (; i < A.nsteps; i++) A.flags[i * A.flag_stride + R.r] = stopped;
    }
    __syncthreads();                     // S is filled for the next realisation
  }
}

// ---- host ----

using MarchKernel = void (*)(const MarchArgs);

// The kernel of a batch: models of at most ms species, all of the reference model's shape
// (known: fixed point for species 4 alone) or not.
inline MarchKernel march_kernel(int ms, bool known, bool sur) {
  if (known) return sur ? k_march<5, 1u << 4, true, MARCH_KNOWN> : k_march<5, 1u << 4, false, MARCH_KNOWN>;
  if (ms == 5) return sur ? k_march<5, 0x1Eu, true, MARCH_MASKS> : k_march<5, 0x1Eu, false, MARCH_MASKS>;
  return sur ? k_march<8, 0xFEu, true, MARCH_RUNTIME> : k_march<8, 0xFEu, false, MARCH_RUNTIME>;
}

// Teams and units of a launch over realisations [r0, r1).
struct MarchPlan {
  int r0 = 0, r1 = 0;
  int teams = 0, size = 0;
  int nseg = 0;                      // segments of the first realisation
  bool known = false;                // march_kernel
  double step_us = 0.0;              // estimated time of a step
  // one allocation, from d_arrived on
  unsigned* d_arrived = nullptr;
  const MarchReal* d_real = nullptr;
  const int* d_first = nullptr;
  const int* d_cuts = nullptr;
};

// Cost of a plane by what its warps meet, and of the rest of a step, in us of a warp with the
// SM's others busy (measured on 100x100x50 grids: two planes of uniform groups 3.3 us, of
// regular ones 4.5, with SERCA flux 6.3; eight uniform planes 14 us).
constexpr double MARCH_US_START = 0.8, MARCH_US_PLANE = 1.25, MARCH_US_REGULAR = 1.9, MARCH_US_FLUX = 2.9,
                 MARCH_US_TILE = 3.0, MARCH_US_BARRIER = 2.5, MARCH_US_SYNC = 0.5;

// Cuts nx planes with prefix cost sums acc[0 .. nx] into n segments of about equal cost;
// returns the largest.
inline double march_cut(const std::vector<double>& acc, int n, std::vector<int>* cuts) {
  const int nx = (int)acc.size() - 1;
  double worst = 0.0;
  int x = 0;
  if (cuts) cuts->assign(1, 0);
  for (int s = 1; s <= n; s++) {
    const double want = acc[nx] * s / n;
    int e = s == n ? nx : x + 1;
    while (e < nx - (n - s) && acc[e] + 0.5 * (acc[e + 1] - acc[e]) <= want) e++;
    worst = std::max(worst, acc[e] - acc[x]);
    if (cuts) cuts->push_back(e);
    x = e;
  }
  return worst;
}

// march_cut's largest segment for 1, 2, ... segments: made once per realisation, since a plan asks
// for it for every number of teams.
inline std::vector<double> march_largest(const std::vector<double>& acc) {
  const int nx = (int)acc.size() - 1, most = std::min(nx, MARCH_CUTS - 1);
  std::vector<double> w(most);
  for (int n = 1; n <= most; n++) w[n - 1] = march_cut(acc, n, nullptr);
  return w;
}

// Estimated time (us) of one step of a realisation (columns ncol, march_largest, `tiles`
// boundary tiles) by a team of `size` CTAs: its items per CTA in rounds of its warps, and the
// barrier.  *nseg: the segments that give it (in: those to use, if positive).
inline double march_cost(long long ncol, const std::vector<double>& largest, long long tiles, int size, int* nseg) {
  const int W = MARCH_T / 32;
  double best = 1e300;
  const int most = (int)largest.size(), given = nseg ? *nseg : 0;
  int found = 1;
  for (int n = given > 0 ? std::min(given, most) : 1; n <= most; n++) {
    const double unit = MARCH_US_START + largest[n - 1];
    const long long nu = (ncol * n + size - 1) / size, nt = (tiles + size - 1) / size;
    const long long full = nu / W, part = nu % W;      // rounds of units, then the tiles
    double t = full * unit;
    const long long left = nt - (part ? W - part : 0);
    if (part) t += std::max(unit, nt > 0 ? MARCH_US_TILE : 0.0);
    if (left > 0) t += (double)((left + W - 1) / W) * MARCH_US_TILE;
    if (t < best) {
      best = t;
      found = n;
    }
    if (given > 0) break;
  }
  if (nseg) *nseg = found;
  return best + (size > 1 ? MARCH_US_BARRIER : MARCH_US_SYNC);
}

}  // namespace csp
