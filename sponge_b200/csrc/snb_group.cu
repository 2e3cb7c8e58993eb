// Lennard-Jones + erfc-screened Coulomb of the fused engine over the grouped
// list (snb_nl.cu, k_group_search): one row of partner atoms per group of up
// to eight sorted atoms of a cell.
//
// One warp takes a row 32 entries at a time, a partner atom j per lane, and
// runs over the group's i atoms, which it reads from shared memory as
// broadcasts.  The j atom is loaded once for eight pairs, its force stays in
// the lane's registers and is added to the accumulators once, and the i
// forces stay in registers for the whole row.  An entry carries an 8-bit mask
// of the i atoms it may pair with; the rows are sorted by distance to the
// group, so that for a far batch pairs of i atoms drop out by a warp vote
// before the expensive terms.
//
// What bounds it is instruction issue and its latencies: no pipe is above 40 %
// of its peak, DRAM moves 30 MB, L2 takes 5.2 M sector updates (a row kernel
// with one atom per row took 62 M single adds).  On the 99,639-atom box
// (cutoff 10 A, skin 2 A) the launch takes 150 us, where the row kernel with
// pruned rows took 187 us; on the 1M-atom soft-core box 1.28-1.34 ms against
// 1.95-2.03 ms; on 64 boxes of 200-2,000 waters 208 us against 280 us.
//
// A partner's force is summed over the group's atoms in 32 bits (two chains of
// four) and added once in 64, an i atom's along the lanes' shares of its row;
// energies and virials go to 64 bits after at most eight pairs.  The error of
// the forces against 64 bits over 30 boxes of 600 to 39,000 atoms is 0.99 of
// the row kernel's (geometric mean; median 1.01, 0.5 to 1.4).
//
// Five blocks of four warps per SM (96 registers): four blocks 158 us, six
// (spilling) 158 us.  Four i atoms at a time 158-164 us; the polynomial on
// unpaired FMAs 153 us; rows handed out by an atomic counter 170-180 us (the
// launch waits longer for its loads than the even end saves).
#include <algorithm>
#include <cfloat>
#include <mutex>
#include <type_traits>
#include <vector>

#include "snb_internal.h"

namespace snb {

constexpr int kGroupWarps = 4;
constexpr float kFarAway = 1e15f;  // beyond every cutoff, its square finite

// The hardware approximations without the scaling of subnormal arguments and
// results that rsqrtf, __expf and __fdividef add around them: a squared
// distance, exp(-x^2) for x <= 4 and 1 + x / 2 are normal numbers.
__device__ __forceinline__ float rsqrt_fast(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_fast(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two pairs at a time: the paired FP32 instructions of sm_100 take one issue
// slot for both, and the two chains hide each other's latency.
__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

// A kernel argument held in a register: left to itself the compiler reads it
// from the constant bank again for every pair (an eighth of all instructions).
__device__ __forceinline__ float in_register(float x) {
  float y;
  asm volatile("mov.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
struct PairConst {
  float cutoff2;
  float kx;     // beta 2 / sqrt(pi)
  float arg;    // -beta^2 log2(e)
  float half;   // beta / 2
};

// The screened-Coulomb factors erfc(x) and exp(-x^2) of two x = beta r, as
// erfc_and_exp forms them (its polynomial in 1 / (1 + x / 2) up to x = 4; FAR:
// also beyond).
template <bool FAR>
__device__ __forceinline__ float2 erfc_exp2(float2 r, float2 r2, const PairConst& c, float2* ex) {
  if (FAR) {
    float2 q;
    q.x = erfc_and_exp(2.0f * c.half * r.x, &ex->x);
    q.y = erfc_and_exp(2.0f * c.half * r.y, &ex->y);
    return q;
  }
  const float2 arg = __fmul2_rn(r2, both(c.arg));
  const float2 e = make_float2(exp2_fast(arg.x), exp2_fast(arg.y));
  *ex = e;
  const float2 u = __ffma2_rn(r, both(c.half), both(1.0f));
  const float2 t = make_float2(rcp_fast(u.x), rcp_fast(u.y));
  const float2 p = erfcx_poly(
      t, both(kErfcxFirst), [](float2 a, float2 x, float b) { return __ffma2_rn(a, x, both(b)); });
  return __fmul2_rn(p, e);
}

// Soft-core pair forms (LJ_soft_core.h:33-149) of a pair whose end states
// differ: force over r, LJ and Coulomb energies.
__device__ __noinline__ void soft_terms(float lam, float alp_A, float alp_B, float s6,
                                        float s6min, float beta, float AA, float AB, float BA,
                                        float BB, float r2, float qq, float* fs, float* elj,
                                        float* ec) {
  const float lam_ = 1.0f - lam;
  if (BA * AA != 0.f || BA + AA == 0.f) {
    const float r = sqrtf(r2), ir2 = 1.0f / r2, ir6 = ir2 * ir2 * ir2, br = beta * r;
    *fs = lam_ * (AB - AA * ir6) * ir6 * ir2 + lam * (BB - BA * ir6) * ir6 * ir2 -
          qq / (r * r * r) * (br * kTwoOverSqrtPi * expf(-br * br) + erfcf(br));
    *elj = lam_ * lj_energy(AA, AB, ir6) + lam * lj_energy(BA, BB, ir6);
    *ec = qq * erfcf(br) / r;
    return;
  }
  const float sA = sc_sigma6(AA, AB, s6, s6min), sB = sc_sigma6(BA, BB, s6, s6min);
  const float r6 = r2 * r2 * r2, r4 = r2 * r2;
  const float rA = powf(r6 + alp_A * sA, 0.16666667f);
  const float rB = powf(r6 + alp_B * sB, 0.16666667f);
  const float iA2 = 1.0f / (rA * rA), iA6 = iA2 * iA2 * iA2;
  const float iB2 = 1.0f / (rB * rB), iB6 = iB2 * iB2 * iB2;
  const float bA = beta * rA, bB = beta * rB;
  const float eA = erfcf(bA) / rA, eB = erfcf(bB) / rB;
  const float fA = r4 * (AB - AA * iA6) * iA6 * iA6 -
                   qq * r4 * (expf(-bA * bA) * kTwoOverSqrtPi * beta + eA) * iA6;
  const float fB = r4 * (BB - BA * iB6) * iB6 * iB6 -
                   qq * r4 * (expf(-bB * bB) * kTwoOverSqrtPi * beta + eB) * iB6;
  *fs = lam_ * fA + lam * fB;
  *elj = lam_ * lj_energy(AA, AB, iA6) + lam * lj_energy(BA, BB, iB6);
  *ec = qq * (lam_ * eA + lam * eB);
}

// Sums the 24 values over the 32 lanes: on return lane 4 g + t holds in v[t]
// the sum of value 3 g + t (t < 3).  Each step halves the values a lane
// keeps and sends the other half to its partner.
__device__ __forceinline__ void reduce24(float* v, int lane) {
#pragma unroll
  for (int h = 12, o = 16; h >= 3; h >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int k = 0; k < h; ++k) {
      const float send = up ? v[k] : v[k + h];
      const float keep = up ? v[k + h] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    v[k] += __shfl_xor_sync(0xffffffffu, v[k], 2);
    v[k] += __shfl_xor_sync(0xffffffffu, v[k], 1);
  }
}

__device__ __forceinline__ long long warp_sum_ll(long long x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Rows of the pair tables: 8 bytes an entry; flag of the row's atom.
constexpr int kRowNoLJ = 1;
__device__ __forceinline__ float2 table_entry(const float2* t, int bytes) {
  return *reinterpret_cast<const float2*>(reinterpret_cast<const char*>(t) + (unsigned)bytes);
}

enum { kPlain, kPass, kGeneral };  // how a batch is taken
template <int H>
using how_c = std::integral_constant<int, H>;

// Minimum image of two displacements along an axis.
__device__ __forceinline__ float2 image2(float2 d, float L, float rL) {
  return make_float2(min_image_axis(d.x, L, rL), min_image_axis(d.y, L, rL));
}

// SOFT: plain LJ, or of a soft-core box the rows of groups without a marked
// atom, or those with one.  Nearly all pairs of a marked row take the soft-core
// terms, so one such row by one warp outlasts the rest of the launch on boxes
// of less than 50,000 atoms: the marked rows have a launch of their own beside
// the others, in parts of about a batch (step of 19,200, 42,000 and 300,000
// atoms with 35 to 64 marked sites: 89, 116 and 565 us, in one launch with whole
// rows 112, 159 and 599).
enum { kNoSoft, kPlainRows, kMarkedRows };

template <bool ENERGY, bool VIRIAL, bool BATCH, int SOFT, bool FAR>
__global__ void __launch_bounds__(32 * kGroupWarps, ENERGY || VIRIAL ? 1 : 5)
k_lj_groups(GroupArgs a, Accumulators acc) {
  // a group's atoms by pairs: {-x0, -x1, -y0, -y1}, {-z0, -z1, q0, q1}
  __shared__ float4 sh_i[kGroupWarps][4][2];
  // their rows of the pair tables (byte offset, with flags in its low bits)
  __shared__ int2 sh_t[kGroupWarps][4];
  __shared__ int2 sh_tb[SOFT ? kGroupWarps : 1][4];
  __shared__ long long sh_f[kGroupWarps][96];
  if (a.nl_flags[kFlagListOverflow]) return;  // rows not written
  const int lane = threadIdx.x & 31;
  const int w = threadIdx.x >> 5;
  // A pass that keeps: every batch of every row is taken, and the i atoms
  // with a partner of the batch within cutoff + margin are noted in its
  // byte; the steps after it take only those (the others are beyond the
  // cutoff until the next pass, so the sums are the same bit for bit).
  const bool pass = a.prune != nullptr && a.prune[0] != 0;
  const bool kept = a.prune != nullptr && !pass;
  const float rmax = pass ? a.prune_r : a.cutoff;
  const PairConst pc{in_register(a.cutoff2), in_register(a.beta * kTwoOverSqrtPi),
                     in_register(-a.beta * a.beta * 1.4426950408889634f),
                     in_register(0.5f * a.beta)};
  // component c = lane + 32 r of the 32 x 3 forces of a batch: its atom's
  // lane and its axis
  int src[3], axis[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    src[r] = (lane + 32 * r) / 3;
    axis[r] = ((lane + 32 * r) - 3 * src[r]) * acc.fc;
  }
  // the marked rows are cut into parts of about a batch
  int units = a.ngroups << a.split_log2, split = a.split_log2;
  if (SOFT == kMarkedRows) {
    const int m = *a.nmarked;
    for (split = 4; split > 0 && (m << split) > (int)gridDim.x * kGroupWarps; --split) {
    }
    units = m << split;
  }
  for (int u = blockIdx.x * kGroupWarps + w; u < units; u += gridDim.x * kGroupWarps) {
    const int part = u & ((1 << split) - 1);
    const int id = SOFT == kMarkedRows ? a.marked[u >> split] : u >> split;
    const int2 g = a.group[id];
    if (g.y == 0) continue;
    const int cnt = a.row_count[id];
    const int nb = (cnt + 31) >> 5;
    const int b0 = (nb * part) >> split, b1 = (nb * (part + 1)) >> split;
    if (b0 == b1 && !(pass && part == 0)) continue;
    const SysGeom* gs = BATCH ? a.bv.sys + a.bv.sys_of[g.x] : nullptr;
    const float Lx = BATCH ? gs->cell.a11 : a.cell.a11, rLx = BATCH ? gs->rcell.a11 : a.rcell.a11;
    const float Ly = BATCH ? gs->cell.a22 : a.cell.a22, rLy = BATCH ? gs->rcell.a22 : a.rcell.a22;
    const float Lz = BATCH ? gs->cell.a33 : a.cell.a33, rLz = BATCH ? gs->rcell.a33 : a.rcell.a33;
    // the i atoms relative to the first one (nearest image)
    const int li = g.x + min(lane & 7, g.y - 1);
    const float4 p = a.pos[li];
    const int tl = a.type[li];
    const float cx = __shfl_sync(0xffffffffu, p.x, 0), cy = __shfl_sync(0xffffffffu, p.y, 0),
                cz = __shfl_sync(0xffffffffu, p.z, 0);
    const float ix = min_image_axis(p.x - cx, Lx, rLx), iy = min_image_axis(p.y - cy, Ly, rLy),
                iz = min_image_axis(p.z - cz, Lz, rLz);
    if (SOFT == kPlainRows && __any_sync(0xffffffffu, tl < 0)) continue;
    const int ta = (SOFT ? tl & 0x7fff : tl & ~kTypeNoLJ) * a.n_types * 8;
    const bool has_lj = !(tl & kTypeNoLJ);
    __syncwarp();
    if (lane < 8) {
      // beyond the group's end: an atom out of everything's reach
      float* s = reinterpret_cast<float*>(sh_i[w][lane >> 1]) + (lane & 1);
      s[0] = lane < g.y ? -ix : kFarAway;
      s[2] = -iy;
      s[4] = -iz;
      s[6] = p.w;
      const bool lj = has_lj && lane < g.y;
      reinterpret_cast<int*>(sh_t[w])[lane] = ta + (lj ? 0 : kRowNoLJ);
      if (SOFT)
        reinterpret_cast<int*>(sh_tb[w])[lane] = ((tl >> 15) & 0x7fff) * a.n_types_b * 8;
    }
    // The partners are taken in the image nearest to the first atom.  That
    // image is the nearest one to every i atom too, for all pairs within
    // rmax, when rmax plus the group's reach along an axis stays below half
    // the box; otherwise (a box of about two cutoffs) each pair is imaged.
    float slack = fminf(0.5f * Lx - fabsf(ix), fminf(0.5f * Ly - fabsf(iy), 0.5f * Lz - fabsf(iz)));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) slack = fminf(slack, __shfl_xor_sync(0xffffffffu, slack, o));
    const bool wide = !(slack > rmax * 1.0001f);
    const bool general = wide || SOFT == kMarkedRows;
    __syncwarp();
    float2 f[4][3];
#pragma unroll
    for (int k = 0; k < 4; ++k) f[k][0] = f[k][1] = f[k][2] = make_float2(0.f, 0.f);
    long long s_lj = 0, s_c = 0, s_v[6] = {0, 0, 0, 0, 0, 0};
    const unsigned* row = a.entry + (size_t)id * a.cap;
    unsigned char* bytes = a.mask + (size_t)id * (a.cap >> 5);
    const unsigned own_bits = (1u << g.y) - 1u;

    // One batch: the lane's partner at (jx, jy, jz) relative to the first
    // atom, two i atoms at a time.  kPass: a batch of a pass; kGeneral: pairs
    // imaged one by one or soft-core pairs, in a pass or not.  Returns whether
    // anything was within the cutoff.
    auto batch = [&](auto how, unsigned take, unsigned e, float jx, float jy, float jz, float qj,
                     int tj, float2* fj, float* en, float* v, unsigned* near) {
      constexpr bool GENERAL = decltype(how)::value == kGeneral;
      constexpr bool PASS = decltype(how)::value != kPlain;
      const unsigned em = e & own_bits;
      const int tj_row = (SOFT ? tj & 0x7fff : tj & ~kTypeNoLJ) * 8;
      bool some = false;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (!((take >> (2 * k)) & 3u)) continue;
        const float4 xy = sh_i[w][k][0], zq = sh_i[w][k][1];
        float2 dx = __fadd2_rn(both(jx), make_float2(xy.x, xy.y)),
               dy = __fadd2_rn(both(jy), make_float2(xy.z, xy.w)),
               dz = __fadd2_rn(both(jz), make_float2(zq.x, zq.y));
        if (GENERAL && wide) {
          dx = image2(dx, Lx, rLx);
          dy = image2(dy, Ly, rLy);
          dz = image2(dz, Lz, rLz);
        }
        const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
        bool in0 = r2.x < pc.cutoff2, in1 = r2.y < pc.cutoff2;
        in0 = in0 && (em >> (2 * k) & 1u);
        in1 = in1 && (em >> (2 * k) & 2u);
        if (PASS && pass) {
          const unsigned bits = em >> (2 * k);
          *near |= __any_sync(0xffffffffu, (bits & 1u) && r2.x < a.prune2) ? 1u << (2 * k) : 0u;
          *near |= __any_sync(0xffffffffu, (bits & 2u) && r2.y < a.prune2) ? 2u << (2 * k) : 0u;
        }
        if (!__any_sync(0xffffffffu, in0 || in1)) continue;
        some = true;
        const float2 rinv = make_float2(rsqrt_fast(r2.x), rsqrt_fast(r2.y));
        const float2 r = __fmul2_rn(r2, rinv);
        const float2 ir2 = __fmul2_rn(rinv, rinv);
        const float2 ir3 = __fmul2_rn(ir2, rinv);
        float2 ex;
        const float2 erfc_br = erfc_exp2<FAR>(r, r2, pc, &ex);
        const float2 hc = __ffma2_rn(__fmul2_rn(r, both(pc.kx)), ex, erfc_br);
        const float2 qq = __fmul2_rn(make_float2(zq.z, zq.w), both(-qj));
        float2 fs = __fmul2_rn(__fmul2_rn(qq, ir3), hc);
        float2 e_c = both(0.f), e_lj = both(0.f);
        if (ENERGY) e_c = __fmul2_rn(__fmul2_rn(neg2(qq), erfc_br), rinv);
        const int2 ti = sh_t[w][k];
        // water H: a type without LJ against every type (warp-uniform)
        if (!(ti.x & ti.y & kRowNoLJ)) {
          const float2 ab0 = table_entry(a.lj, (ti.x & ~7) + tj_row),
                       ab1 = table_entry(a.lj, (ti.y & ~7) + tj_row);
          const float2 ir6 = __fmul2_rn(ir3, ir3);
          float2 ir8 = __fmul2_rn(ir6, ir2);
          fs.x = fmaf(fmaf(-ab0.x, ir6.x, ab0.y), ir8.x, fs.x);
          fs.y = fmaf(fmaf(-ab1.x, ir6.y, ab1.y), ir8.y, fs.y);
          if (ENERGY) {
            e_lj.x = lj_energy(ab0.x, ab0.y, ir6.x);
            e_lj.y = lj_energy(ab1.x, ab1.y, ir6.y);
          }
          if (SOFT && GENERAL) {
            const int2 tb = sh_tb[w][k];
            const int tjb_row = ((tj >> 15) & 0x7fff) * 8;
            const float2 cd0 = table_entry(a.lj_b, tb.x + tjb_row),
                         cd1 = table_entry(a.lj_b, tb.y + tjb_row);
            if (in0 && (ab0.x != cd0.x || ab0.y != cd0.y))
              soft_terms(a.lambda, a.alp_A, a.alp_B, a.sigma6, a.sigma6_min, a.beta, ab0.x,
                         ab0.y, cd0.x, cd0.y, r2.x, -qq.x, &fs.x, &e_lj.x, &e_c.x);
            if (in1 && (ab1.x != cd1.x || ab1.y != cd1.y))
              soft_terms(a.lambda, a.alp_A, a.alp_B, a.sigma6, a.sigma6_min, a.beta, ab1.x,
                         ab1.y, cd1.x, cd1.y, r2.y, -qq.y, &fs.y, &e_lj.y, &e_c.y);
          }
        }
        fs.x = in0 ? fs.x : 0.f;
        fs.y = in1 ? fs.y : 0.f;
        f[k][0] = __ffma2_rn(fs, dx, f[k][0]);
        f[k][1] = __ffma2_rn(fs, dy, f[k][1]);
        f[k][2] = __ffma2_rn(fs, dz, f[k][2]);
        fj[0] = __ffma2_rn(fs, dx, fj[0]);
        fj[1] = __ffma2_rn(fs, dy, fj[1]);
        fj[2] = __ffma2_rn(fs, dz, fj[2]);
        if (ENERGY) {
          en[0] += (in0 ? e_lj.x : 0.f) + (in1 ? e_lj.y : 0.f);
          en[1] += (in0 ? e_c.x : 0.f) + (in1 ? e_c.y : 0.f);
        }
        if (VIRIAL) {
          const float2 hx = __fmul2_rn(fs, dx), hy = __fmul2_rn(fs, dy), hz = __fmul2_rn(fs, dz);
          v[0] -= hx.x * dx.x + hx.y * dx.y;
          v[1] -= 2.0f * (hx.x * dy.x + hx.y * dy.y);
          v[2] -= hy.x * dy.x + hy.y * dy.y;
          v[3] -= 2.0f * (hx.x * dz.x + hx.y * dz.y);
          v[4] -= 2.0f * (hy.x * dz.x + hy.y * dz.y);
          v[5] -= hz.x * dz.x + hz.y * dz.y;
        }
      }
      return some;
    };

    for (int c0 = b0; c0 < b1; c0 += 32) {
      // the next (up to) 32 batches: lane k holds the i atoms of batch c0 + k
      const unsigned mine = c0 + lane < b1 ? (kept ? (unsigned)bytes[c0 + lane] : 0xffu) : 0u;
      unsigned todo = __ballot_sync(0xffffffffu, mine != 0u);
      if (todo == 0u) continue;
      // entries are loaded two batches ahead, partners one ahead
      auto entry_of = [&](unsigned t) {
        const int k = 32 * (c0 + __ffs(t) - 1) + lane;
        return t != 0u && k < cnt ? row[k] : 0u;
      };
      unsigned e1 = entry_of(todo), e2 = entry_of(todo & (todo - 1));
      float4 p1 = a.pos[e1 >> 8];
      int t1 = a.type[e1 >> 8];
      while (todo != 0u) {
        const int bk = __ffs(todo) - 1;
        todo &= todo - 1;
        const unsigned take = __shfl_sync(0xffffffffu, mine, bk);
        const unsigned e = e1;
        const float4 pj = p1;
        const int tj = t1;
        e1 = e2;
        p1 = a.pos[e1 >> 8];
        t1 = a.type[e1 >> 8];
        e2 = entry_of(todo & (todo - 1));
        // a lane without an entry (mask 0): out of everything's reach
        const bool none = (e & 0xffu) == 0u;
        const float jx = none ? kFarAway : min_image_axis(pj.x - cx, Lx, rLx);
        const float jy = min_image_axis(pj.y - cy, Ly, rLy);
        const float jz = min_image_axis(pj.z - cz, Lz, rLz);
        float2 fj[3] = {both(0.f), both(0.f), both(0.f)};
        float en[2] = {0.f, 0.f};
        float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        unsigned near = 0u;
        const bool marked = SOFT && tj < 0;
        bool some;
        if (general || (SOFT && __any_sync(0xffffffffu, marked)))
          some = batch(how_c<kGeneral>(), take, e, jx, jy, jz, pj.w, tj, fj, en, v, &near);
        else if (pass)
          some = batch(how_c<kPass>(), take, e, jx, jy, jz, pj.w, tj, fj, en, v, &near);
        else
          some = batch(how_c<kPlain>(), take, e, jx, jy, jz, pj.w, tj, fj, en, v, &near);
        if (pass && lane == 0) bytes[c0 + bk] = (unsigned char)near;
        if (!some) continue;
        if (ENERGY) {
          s_lj += to_fixed_energy(en[0]);
          s_c += to_fixed_energy(en[1]);
        }
        if (VIRIAL) {
#pragma unroll
          for (int c = 0; c < 6; ++c) s_v[c] += to_fixed_energy(v[c]);
        }
        // The batch's forces by component: consecutive lanes take the three
        // components of an atom, which lie in one 32-byte sector, so a
        // partner costs one sector update instead of three.
        const int j4 = (int)(e >> 8) * acc.fs;
        long long* sf = sh_f[w];
        sf[3 * lane] = to_fixed_force(-(fj[0].x + fj[0].y));
        sf[3 * lane + 1] = to_fixed_force(-(fj[1].x + fj[1].y));
        sf[3 * lane + 2] = to_fixed_force(-(fj[2].x + fj[2].y));
        __syncwarp();
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          const long long q = sf[lane + 32 * r];
          const int at = __shfl_sync(0xffffffffu, j4, src[r]);
          if (q != 0) red_add(acc.d_f + at + axis[r], q);
        }
        __syncwarp();
      }
    }

    float s[24];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        s[6 * k + c] = f[k][c].x;
        s[6 * k + 3 + c] = f[k][c].y;
      }
    reduce24(s, lane);
    {
      const int t = lane & 3, ia = lane >> 2;
      const float x = t == 0 ? s[0] : (t == 1 ? s[1] : s[2]);
      if (t < 3 && ia < g.y)
        red_add(acc.d_f + (g.x + ia) * acc.fs + t * acc.fc, to_fixed_force(x));
    }
    if (ENERGY) {
      s_lj = warp_sum_ll(s_lj);
      s_c = warp_sum_ll(s_c);
      if (lane == 0) {
        red_add(acc.d_e + g.x, s_lj + s_c);
        red_add(acc.d_elj + g.x, s_lj);
        red_add(acc.d_ec + g.x, s_c);
      }
    }
    if (VIRIAL) {
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        const long long x = warp_sum_ll(s_v[c]);
        if (lane == 0) red_add(acc.d_v + c * acc.n + g.x, x);
      }
    }
    if (pass && part == 0 && lane < g.y) a.prune_ref[g.x + lane] = p;
  }
}

using GroupKern = void (*)(GroupArgs, Accumulators);

template <bool BATCH, int SOFT, bool FAR>
static GroupKern group_kernel(bool energy, bool virial) {
  return energy ? (virial ? k_lj_groups<true, true, BATCH, SOFT, FAR>
                          : k_lj_groups<true, false, BATCH, SOFT, FAR>)
                : (virial ? k_lj_groups<false, true, BATCH, SOFT, FAR>
                          : k_lj_groups<false, false, BATCH, SOFT, FAR>);
}

template <bool FAR>
static GroupKern group_kernel(bool batch, int soft, bool energy, bool virial) {
  return soft == kPlainRows    ? group_kernel<false, kPlainRows, FAR>(energy, virial)
         : soft == kMarkedRows ? group_kernel<false, kMarkedRows, FAR>(energy, virial)
         : batch               ? group_kernel<true, kNoSoft, FAR>(energy, virial)
                               : group_kernel<false, kNoSoft, FAR>(energy, virial);
}

static GroupKern group_kernel(const GroupArgs& a, int soft, bool energy, bool virial) {
  const bool batch = a.bv.nsys > 0;
  return a.beta * a.cutoff > 4.0f ? group_kernel<true>(batch, soft, energy, virial)
                                  : group_kernel<false>(batch, soft, energy, virial);
}

// The SM's shared memory is laid out for the first kernel on it, and a kernel
// that needs more waits until the SM has drained.  The pair kernel's own 19 KB
// would keep the PME branch's spread by tiles off its SMs, so that the tiles
// pile up on the first ones to finish: with 6 boxes of 420 waters the spread
// took 32 us beside it and the step 85 us, with 64 KB laid out 73 us (15 % and
// less: 85, 25 to 100 %: 73; boxes of 648 to 100,000 atoms: no difference).
static void leave_shared_memory(GroupKern k) {
  static std::mutex mu;
  static std::vector<GroupKern> done;
  std::lock_guard<std::mutex> lock(mu);
  if (std::find(done.begin(), done.end(), k) != done.end()) return;
  cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 30);
  done.push_back(k);
}

static int multiprocessors() {
  static int sms = 0;
  if (!sms) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0);
  return sms;
}

int launch_marked_groups(GroupArgs a, Accumulators& acc, bool energy, bool virial,
                         cudaStream_t st) {
  if (a.n <= 0) return kOk;
  GroupKern kern = group_kernel(a, kMarkedRows, energy, virial);
  leave_shared_memory(kern);
  // all resident blocks: the marked groups may be all of them (every water's LJ
  // changed, 28,000 waters: step 251 us, with one block per SM 613)
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kGroupWarps, 0);
  const int blocks = std::min(ceil_div((long long)a.ngroups << 4, kGroupWarps),
                              multiprocessors() * std::max(per_sm, 1));
  kern<<<blocks, 32 * kGroupWarps, 0, st>>>(a, acc);
  SNB_CUDA_TRY(cudaGetLastError());
  return kOk;
}

int launch_pair_groups(GroupArgs a, Accumulators& acc, bool energy, bool virial,
                       cudaStream_t st) {
  if (a.n <= 0) return kOk;
  GroupKern kern = group_kernel(a, a.lj_b ? kPlainRows : kNoSoft, energy, virial);
  leave_shared_memory(kern);
  const int sms = multiprocessors();
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kGroupWarps, 0);
  per_sm = std::max(per_sm, 1);
  // (a caller's limit is in units of 512 threads; five blocks of 128 fit, so
  // only a limit of one is below the occupancy maximum)
  if (a.blocks_per_sm > 0) per_sm = std::min(per_sm, a.blocks_per_sm * (16 / kGroupWarps));
  // The rows of a small box are cut into parts until there are enough for the
  // 2,960 warps to have work (9,000 atoms: 26 us in two parts, 32 us whole);
  // a larger box's are taken whole, because every part costs a chain of loads
  // and a reduction (100k atoms in two parts each: 181 us against 151 us).
  a.split_log2 = 0;
  while (a.split_log2 < 3 && ((long long)a.ngroups << a.split_log2) < 2048) ++a.split_log2;
  // Persistent blocks, except where one unit per warp needs no more than twice
  // as many: a second round for a few warps is longer than a second wave of
  // blocks (9,000 atoms: the step 55.9 us against 58.4 us; on 100,000 the
  // second wave costs 10 us instead).
  const int resident = sms * per_sm;
  const int all = ceil_div((long long)a.ngroups << a.split_log2, kGroupWarps);
  const int blocks = std::max(1, all <= 2 * resident ? all : resident);
  kern<<<blocks, 32 * kGroupWarps, 0, st>>>(a, acc);
  SNB_CUDA_TRY(cudaGetLastError());
  return kOk;
}

}  // namespace snb
