// Direct-space Lennard-Jones + erfc-screened Coulomb over the sorted half list:
// the Lennard_Jones_And_Direct_Coulomb_Device path
// (Lennard_Jones_force.cpp:45-137, pair terms Lennard_Jones_force.h:45-75)
// re-designed for sm_100a.
//
// Per listed pair (i, j) with r = |r_j - r_i| (minimum image) below cutoff:
//   F/r = (B' - A' r^-6) r^-8 - q_i q_j r^-3 (2 beta r/sqrt(pi) e^{-beta^2 r^2}
//         + erfc(beta r))
//   f_i += (F/r) dr, f_j -= (F/r) dr
//   E_LJ = (A'/12 r^-6 - B'/6) r^-6, E_C = q_i q_j erfc(beta r)/r
//   virial -= (F/r) dr (x) dr   (LTMatrix3 with summed off-diagonals)
// Energy and virial of a pair go to the atom with the smaller global id, as
// the reference's half list (global_j > global_i) assigns them.
//
// Layout: one warp per sorted atom i, lanes stride its CSR row (coalesced
// 4-byte index loads, 16-byte float4 {x,y,z,q} gathers that hit L1/L2 since
// the rows of neighbouring i are spatial neighbours).  The i force stays in
// registers and is reduced with warp shuffles; j forces go straight to the
// accumulators: 64-bit fixed point (deterministic, order-independent) or
// float atomics (the plain path).
#include <algorithm>
#include <cfloat>

#include <mutex>
#include <utility>
#include <vector>

#include "snb_internal.h"

namespace snb {

template <int ACCUM>
__device__ __forceinline__ void add_force(Accumulators& acc, int s, float fx,
                                          float fy, float fz) {
  const int N = acc.n;
  if (ACCUM == kAccumFixed) {
    red_add(acc.d_f + s * acc.fs, to_fixed_force(fx));
    red_add(acc.d_f + s * acc.fs + acc.fc, to_fixed_force(fy));
    red_add(acc.d_f + s * acc.fs + 2 * acc.fc, to_fixed_force(fz));
  } else {
    atomicAdd(acc.d_ff + s, fx);
    atomicAdd(acc.d_ff + N + s, fy);
    atomicAdd(acc.d_ff + 2 * N + s, fz);
  }
}

template <int ACCUM>
__device__ __forceinline__ void add_energy(Accumulators& acc, int s, float e,
                                           float elj, float ec) {
  const int N = acc.n;
  if (ACCUM == kAccumFixed) {
    red_add(acc.d_e + s, to_fixed_energy(e));
    red_add(acc.d_elj + s, to_fixed_energy(elj));
    red_add(acc.d_ec + s, to_fixed_energy(ec));
  } else {
    atomicAdd(acc.d_fe + s, e);
    atomicAdd(acc.d_fe + N + s, elj);
    atomicAdd(acc.d_fe + 2 * N + s, ec);
  }
}

template <int ACCUM>
__device__ __forceinline__ void add_virial(Accumulators& acc, int s, const float* v) {
  const int N = acc.n;
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    if (ACCUM == kAccumFixed)
      red_add(acc.d_v + c * N + s, to_fixed_energy(v[c]));
    else
      atomicAdd(acc.d_fv + c * N + s, v[c]);
  }
}

// Each warp owns one row at a time and takes it in two phases.  Phase 1
// scans the listed candidates, four per lane in flight (index loads, then
// float4 gathers), and appends the j inside the cutoff to a per-warp list in
// shared memory (ballot + popc).  Phase 2 runs the pair terms over that list
// 32 pairs at a time, so every lane of the expensive part does useful work
// and the scan carries no force state.  A row with more hits than the list
// holds is taken in several rounds.
constexpr int kWarps = 8;      // rows in flight per block (warps per block)
constexpr int kHitCap = 512;   // per-warp hit list (entries)
constexpr int kScanU = 4;      // candidates per lane per scan round

// The pair terms of i and j with the LJ coefficients A' = 12 A, B' = 6 B of
// their type pair.  COUL_ONLY: atom i's type has A' = B' = 0 with every
// type, so the LJ terms are exact zeros and are not formed (the results are
// bitwise the same).
template <int ACCUM, bool ENERGY, bool VIRIAL, bool COUL_ONLY = false, typename Args>
__device__ __forceinline__ void lj_pair_ab(const Args& a, Accumulators& acc, float A,
                                           float B, float qi, int gi, float4 e, int j,
                                           float& fx, float& fy, float& fz, float& e_lj,
                                           float& e_c, float* vir) {
  const float r2 = e.x * e.x + e.y * e.y + e.z * e.z;
  const float rinv = rsqrtf(r2);
  const float r = r2 * rinv;
  const float ir2 = rinv * rinv;
  const float ir6 = ir2 * ir2 * ir2;
  const float flj = COUL_ONLY ? 0.f : (B - A * ir6) * ir6 * ir2;
  const float qq = qi * e.w;
  const float br = a.beta * r;
  float ex;
  const float erfc_br = erfc_and_exp(br, &ex);
  const float fc = qq * rinv * ir2 * (br * kTwoOverSqrtPi * ex + erfc_br);
  const float fs = flj - fc;
  const float gx = fs * e.x, gy = fs * e.y, gz = fs * e.z;
  fx += gx;
  fy += gy;
  fz += gz;
  add_force<ACCUM>(acc, j, -gx, -gy, -gz);
  if (ENERGY || VIRIAL) {
    const bool own_i = gi < a.global[j];
    if (ENERGY) {
      const float elj = COUL_ONLY ? 0.f : lj_energy(A, B, ir6);
      const float ec = qq * erfc_br * rinv;
      if (own_i) {
        e_lj += elj;
        e_c += ec;
      } else {
        add_energy<ACCUM>(acc, j, elj + ec, elj, ec);
      }
    }
    if (VIRIAL) {
      float v[6];
      v[0] = -(gx * e.x);
      v[1] = -(gx * e.y + gy * e.x);
      v[2] = -(gy * e.y);
      v[3] = -(gx * e.z + gz * e.x);
      v[4] = -(gy * e.z + gz * e.y);
      v[5] = -(gz * e.z);
      if (own_i) {
#pragma unroll
        for (int c = 0; c < 6; ++c) vir[c] += v[c];
      } else {
        add_virial<ACCUM>(acc, j, v);
      }
    }
  }
}

// The same with the coefficients looked up from the types' pair index.
template <int ACCUM, bool ENERGY, bool VIRIAL, bool COUL_ONLY = false, typename Args>
__device__ __forceinline__ void lj_pair(const Args& a, Accumulators& acc,
                                        const float* sA, const float* sB, int ti,
                                        float qi, int gi, float4 e, int j, int tj,
                                        float& fx, float& fy, float& fz, float& e_lj,
                                        float& e_c, float* vir) {
  float A = 0.f, B = 0.f;
  if (!COUL_ONLY) {
    const int p = lj_pair_index(ti, tj);
    A = sA[p];
    B = sB[p];
  }
  lj_pair_ab<ACCUM, ENERGY, VIRIAL, COUL_ONLY>(a, acc, A, B, qi, gi, e, j, fx, fy, fz, e_lj,
                                               e_c, vir);
}

// SOLV 1 / 2: the solvent split of PairArgs::solvent_mode (pairs with both
// global ids >= solvent_begin left out / taken alone); 0: every pair.
template <int ACCUM, bool ENERGY, bool VIRIAL, bool ORTHO, bool BATCH, int SOLV = 0>
__global__ void __launch_bounds__(32 * kWarps, 32 / kWarps)
k_lj_direct(PairArgs a, Accumulators acc) {
  static_assert(32 * kScanU < kHitCap, "scan round exceeds the hit list");
  extern __shared__ float sh_dyn[];
  __shared__ int hits_all[kWarps][kHitCap];
  const int npair = a.n_types * (a.n_types + 1) / 2;
  float* sA = sh_dyn;
  float* sB = sA + npair;
  for (int k = threadIdx.x; k < npair; k += blockDim.x) {
    sA[k] = a.A[k];
    sB[k] = a.B[k];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int w = threadIdx.x >> 5;
  int* hits = hits_all[w];
  if (a.nl_flags && a.nl_flags[1]) return;  // list overflowed: rows not written
  const int* __restrict__ cols = a.cols;
  const int* __restrict__ rcount = a.row_count;
  // Each block owns a contiguous range of sorted atoms, so the neighbours its
  // warps gather overlap and stay in this SM's L1.
  const int per_block = (a.n + gridDim.x - 1) / gridDim.x;
  const int i_begin = blockIdx.x * per_block;
  const int i_end = min(a.n, i_begin + per_block);
  const unsigned lt = (1u << lane) - 1u;
  for (int i = i_begin + w; i < i_end; i += kWarps) {
  const float4 pi = a.pos[i];
  const float3 ri = make_float3(pi.x, pi.y, pi.z);
  const int ti = a.type[i];
  const int gi = ENERGY || VIRIAL || SOLV ? a.global[i] : 0;
  const bool i_solvent = SOLV && gi >= a.solvent_begin;
  // box of atom i (and of all its pairs)
  const SysGeom* gs = BATCH ? a.bv.sys + a.bv.sys_of[i] : nullptr;
  const Cell& cell = BATCH ? gs->cell : a.cell;
  const Cell& rcell = BATCH ? gs->rcell : a.rcell;
  float fx = 0.f, fy = 0.f, fz = 0.f;
  float e_lj = 0.f, e_c = 0.f;
  float vir[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const int k0 = a.row_start[i], k1 = k0 + rcount[i];
  // a type without LJ against every type (water H): Coulomb-only row
  bool coul_only = true;
  for (int t = lane; t < a.n_types; t += 32) {
    const int p = lj_pair_index(ti, t);
    coul_only = coul_only && sA[p] == 0.f && sB[p] == 0.f;
  }
  coul_only = __all_sync(0xffffffffu, coul_only);
  {
    // the warp's next row: start pulling its indices from HBM into L2 now
    // (row starts are multiples of 8 entries, so 16-byte aligned)
    const int inext = i + kWarps;
    if (lane == 0 && inext < i_end) {
      const int cn = rcount[inext];
      if (cn > 0)
        prefetch_l2(cols + a.row_start[inext], (unsigned)(cn * 4 + 15) & ~15u);
    }
  }
  // hits of the row taken in earlier rounds: lane l takes the row's hits
  // l, l + 32, ... in order whatever the rounds, so the float sums of i's
  // force do not depend on how the rounds fall
  int done = 0;
  // each round's indices are loaded one round ahead, so the gathers of a
  // round wait only on their own load.  The index stream is read once:
  // loaded evict-first (__ldcs) so that L1 keeps the positions the rows share.
  int jn[kScanU];
#pragma unroll
  for (int u = 0; u < kScanU; ++u) {
    const int k = k0 + 32 * u + lane;
    jn[u] = k < k1 ? __ldcs(cols + k) : -1;
  }
  for (int base = k0; base < k1;) {
    // phase 1: candidates -> hit list
    int count = 0;
    for (; base < k1 && count <= kHitCap - 32 * kScanU; base += 32 * kScanU) {
      int jj[kScanU];
#pragma unroll
      for (int u = 0; u < kScanU; ++u) {
        jj[u] = jn[u];
        const int k = base + 32 * (kScanU + u) + lane;
        jn[u] = k < k1 ? __ldcs(cols + k) : -1;
      }
      float4 pp[kScanU];
#pragma unroll
      for (int u = 0; u < kScanU; ++u)
        if (jj[u] >= 0) pp[u] = a.pos[jj[u]];
#pragma unroll
      for (int u = 0; u < kScanU; ++u) {
        bool in = false;
        if (jj[u] >= 0) {
          const float3 dr = min_image_fast<ORTHO>(make_float3(pp[u].x, pp[u].y, pp[u].z),
                                                  ri, cell, rcell);
          in = dr.x * dr.x + dr.y * dr.y + dr.z * dr.z < a.cutoff2;
          if (SOLV && in) {
            const bool both = i_solvent && a.global[jj[u]] >= a.solvent_begin;
            in = SOLV == 1 ? !both : both;
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) hits[count + __popc(m & lt)] = jj[u];
        count += __popc(m);
      }
    }
    __syncwarp();
    // phase 2: pair terms over the hit list
    const int h0 = (lane - done) & 31;
    if (coul_only) {
      for (int h = h0; h < count; h += 32) {
        const int j = hits[h];
        const float4 pj = a.pos[j];
        const float3 dr = min_image_fast<ORTHO>(make_float3(pj.x, pj.y, pj.z), ri, cell,
                                                rcell);
        lj_pair<ACCUM, ENERGY, VIRIAL, true>(a, acc, sA, sB, ti, pi.w, gi,
                                             make_float4(dr.x, dr.y, dr.z, pj.w), j, 0, fx,
                                             fy, fz, e_lj, e_c, vir);
      }
    } else {
      for (int h = h0; h < count; h += 32) {
        const int j = hits[h];
        const float4 pj = a.pos[j];
        const int tj = a.type[j];
        const float3 dr = min_image_fast<ORTHO>(make_float3(pj.x, pj.y, pj.z), ri, cell,
                                                rcell);
        lj_pair<ACCUM, ENERGY, VIRIAL>(a, acc, sA, sB, ti, pi.w, gi,
                                       make_float4(dr.x, dr.y, dr.z, pj.w), j, tj, fx, fy,
                                       fz, e_lj, e_c, vir);
      }
    }
    done += count;
    __syncwarp();
  }
  fx = warp_sum(fx);
  fy = warp_sum(fy);
  fz = warp_sum(fz);
  if (ENERGY) {
    e_lj = warp_sum(e_lj);
    e_c = warp_sum(e_c);
  }
  if (VIRIAL) {
#pragma unroll
    for (int c = 0; c < 6; ++c) vir[c] = warp_sum(vir[c]);
  }
  if (lane == 0) {
    add_force<ACCUM>(acc, i, fx, fy, fz);
    if (ENERGY) add_energy<ACCUM>(acc, i, e_lj + e_c, e_lj, e_c);
    if (VIRIAL) add_virial<ACCUM>(acc, i, vir);
  }
  }
}

using RowKern = void (*)(PairArgs, Accumulators);

// Raises a kernel's dynamic shared memory limit once, when it needs more
// than the default 48 KB.
static void allow_smem(RowKern k, size_t smem) {
  static std::mutex mu;
  static std::vector<std::pair<RowKern, size_t>> done;
  if (smem <= 48 * 1024) return;
  std::lock_guard<std::mutex> lock(mu);
  for (auto& d : done)
    if (d.first == k && d.second >= smem) return;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  done.push_back({k, smem});
}

template <int ACCUM, bool ENERGY, bool VIRIAL>
static void launch3(const PairArgs& a, Accumulators& acc, bool ortho, cudaStream_t st) {
  const size_t smem = sizeof(float) * a.n_types * (a.n_types + 1);
  RowKern kern;
  if (a.solvent_mode != 0 && a.bv.nsys == 0)
    kern = ortho ? (a.solvent_mode == 1 ? k_lj_direct<ACCUM, ENERGY, VIRIAL, true, false, 1>
                                        : k_lj_direct<ACCUM, ENERGY, VIRIAL, true, false, 2>)
                 : (a.solvent_mode == 1 ? k_lj_direct<ACCUM, ENERGY, VIRIAL, false, false, 1>
                                        : k_lj_direct<ACCUM, ENERGY, VIRIAL, false, false, 2>);
  else if (a.bv.nsys > 0)
    kern = k_lj_direct<ACCUM, ENERGY, VIRIAL, true, true>;
  else
    kern = ortho ? k_lj_direct<ACCUM, ENERGY, VIRIAL, true, false>
                 : k_lj_direct<ACCUM, ENERGY, VIRIAL, false, false>;
  allow_smem(kern, smem);
  // persistent grid: as many blocks as fit at once
  static int sms = 0;
  if (!sms) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kWarps, smem);
  per_sm = std::max(per_sm, 1);
  const int blocks = std::max(1, std::min(sms * per_sm, ceil_div(a.n, kWarps)));
  kern<<<blocks, 32 * kWarps, smem, st>>>(a, acc);
}

template <int ACCUM>
static void launch2(const PairArgs& a, Accumulators& acc, bool energy, bool virial,
                    bool ortho, cudaStream_t st) {
  if (energy && virial)
    launch3<ACCUM, true, true>(a, acc, ortho, st);
  else if (energy)
    launch3<ACCUM, true, false>(a, acc, ortho, st);
  else if (virial)
    launch3<ACCUM, false, true>(a, acc, ortho, st);
  else
    launch3<ACCUM, false, false>(a, acc, ortho, st);
}

int launch_pair(const PairArgs& a, Accumulators& acc, int accum, bool energy,
                bool virial, bool ortho, cudaStream_t st) {
  if (a.n <= 0) return kOk;
  if (accum == kAccumFixed)
    launch2<kAccumFixed>(a, acc, energy, virial, ortho, st);
  else
    launch2<kAccumFloat>(a, acc, energy, virial, ortho, st);
  SNB_CUDA_TRY(cudaGetLastError());
  return kOk;
}

// ---------------------------------------------------------------------------
// Soft-core variant: Lennard_Jones_And_Direct_Coulomb_Soft_Core_CUDA
// (LJ_soft_core.cpp:196-461; pair terms LJ_soft_core.h:33-149).
// A pair whose end states both have LJ (A'_A * A'_B != 0), or neither has
// (A'_A + A'_B == 0), mixes the hard-core forms linearly in lambda; any other
// pair uses the soft-core radius r_sc = (r^6 + alpha lambda^p sigma^6)^(1/6)
// for state A and (r^6 + alpha (1-lambda)^p sigma^6)^(1/6) for state B, with
// sigma^6 = max(A'/(2B'), sigma_min^6), or the input sigma^6 when A' or B' is 0.
// dU/dlambda chain term (Get_Soft_Core_dU_dlambda, LJ_soft_core.h:142-149)
__device__ __forceinline__ float sc_dudl(float F, float sigma, float rsc, float alpha,
                                         float p, float lambda) {
  float rsc2 = rsc * rsc;
  return 0.16666667f * p * alpha * (1.0f - lambda) * powf(lambda + FLT_MIN, p - 1.0f) *
         F / (rsc2 * rsc2) * sigma;
}
__device__ __forceinline__ float coul_e(float qq, float beta, float r) {
  return qq * erfcf(beta * r) / r;
}
__device__ __forceinline__ float coul_f(float qq, float beta, float r) {
  float br = beta * r;
  return qq / (r * r * r) * (br * kTwoOverSqrtPi * expf(-br * br) + erfcf(br));
}

template <int ACCUM, bool ENERGY, bool VIRIAL, bool DUDL>
__global__ void __launch_bounds__(256)
k_lj_soft(SoftArgs a, Accumulators acc, long long* dudl_total) {
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= a.n) return;
  if (a.nl_flags && a.nl_flags[1]) return;  // list overflowed: rows not written
  const float lam = a.lambda, lam_ = 1.0f - a.lambda;
  const float alp_A = a.alpha * powf(lam, a.p);
  const float alp_B = a.alpha * powf(lam_, a.p);
  const float4 pi = a.pos[i];
  const float3 ri = make_float3(pi.x, pi.y, pi.z);
  const int2 pri = a.par[i];
  const int tAi = pri.x & 0xffff, tBi = pri.x >> 16;
  const float dqi = DUDL && a.dq ? a.dq[i] : 0.f;
  const int gi = ENERGY || VIRIAL ? a.global[i] : 0;
  float fx = 0.f, fy = 0.f, fz = 0.f;
  float e_lj = 0.f, e_c = 0.f, e_inter = 0.f, e_intra = 0.f;
  float du_lj = 0.f, du_c = 0.f;
  float vir[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const int k0 = a.row_start[i], k1 = k0 + a.row_count[i];
  for (int k = k0 + lane; k < k1; k += 32) {
    const int j = a.cols[k];
    const float4 pj = a.pos[j];
    const float3 dr = min_image_fast<false>(make_float3(pj.x, pj.y, pj.z), ri, a.cell,
                                            a.rcell);
    const float r2 = dr.x * dr.x + dr.y * dr.y + dr.z * dr.z;
    if (!(r2 < a.cutoff2)) continue;
    const int2 prj = a.par[j];
    const int tAj = prj.x & 0xffff, tBj = prj.x >> 16;
    const int pA = lj_pair_index(tAi, tAj), pB = lj_pair_index(tBi, tBj);
    const float AA = a.AA[pA], AB = a.AB[pA], BA = a.BA[pB], BB = a.BB[pB];
    const float r = sqrtf(r2);
    const float qq = pi.w * pj.w;
    float fs, elj, ec, dl = 0.f, dc = 0.f;
    if (BA * AA != 0.f || BA + AA == 0.f) {
      const float ir2 = 1.0f / r2, ir6 = ir2 * ir2 * ir2;
      fs = lam_ * (AB - AA * ir6) * ir6 * ir2 + lam * (BB - BA * ir6) * ir6 * ir2 -
           coul_f(qq, a.beta, r);
      elj = lam_ * lj_energy(AA, AB, ir6) + lam * lj_energy(BA, BB, ir6);
      ec = coul_e(qq, a.beta, r);
      if (DUDL) {
        dl = lj_energy(BA, BB, ir6) - lj_energy(AA, AB, ir6);
        const float dqj = a.dq ? a.dq[j] : 0.f;
        dc = erfcf(a.beta * r) * (dqj * pi.w + pj.w * dqi) / r;
      }
    } else {
      const float sA = sc_sigma6(AA, AB, a.sigma6, a.sigma6_min);
      const float sB = sc_sigma6(BA, BB, a.sigma6, a.sigma6_min);
      const float r6 = r2 * r2 * r2;
      const float rA = powf(r6 + alp_A * sA, 0.16666667f);
      const float rB = powf(r6 + alp_B * sB, 0.16666667f);
      const float r4 = r2 * r2;
      const float iA2 = 1.0f / (rA * rA), iA6 = iA2 * iA2 * iA2;
      const float iB2 = 1.0f / (rB * rB), iB6 = iB2 * iB2 * iB2;
      const float flA = r4 * (AB - AA * iA6) * iA6 * iA6;
      const float flB = r4 * (BB - BA * iB6) * iB6 * iB6;
      const float bA = a.beta * rA, bB = a.beta * rB;
      const float fcA = qq * r4 *
                        (expf(-bA * bA) * kTwoOverSqrtPi * a.beta + erfcf(bA) / rA) * iA6;
      const float fcB = qq * r4 *
                        (expf(-bB * bB) * kTwoOverSqrtPi * a.beta + erfcf(bB) / rB) * iB6;
      fs = lam_ * flA + lam * flB - (lam_ * fcA + lam * fcB);
      ec = lam_ * coul_e(qq, a.beta, rA) + lam * coul_e(qq, a.beta, rB);
      elj = lam_ * lj_energy(AA, AB, iA6) + lam * lj_energy(BA, BB, iB6);
      if (DUDL) {
        dl = lj_energy(BA, BB, iB6) - lj_energy(AA, AB, iA6);
        dl += sc_dudl((AB - AA * iA6) * iA6 * iA2, sA, rA, a.alpha, a.p, lam) -
              sc_dudl((BB - BA * iB6) * iB6 * iB2, sB, rB, a.alpha, a.p, lam_);
        const float dqj = a.dq ? a.dq[j] : 0.f;
        const float qd = dqj * pi.w + pj.w * dqi;
        dc = coul_e(qq, a.beta, rB) - coul_e(qq, a.beta, rA);
        dc += sc_dudl(coul_f(qq, a.beta, rB), sB, rB, a.alpha, a.p, lam_) -
              sc_dudl(coul_f(qq, a.beta, rA), sA, rA, a.alpha, a.p, lam);
        dc += lam * erfcf(a.beta * rB) * qd / rB + lam_ * erfcf(a.beta * rA) * qd / rA;
      }
    }
    const float gx = fs * dr.x, gy = fs * dr.y, gz = fs * dr.z;
    if (!DUDL) {
      fx += gx;
      fy += gy;
      fz += gz;
      add_force<ACCUM>(acc, j, -gx, -gy, -gz);
    }
    if (DUDL) {
      du_lj += dl;
      du_c += dc;
    }
    if (ENERGY || VIRIAL) {
      const bool own_i = gi < a.global[j];
      const bool intra = pri.y == prj.y;
      if (ENERGY) {
        if (own_i) {
          e_lj += elj;
          e_c += ec;
          if (intra) e_intra += elj; else e_inter += elj;
        } else {
          add_energy<ACCUM>(acc, j, elj + ec, elj, ec);
          const int N = acc.n;
          if (ACCUM == kAccumFixed)
            red_add(acc.d_eaux + (intra ? N : 0) + j, to_fixed_energy(elj));
          else
            atomicAdd(acc.d_feaux + (intra ? N : 0) + j, elj);
        }
      }
      if (VIRIAL) {
        float v[6];
        v[0] = -(gx * dr.x);
        v[1] = -(gx * dr.y + gy * dr.x);
        v[2] = -(gy * dr.y);
        v[3] = -(gx * dr.z + gz * dr.x);
        v[4] = -(gy * dr.z + gz * dr.y);
        v[5] = -(gz * dr.z);
        if (own_i) {
#pragma unroll
          for (int c = 0; c < 6; ++c) vir[c] += v[c];
        } else {
          add_virial<ACCUM>(acc, j, v);
        }
      }
    }
  }
  if (DUDL) {
    du_lj = warp_sum(du_lj);
    du_c = warp_sum(du_c);
    if (lane == 0) {
      red_add(dudl_total, to_fixed_energy(du_lj));
      red_add(dudl_total + 1, to_fixed_energy(du_c));
    }
    return;
  }
  fx = warp_sum(fx);
  fy = warp_sum(fy);
  fz = warp_sum(fz);
  if (ENERGY) {
    e_lj = warp_sum(e_lj);
    e_c = warp_sum(e_c);
    e_inter = warp_sum(e_inter);
    e_intra = warp_sum(e_intra);
  }
  if (VIRIAL) {
#pragma unroll
    for (int c = 0; c < 6; ++c) vir[c] = warp_sum(vir[c]);
  }
  if (lane == 0) {
    add_force<ACCUM>(acc, i, fx, fy, fz);
    if (ENERGY) {
      add_energy<ACCUM>(acc, i, e_lj + e_c, e_lj, e_c);
      const int N = acc.n;
      if (ACCUM == kAccumFixed) {
        red_add(acc.d_eaux + i, to_fixed_energy(e_inter));
        red_add(acc.d_eaux + N + i, to_fixed_energy(e_intra));
      } else {
        atomicAdd(acc.d_feaux + i, e_inter);
        atomicAdd(acc.d_feaux + N + i, e_intra);
      }
    }
    if (VIRIAL) add_virial<ACCUM>(acc, i, vir);
  }
}

template <int ACCUM>
static void launch_soft2(const SoftArgs& a, Accumulators& acc, bool energy, bool virial,
                         bool dudl, long long* dt, cudaStream_t st) {
  dim3 grid(ceil_div(a.n, 8)), block(256);
  if (dudl)
    k_lj_soft<ACCUM, false, false, true><<<grid, block, 0, st>>>(a, acc, dt);
  else if (energy && virial)
    k_lj_soft<ACCUM, true, true, false><<<grid, block, 0, st>>>(a, acc, dt);
  else if (energy)
    k_lj_soft<ACCUM, true, false, false><<<grid, block, 0, st>>>(a, acc, dt);
  else if (virial)
    k_lj_soft<ACCUM, false, true, false><<<grid, block, 0, st>>>(a, acc, dt);
  else
    k_lj_soft<ACCUM, false, false, false><<<grid, block, 0, st>>>(a, acc, dt);
}

int launch_soft(const SoftArgs& a, Accumulators& acc, int accum, bool energy,
                bool virial, bool dudl, long long* dudl_total, cudaStream_t st) {
  if (a.n <= 0) return kOk;
  if (accum == kAccumFixed)
    launch_soft2<kAccumFixed>(a, acc, energy, virial, dudl, dudl_total, st);
  else
    launch_soft2<kAccumFloat>(a, acc, energy, virial, dudl, dudl_total, st);
  SNB_CUDA_TRY(cudaGetLastError());
  return kOk;
}

}  // namespace snb
