// od_n3.cu — all-pairs ion–ion sums with each unordered pair evaluated once (variant 7).
//
// The screened pair term is antisymmetric: for dx = x_i - x_j the contribution to ion i is
// c(r)·dx and the contribution to ion j is -c(r)·dx, with the same FP32 bits (IEEE subtraction
// is exactly antisymmetric and r^2 depends on dx^2 only). Evaluating every unordered pair once
// and applying both contributions halves the SFU and FP32 work of the directed-pair kernels
// (the reference's OpenMM CUDA nonbonded kernel also applies each pair force to both atoms).
//
// Decomposition
//   * A group pair is GT = 32·MT target ions (lane l holds ions l + 32k, k < MT, each duplicated in
//     both halves of an f32x2 register) against GS = 32·MS source ions (MS/2 packs per lane). The
//     sources rotate around the warp: at each of 32 lane steps every lane evaluates its targets
//     against the sources it holds, then passes the sources, their positions and their FP32
//     reaction sums, to the previous lane.
//   * The group pairs of the upper triangle are numbered row by row (a row: one target group
//     against the source groups from its own on), and every warp takes L consecutive ones, or,
//     in systems too small to fill the GPU that way, one group pair's lane steps in `split`
//     equal parts. Warps share nothing: there is no block barrier, and a block's warps differ by
//     at most one group pair of work.
//   * The source groups inside a target group are evaluated as directed pairs (no reaction; the
//     self pair contributes exactly 0).
//   * Reactions are summed in FP32 over at most 16 lane steps, target sums over one group pair or
//     part of one (then as two-floats in the warp's shared-memory slice when L > 1); both are added to
//     the ions' 64-bit fixed-point accumulators with integer atomics, so every result bit is
//     independent of scheduling.
//
// What bounds it: operand fetch of the packed FP32 pipe. Measured on GB300, cycles per warp
// instruction and sub-partition: fma.f32x2 with one, two and three distinct register operands
// 2.1, 2.7 to 3.0 and 3.0 to 3.7; rsqrt, sqrt and rcp 8.4, ex2 4.2, shfl 4.2. At 2^18 ions the kernel
// takes 25.3 cycles per 32 unordered pairs and sub-partition (8 x 2; 4 x 4: 26.2), and 23 with every
// SFU operation taken out, so fewer SFU operations, or a scalar form (33), gain nothing. The pair
// term below has the fewest packed operations (17 with the sums).
#include <algorithm>
#include "od_internal.h"

namespace {

constexpr int kSliceWarps = 4;  // warps per block: they are independent, small blocks retire evenly

// Register budget and unrolling per shape (MT targets, MS sources per lane). 2^18 ions, ms per
// evaluation: 8 x 2 21.6 (16 warps per SM of 128 registers, two lane steps unrolled), 4 x 4 22.4 (20
// warps of 96, four steps; with 24 warps of 80 or 16 of 128 registers 2 to 4 % slower), 2 x 2 24.4.
// The tile-pair form this replaces (eight warps per tile pair, one barrier per source group) took
// 23.3 (8 x 2) there, 0.928 against 0.838 now at 50021 ions (4 x 4), and 0.129 (2 x 2, its last wave
// half empty) against 0.100 at 2^14. The registers hold the loop state only just: the split and the
// slice length are template parameters because as variables they spilled (16384 ions 0.115 ms).
template <int MT, int MS>
struct slice_traits {
  static constexpr int GT = 32 * MT, GS = 32 * MS;
  static constexpr int R = GT / GS;  // source groups inside a target group
  static constexpr int MIN_BLOCKS = MT == 8 ? 4 : (MT == 4 ? 5 : 8);
  static constexpr int UNROLL = MT == 8 ? 2 : 4;
};

struct pair_consts {
  od_u64 eps, rho, nl2e;
};

// One pack: target (X, X) against two sources.
template <bool REACT>
__device__ __forceinline__ void pair_once(const pair_consts& k, od_u64 X, od_u64 Y, od_u64 Z,
                                          od_u64 QX, od_u64 QY, od_u64 QZ, od_u64& AX, od_u64& AY,
                                          od_u64& AZ, od_u64& RX, od_u64& RY, od_u64& RZ) {
  const od_u64 DX = sub2(X, QX), DY = sub2(Y, QY), DZ = sub2(Z, QZ);
  od_u64 R2 = fma2(DX, DX, k.eps);
  R2 = fma2(DY, DY, R2);
  R2 = fma2(DZ, DZ, R2);
  const od_u64 C = od_pair_c2(R2, k.rho, k.nl2e);
  AX = fma2(C, DX, AX); AY = fma2(C, DY, AY); AZ = fma2(C, DZ, AZ);
  if (REACT) { RX = fma2(C, DX, RX); RY = fma2(C, DY, RY); RZ = fma2(C, DZ, RZ); }
}

// STEPS lane steps of one group pair
template <int MT, int MS, bool REACT, int STEPS>
__device__ __forceinline__ void lane_steps(const pair_consts& k, const od_u64 (&X)[MT],
                                           const od_u64 (&Y)[MT], const od_u64 (&Z)[MT],
                                           od_u64 (&QX)[MS / 2], od_u64 (&QY)[MS / 2],
                                           od_u64 (&QZ)[MS / 2], od_u64 (&AX)[MT],
                                           od_u64 (&AY)[MT], od_u64 (&AZ)[MT],
                                           od_u64 (&RX)[MS / 2], od_u64 (&RY)[MS / 2],
                                           od_u64 (&RZ)[MS / 2], int src) {
  constexpr int U = slice_traits<MT, MS>::UNROLL;
#pragma unroll U
  for (int st = 0; st < STEPS; st++) {
#pragma unroll
    for (int q = 0; q < MS / 2; q++) {
#pragma unroll
      for (int t = 0; t < MT; t++)
        pair_once<REACT>(k, X[t], Y[t], Z[t], QX[q], QY[q], QZ[q], AX[t], AY[t], AZ[t], RX[q],
                         RY[q], RZ[q]);
      QX[q] = shfl64(QX[q], src); QY[q] = shfl64(QY[q], src); QZ[q] = shfl64(QZ[q], src);
      if (REACT) {
        RX[q] = shfl64(RX[q], src); RY[q] = shfl64(RY[q], src); RZ[q] = shfl64(RZ[q], src);
      }
    }
  }
}

// Unit `unit` of one simulation (one warp): group pairs [unit L, unit L + L) of the row-major
// upper triangle, or (SPLIT > 1, L = 1) part unit % SPLIT of group pair unit / SPLIT.
// h: this lane's column of the warp's shared-memory slice ([6][GT] floats, used when FOLD).
// HALF: the target sums too are added to the accumulators every 16 lane steps.
template <int MT, int MS, int SPLIT, bool FOLD, bool HALF>
__device__ __forceinline__ void n3_slice(const float* __restrict__ sx, const float* __restrict__ sy,
                                         const float* __restrict__ sz, int Npad,
                                         unsigned long long* __restrict__ acc, float rho0,
                                         long long unit, const od_n3_split& sp, float* h) {
  using TR = slice_traits<MT, MS>;
  constexpr int GT = TR::GT, GS = TR::GS, R = TR::R;
  static_assert(!(FOLD && SPLIT > 1), "a split group pair is one unit");
  static_assert(!HALF || (SPLIT == 1 && !FOLD), "halves of a whole group pair");
  const int lane = threadIdx.x & 31, src = (lane + 1) & 31;
  constexpr int STEPS = 32 / SPLIT;        // lane steps of a unit's group pairs
  constexpr int PART = STEPS < 16 ? STEPS : 16;  // lane steps between two reaction flushes
  if (unit >= sp.units) return;
  int g, s, n;  // target group, source group, group pairs left
  int at;       // lane whose sources this lane holds
  {
    const long long f = SPLIT > 1 ? unit / SPLIT : (FOLD ? unit * sp.L : unit);
    at = SPLIT > 1 ? lane + (int)(unit % SPLIT) * STEPS : lane;
    n = FOLD ? (int)min((long long)sp.L, sp.pairs - f) : 1;
    // rows 0 .. g-1 hold g NS - R g (g - 1) / 2 group pairs
    const int NS = Npad / GS;
    const double b = NS + 0.5 * R;
    g = (int)((b - sqrt(fmax(b * b - 2.0 * R * (double)f, 0.0))) / R);
    auto before = [&](long long q) { return q * NS - R * (q * (q - 1) / 2); };
    while (g > 0 && before(g) > f) g--;
    while (before(g + 1) <= f) g++;
    s = g * R + (int)(f - before(g));
  }
  pair_consts k;
  k.eps = p2(1e-30f, 1e-30f); k.rho = p2(rho0, rho0); k.nl2e = p2(OD_NLOG2E, OD_NLOG2E);
  od_pdl_wait();  // the unit is found while the kernel that writes the positions still runs
  for (;;) {
    od_u64 X[MT], Y[MT], Z[MT];
#pragma unroll
    for (int t = 0; t < MT; t++) {
      const int i = g * GT + lane + 32 * t;
      X[t] = p2(sx[i], sx[i]); Y[t] = p2(sy[i], sy[i]); Z[t] = p2(sz[i], sz[i]);
      if (FOLD)
#pragma unroll
        for (int c = 0; c < 6; c++) h[c * GT + 32 * t] = 0.f;
    }
    do {
      od_u64 QX[MS / 2], QY[MS / 2], QZ[MS / 2], RX[MS / 2], RY[MS / 2], RZ[MS / 2];
      od_u64 AX[MT], AY[MT], AZ[MT];
#pragma unroll
      for (int q = 0; q < MS / 2; q++) {
        const int j = s * GS + (at & 31) + 64 * q;
        QX[q] = p2(sx[j], sx[j + 32]); QY[q] = p2(sy[j], sy[j + 32]); QZ[q] = p2(sz[j], sz[j + 32]);
      }
#pragma unroll
      for (int t = 0; t < MT; t++) AX[t] = AY[t] = AZ[t] = 0ull;
      const auto add_targets = [&] {
#pragma unroll
        for (int t = 0; t < MT; t++) {
          unsigned long long* a = acc + g * GT + lane + 32 * t;
          od_fix_add1(a, sum2(AX[t]));
          od_fix_add1(a + Npad, sum2(AY[t]));
          od_fix_add1(a + 2 * (size_t)Npad, sum2(AZ[t]));
          AX[t] = AY[t] = AZ[t] = 0ull;
        }
      };
      if (s >= g * R + R) {
        // each part's reactions are added to the accumulators of the sources where they stand
        // (the force on a source is minus the accumulated terms)
#pragma unroll 1
        for (int st = PART; st <= STEPS; st += PART) {
#pragma unroll
          for (int q = 0; q < MS / 2; q++) RX[q] = RY[q] = RZ[q] = 0ull;
          lane_steps<MT, MS, true, PART>(k, X, Y, Z, QX, QY, QZ, AX, AY, AZ, RX, RY, RZ, src);
#pragma unroll
          for (int q = 0; q < MS / 2; q++) {
            const float2 rx = up2(RX[q]), ry = up2(RY[q]), rz = up2(RZ[q]);
            unsigned long long* e = acc + s * GS + ((at + st) & 31) + 64 * q;
            od_fix_add1(e, -rx.x); od_fix_add1(e + 32, -rx.y);
            e += Npad;
            od_fix_add1(e, -ry.x); od_fix_add1(e + 32, -ry.y);
            e += Npad;
            od_fix_add1(e, -rz.x); od_fix_add1(e + 32, -rz.y);
          }
          if (HALF) add_targets();
        }
      } else if (HALF) {
#pragma unroll 1
        for (int st = PART; st <= STEPS; st += PART) {
          lane_steps<MT, MS, false, PART>(k, X, Y, Z, QX, QY, QZ, AX, AY, AZ, RX, RY, RZ, src);
          add_targets();
        }
      } else {
        lane_steps<MT, MS, false, STEPS>(k, X, Y, Z, QX, QY, QZ, AX, AY, AZ, RX, RY, RZ, src);
      }
      if (!FOLD) {
        if (!HALF) add_targets();
        return;
      }
#pragma unroll
      for (int t = 0; t < MT; t++) {
        od_acc2(h[32 * t], h[3 * GT + 32 * t], sum2(AX[t]));
        od_acc2(h[GT + 32 * t], h[4 * GT + 32 * t], sum2(AY[t]));
        od_acc2(h[2 * GT + 32 * t], h[5 * GT + 32 * t], sum2(AZ[t]));
      }
      n--;
      s++;
    } while (n > 0 && s * GS < Npad);
#pragma unroll
    for (int t = 0; t < MT; t++)
#pragma unroll
      for (int c = 0; c < 3; c++)
        od_fix_add(acc + (size_t)c * Npad + g * GT + lane + 32 * t, h[c * GT + 32 * t],
                   h[(3 + c) * GT + 32 * t]);
    if (n <= 0) return;
    g++;
    s = g * R;
  }
}

template <int MT, int MS, int SPLIT, bool FOLD, bool HALF>
__global__ void __launch_bounds__(kSliceWarps * 32, (slice_traits<MT, MS>::MIN_BLOCKS))
    k_pairs_n3(const float* __restrict__ sx, const float* __restrict__ sy,
               const float* __restrict__ sz, int Npad, unsigned long long* __restrict__ acc,
               float rho0, const __grid_constant__ od_n3_split sp) {
  __shared__ float sm[FOLD ? kSliceWarps * 6 * slice_traits<MT, MS>::GT : 1];
  const int w = threadIdx.x >> 5;
  od_pdl_trigger();
  n3_slice<MT, MS, SPLIT, FOLD, HALF>(sx, sy, sz, Npad, acc, rho0,
                                      (long long)blockIdx.x * kSliceWarps + w, sp,
                                      sm + (FOLD ? w * 6 * slice_traits<MT, MS>::GT +
                                                       (threadIdx.x & 31)
                                                 : 0));
}

// Batched form: block k takes block items[k].y of member items[k].x; the table lists every block of
// every member using this form.
template <int MT, int MS, int SPLIT, bool FOLD, bool HALF>
__global__ void __launch_bounds__(kSliceWarps * 32, (slice_traits<MT, MS>::MIN_BLOCKS))
    k_b_pairs_n3(const od_simdesc* __restrict__ sims, const int2* __restrict__ items) {
  __shared__ float sm[FOLD ? kSliceWarps * 6 * slice_traits<MT, MS>::GT : 1];
  od_pdl_trigger();
  const int2 it = items[blockIdx.x];
  const od_simdesc& d = sims[it.x];
  if (!od_evaluates(d.dp->force_every, d.ds->step)) {  // force interval: no evaluation
    od_pdl_wait();  // the next kernel may start when this grid is done: it needs the one before too
    return;
  }
  const int w = threadIdx.x >> 5;
  n3_slice<MT, MS, SPLIT, FOLD, HALF>(d.b.sx, d.b.sy, d.b.sz, d.Npad, d.b.n3, d.rho0,
                                      (long long)it.y * kSliceWarps + w, d.n3,
                                      sm + (FOLD ? w * 6 * slice_traits<MT, MS>::GT +
                                                       (threadIdx.x & 31)
                                                 : 0));
}

// Accumulators -> slab 0 of (ph, pl) as two-float sums, and cleared for the next evaluation.
__global__ void k_n3_take(unsigned long long* __restrict__ acc, int Npad, float4* __restrict__ ph,
                          float4* __restrict__ pl) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Npad) return;
  float3 hi, lo;
  od_fix_take(acc + i, (size_t)Npad, hi, lo);
  ph[i] = make_float4(hi.x, hi.y, hi.z, 0.f);
  pl[i] = make_float4(lo.x, lo.y, lo.z, 0.f);
}

template <int MT, int MS, int SPLIT, bool FOLD, bool HALF = false>
cudaError_t launch_n3(const od_pair_io& io, int Npad, float rho0, const od_n3_split& sp,
                      cudaStream_t s) {
  return od_launch_pdl(k_pairs_n3<MT, MS, SPLIT, FOLD, HALF>, dim3((unsigned)od_n3_blocks(sp)),
                       dim3(kSliceWarps * 32), s, io.sx, io.sy, io.sz, Npad, io.n3, rho0, sp);
}

}  // namespace

bool od_n3_supported(int ipt, int tile) {
  switch (ipt * 10000 + tile) {
    case 20512: case 21024: case 22048: case 24096: case 41024: case 42048: case 44096:
    case 82048: case 84096:
      return true;
  }
  return false;
}

long long od_n3_blocks(const od_n3_split& sp) { return (sp.units + kSliceWarps - 1) / kSliceWarps; }

// Work split of (ipt targets per lane, tile) for Npad ions, the same on every GPU so that results
// do not depend on the device.
//   * 4 x 4: one group pair (128 x 128 ions, 512 pair terms per lane) per warp. 50021 ions 0.838 ms,
//     against 0.848 and 0.859 with 4 and 8 per warp (a longer last wave; the flush of the target
//     sums that longer slices save is small). In small systems the group pairs leave warp slots
//     empty (3040 on 152 SMs; 4656 group pairs at 12000) and a single warp's dependency chain sets
//     the time, so they are split by lane steps. Steps of 2048, 4096, 5000, 7680, 8192 and 14000
//     ions in us: whole 29.0, 31.1, 52.4, 54.7, 55.3, 94.5; two parts 24.4, 28.9, 37.5, 44.7, 44.4,
//     90.7; four 22.8, 27.0, 30.1, 42.6, 46.0, 97.5. Two parts still gain 1.5 % at 2^14, but there
//     batches would run them apart from their larger members, with a last wave of their own.
//     Tiles of 2048 and 4096 ions: the target sums of whole group pairs are added after each half, so
//     that the FP32 chains have 32 terms instead of 64: median relative error per ion at 16385, 20011 and 32768
//     ions 5.5e-8, 5.2e-8, 4.7e-8 against 6.0e-8, 5.7e-8, 5.1e-8. No slower for a single simulation (325
//     us per step at 30000 ions), 2.5 % in batches.
//   * 8 x 2 (256 x 64 ions) and 2 x 2: a tile names how many group pairs a slice may hold (tile / 64),
//     at least 16 slices per resident warp. 8 x 2 at 2^18 ions: 21.6 ms with 8 or 16, 22.3 with 1.
od_n3_split od_n3_split_of(int Npad, int ipt, int tile) {
  const long long GT = 32 * ipt, GS = ipt == 8 ? 64 : GT, R = GT / GS, NG = Npad / GT, NS = Npad / GS;
  od_n3_split sp{};
  sp.pairs = NG * NS - R * (NG * (NG - 1) / 2);
  sp.split = 1;
  long long L = 1;
  if (ipt == 4) {
    if (Npad < 16384) sp.split = Npad <= 7680 ? 4 : 2;
  } else {
    const long long warps = 152ll * kSliceWarps * (ipt == 8 ? 4 : 8);
    L = std::max(1ll, std::min<long long>(tile / 64, sp.pairs / (warps * 16)));
  }
  while (sp.pairs / L / kSliceWarps >= 0x7fffffff) L *= 2;  // the grid holds 2^31 - 1 blocks
  sp.L = (int)L;
  sp.half = ipt == 4 && tile > 1024 && sp.split == 1 && L == 1;
  sp.units = sp.split > 1 ? sp.pairs * sp.split : (sp.pairs + L - 1) / L;
  return sp;
}

cudaError_t od_launch_pairs_n3(const od_pair_plan& pl, const od_pair_io& io, int Npad, float4* ph,
                               float4* plo, float rho0, cudaStream_t s, bool take) {
  if (!io.n3 || !od_n3_supported(pl.ipt, pl.tile)) return cudaErrorInvalidValue;
  const od_n3_split sp = od_n3_split_of(Npad, pl.ipt, pl.tile);
  cudaError_t e;
  if (pl.ipt == 2) e = launch_n3<2, 2, 1, true>(io, Npad, rho0, sp, s);
  else if (pl.ipt == 8) e = launch_n3<8, 2, 1, true>(io, Npad, rho0, sp, s);
  else if (sp.split == 4) e = launch_n3<4, 4, 4, false>(io, Npad, rho0, sp, s);
  else if (sp.split == 2) e = launch_n3<4, 4, 2, false>(io, Npad, rho0, sp, s);
  else if (sp.L > 1) e = launch_n3<4, 4, 1, true>(io, Npad, rho0, sp, s);
  else if (sp.half) e = launch_n3<4, 4, 1, false, true>(io, Npad, rho0, sp, s);
  else e = launch_n3<4, 4, 1, false>(io, Npad, rho0, sp, s);
  if (e != cudaSuccess) return e;
  if (take) k_n3_take<<<(Npad + 255) / 256, 256, 0, s>>>(io.n3, Npad, ph, plo);
  return cudaGetLastError();
}

int od_n3_default(int Npad, size_t budget_bytes, int* ipt) {
  // as a batch member: 4 x 4 up to 2^16 ions, 8 x 2 above: 100000 ions 3.33 and 3.22 ms, 50021 ions 0.838
  // and 0.824 ms, 16384 ions 0.100 and 0.102 ms (the accumulators fit any budget that holds the
  // ions: 24 bytes per ion). From 2^14 to 2^15 ions with halves, as accurate as the 2 x 2 shape
  // that was the default there (5.8e-8, 5.6e-8 and 5.0e-8 at 16385, 20011 and 32768 ions).
  const int tile = od_n3_batch_plan(Npad, budget_bytes, ipt);
  return tile == 1024 && Npad >= 16384 && Npad <= 32768 ? 2048 : tile;
}

size_t od_n3_floats(int Npad, int T) {
  // three 64-bit fixed-point accumulators per ion, whatever the tile
  if (T <= 0) return 0;
  return 6 * (size_t)Npad;
}

int od_n3_form(int ipt, const od_n3_split& sp) {
  if (ipt == 8) return 3;
  if (ipt == 2) return 5;
  if (sp.half) return 6;
  return sp.split == 4 ? 2 : (sp.split == 2 ? 1 : (sp.L > 1 ? 4 : 0));
}

cudaError_t od_launch_batch_pairs_n3(const od_batchview& v, unsigned pairs, cudaStream_t s) {
  // the forms batch members use: those of od_n3_batch_plan, and 2 x 2 and halves, which a member's own
  // handle may be given (od_set_pair_plan)
  cudaError_t e = cudaSuccess;
#define OD_B_N3(f, MT, MS, SPLIT, FOLD, HALF)                                                \
  if (v.n3_nitems[f] > 0 && (pairs >> f & 1) && e == cudaSuccess)                            \
  e = od_launch_pdl(k_b_pairs_n3<MT, MS, SPLIT, FOLD, HALF>, dim3(v.n3_nitems[f]),           \
                    dim3(kSliceWarps * 32), s, v.sims, (const int2*)v.n3_items[f])
  OD_B_N3(3, 8, 2, 1, true, false);
  OD_B_N3(0, 4, 4, 1, false, false);
  OD_B_N3(6, 4, 4, 1, false, true);
  OD_B_N3(1, 4, 4, 2, false, false);
  OD_B_N3(2, 4, 4, 4, false, false);
  OD_B_N3(4, 4, 4, 1, true, false);
  OD_B_N3(5, 2, 2, 1, true, false);
#undef OD_B_N3
  return e != cudaSuccess ? e : cudaGetLastError();
}

int od_n3_batch_plan(int Npad, size_t budget_bytes, int* ipt) {
  // batch members: 4 x 4 ions per lane up to 2^16 ions, 8 x 2 above; 0 when the accumulators do not
  // fit (the member then takes the directed-pair kernel)
  const int T = Npad <= (1 << 16) ? 1024 : 2048;
  if (sizeof(float) * od_n3_floats(Npad, T) > budget_bytes) return 0;
  *ipt = T == 1024 ? 4 : 8;
  return T;
}
