// od_cutn3.cu — ion–ion forces within a cutoff (cutoff variant 3): ions sorted along a Hilbert curve
// of a cell grid, blocks of 32 consecutive sorted ions with their bounding boxes, each unordered
// pair inside the cutoff evaluated once, and the sums added as 64-bit fixed point with integer
// atomics to per-slot accumulators. Every result bit is independent of scheduling.
//
// A warp works alone: it takes a source group of 64 slots (two blocks) and a run of 512-slot tiles
// at or above it, lists the target blocks of those tiles whose boxes come within the cutoff
// (tile boxes first, then block boxes, one lane per box and a ballot), and evaluates them four
// blocks at a time: 4 targets and 2 sources per lane, the sources rotating around the warp as in
// the all-pairs kernel (od_n3.cu). Blocks wholly inside the switching radius (hard cutoff: the
// cutoff) take the plain screened term, the others the switched one.
//
// What bounds it: as the all-pairs kernel, operand fetch of the packed FP32 pipe (17 packed
// operations per pair of pairs for the plain term, 27 with switching), plus the pairs of the
// listed blocks that lie beyond the cutoff. field_chain (2^19 ions, 2 lambda): 1.63 pairs
// listed per pair inside (1.35 evaluated), 21.9 ms per evaluation. The tile-pair form this replaces (512-ion
// tile pairs, 64 x 64 group lists built by one warp between two block barriers, 2 x 2 ions per
// lane, sums in shared memory with compare-and-swap atomics) took 32.2 ms there; 65536 ions in
// the 12 lambda tall cylinder at 3.2 lambda 1.28 -> 0.70 ms, 20011 ions at 2 lambda 0.197 -> 0.077 ms.
#include "od_hilbert.h"
#include "od_internal.h"
#include <algorithm>
#include <cmath>

namespace {

// Cell grid of G^3 cells over the cube [lo, lo + G/inv_s)^3; a cell's key is its index along
// a Hilbert curve (od_hilbert.h), so that the ions sorted by key fill tiles and 64-ion groups
// with compact bounding boxes: at 2^19 ions in the 3 x 6 lambda cylinder the boxes of 64-ion
// groups keep 1.73x the pairs inside a 2 lambda cutoff, against 1.94x in Morton order.
//
// Cubes of G^3 cells stacked nb deep along z (nb = 1 for a compact domain); a cell's key is its
// cube's index times G^3 plus its index along the cube's Hilbert curve. The counts are zero between
// evaluations (k_mc_sort clears them); an ion's rank is the count that it found.
__global__ void k_mc_count(int n, const float4* __restrict__ pos, float lo, float lo_z,
                           float inv_s, int G, int nb, int32_t* __restrict__ cell_of,
                           int32_t* __restrict__ rank_of, int32_t* __restrict__ count,
                           unsigned long long* __restrict__ next) {
  od_pdl_wait();
  od_pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *next = 0ull;  // the pair kernel's work counter
  if (i >= n) return;
  const float4 p = pos[i];
  const int bits = 31 - __clz(G);
  const int cx = min(max((int)floorf((p.x - lo) * inv_s), 0), G - 1);
  const int cy = min(max((int)floorf((p.y - lo) * inv_s), 0), G - 1);
  const int cz = min(max((int)floorf((p.z - lo_z) * inv_s), 0), nb * G - 1);
  const int c = ((cz >> bits) << (3 * bits)) +
                (int)od_hilbert3((uint32_t)cx, (uint32_t)cy, (uint32_t)(cz & (G - 1)), bits);
  cell_of[i] = c;
  rank_of[i] = atomicAdd(&count[c], 1);
}

// exclusive scan over the block's 1024 threads
__device__ __forceinline__ int block_scan_1024(int a) {
  __shared__ int s_w[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int ia = a;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, ia, o);
    if (lane >= o) ia += y;
  }
  if (lane == 31) s_w[wid] = ia;
  __syncthreads();
  if (wid == 0) {
    const int v = s_w[lane];
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    s_w[lane] = x - v;
  }
  __syncthreads();
  return s_w[wid] + ia - a;
}

// exclusive scan of in[0..n) into out[0..n], out[n] = total (one 1024-thread block)
__global__ void __launch_bounds__(1024) k_scan_excl(int n, const int32_t* in, int32_t* out) {
  od_pdl_wait();
  od_pdl_trigger();
  const int tid = threadIdx.x, per = (n + 1023) / 1024;
  const int c0 = min(tid * per, n), c1 = min(c0 + per, n);
  int a = 0;
  for (int c = c0; c < c1; c++) a += in[c];
  int off = block_scan_1024(a);
  for (int c = c0; c < c1; c++) {
    const int v = in[c];
    out[c] = off;
    off += v;
  }
  if (tid == 1023) out[n] = off;
}

// The same in two kernels where n is a multiple of 4096 (262144 cells at 2^19 ions: 7.6 us, one
// block 119): blocks of 4096 entries with their totals, then the totals before each block added.
constexpr int kScanBlock = 4096;
__global__ void __launch_bounds__(1024) k_scan_blocks(const int32_t* in, int32_t* out,
                                                      int32_t* __restrict__ totals) {
  od_pdl_wait();
  od_pdl_trigger();
  const int c = blockIdx.x * kScanBlock + 4 * threadIdx.x;
  const int4 v = *reinterpret_cast<const int4*>(in + c);
  const int sum = (v.x + v.y) + (v.z + v.w), off = block_scan_1024(sum);
  *reinterpret_cast<int4*>(out + c) = make_int4(off, off + v.x, off + v.x + v.y, off + v.x + v.y + v.z);
  if (threadIdx.x == 1023) totals[blockIdx.x] = off + sum;
}
__global__ void __launch_bounds__(1024) k_scan_add(int n, const int32_t* totals, int32_t* out) {
  __shared__ int s_before, s_all;
  od_pdl_wait();
  od_pdl_trigger();
  if (threadIdx.x == 0) s_before = s_all = 0;
  __syncthreads();
  int before = 0, all = 0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += 1024) {
    const int v = totals[b];
    all += v;
    if (b < (int)blockIdx.x) before += v;
  }
  before = __reduce_add_sync(0xffffffffu, before);
  all = __reduce_add_sync(0xffffffffu, all);
  if ((threadIdx.x & 31) == 0) { atomicAdd(&s_before, before); atomicAdd(&s_all, all); }
  __syncthreads();
  int4* const o = reinterpret_cast<int4*>(out + blockIdx.x * kScanBlock) + threadIdx.x;
  int4 v = *o;
  v.x += s_before; v.y += s_before; v.z += s_before; v.w += s_before;
  *o = v;
  if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = s_all;
}

__global__ void k_mc_scatter(int n, const int32_t* __restrict__ cell_of,
                             const int32_t* __restrict__ rank_of,
                             const int32_t* __restrict__ start,
                             int32_t* __restrict__ unsorted) {
  od_pdl_wait();
  od_pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsorted[start[cell_of[i]] + rank_of[i]] = i;
}

// The same with the scan: up to kScanCells cells every block scans the counts for itself (16 KB at 4096
// cells, from L2), which takes less than the launch of a scan of its own (20011 ions: 4.8 + 2.5 us ->
// 4.1, the ranks of k_mc_count instead of a second round of atomics included). A multiple of 512 cells.
constexpr int kScanCells = 8192;
__global__ void __launch_bounds__(256) k_mc_scan_scatter(int n, int ncells,
                                                         const int32_t* __restrict__ cell_of,
                                                         const int32_t* __restrict__ rank_of,
                                                         const int32_t* count,
                                                         int32_t* __restrict__ start,
                                                         int32_t* __restrict__ unsorted) {
  extern __shared__ int32_t s_start[];  // cell c at c + c / 16, so that a thread's run has no conflicts
  __shared__ int s_w[8];
  od_pdl_wait();
  od_pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, per = ncells / 256, c0 = tid * per;
  int sum = 0;
  for (int c = 0; c < per; c += 2) {
    const int2 v = *reinterpret_cast<const int2*>(count + c0 + c);
    s_start[c0 + c + ((c0 + c) >> 4)] = v.x;
    s_start[c0 + c + 1 + ((c0 + c + 1) >> 4)] = v.y;
    sum += v.x + v.y;
  }
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_w[w] = incl;
  __syncthreads();
  int off = incl - sum;
  for (int k = 0; k < w; k++) off += s_w[k];
  for (int c = c0; c < c0 + per; c++) {
    const int v = s_start[c + (c >> 4)];
    s_start[c + (c >> 4)] = off;
    off += v;
  }
  __syncthreads();
  if (blockIdx.x == 0) {
    for (int c = tid; c < ncells; c += 256) start[c] = s_start[c + (c >> 4)];
    if (tid == 0) start[ncells] = n;
  }
  const int i = blockIdx.x * 256 + tid;
  if (i >= n) return;
  const int c = cell_of[i];
  unsorted[s_start[c + (c >> 4)] + rank_of[i]] = i;
}

// Sorts every cell's ions by index (the order of the atomic ranks is not reproducible, the sorted
// order is) and writes their positions; the counts are cleared for the next evaluation. A
// thread takes an unsorted slot and counts the smaller indices in its cell: neighbouring threads read
// the same few entries, and the work does not depend on the number of cells (20011 ions 6.0 -> 3.5 us
// against a block per cell with a bitonic sort).
constexpr int kCellMax = 2048;
__global__ void __launch_bounds__(256) k_mc_sort(int n, const int32_t* __restrict__ cell_of,
                                                 const int32_t* __restrict__ start,
                                                 const int32_t* __restrict__ unsorted,
                                                 const float4* __restrict__ pos, int32_t* count,
                                                 int32_t* __restrict__ perm,
                                                 float* __restrict__ xs, float* __restrict__ ys,
                                                 float* __restrict__ zs, uint32_t* __restrict__ err) {
  od_pdl_wait();
  od_pdl_trigger();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int i = unsorted[s], c = cell_of[i], s0 = start[c], n0 = start[c + 1] - s0;
  const float4 p = pos[i];
  int slot = s0;
  if (n0 <= kCellMax) {
#pragma unroll 4
    for (int k = 0; k < n0; k++) slot += unsorted[s0 + k] < i;
  } else {  // left unsorted, with an error
    slot = s;
    if (s == s0) atomicOr(err, OD_DERR_CELL);
  }
  if (s == s0) count[c] = 0;
  perm[slot] = i;
  xs[slot] = p.x; ys[slot] = p.y; zs[slot] = p.z;
}

// Bounding boxes of the 16 blocks of every 512-slot tile and of the tile itself: (min x, min y,
// min z, max x) and (max y, max z, -, -). Real ions only: a block without ions gets an inverted
// box that is never within range. Slots past the ions become far-away sentinels that no ion owns.
constexpr int kTile = 512, kBlk = 32, kTB = kTile / kBlk;
__global__ void __launch_bounds__(kTile) k_tile_box(int n, float* __restrict__ xs,
                                                    float* __restrict__ ys, float* __restrict__ zs,
                                                    int32_t* __restrict__ perm,
                                                    float4* __restrict__ bbox,
                                                    float4* __restrict__ tbox) {
  od_pdl_wait();
  od_pdl_trigger();
  __shared__ float tb[kTB][6];
  const int t = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = t * kTile + threadIdx.x;
  float b[6] = {3e38f, 3e38f, 3e38f, -3e38f, -3e38f, -3e38f};
  if (i < n) {
    b[0] = b[3] = xs[i]; b[1] = b[4] = ys[i]; b[2] = b[5] = zs[i];
  } else {
    xs[i] = ys[i] = zs[i] = OD_SENTINEL;
    perm[i] = -1;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int d = 0; d < 3; d++) {
      b[d] = fminf(b[d], __shfl_xor_sync(0xffffffffu, b[d], o));
      b[3 + d] = fmaxf(b[3 + d], __shfl_xor_sync(0xffffffffu, b[3 + d], o));
    }
  if (lane == 0) {
    bbox[2 * (t * kTB + w)] = make_float4(b[0], b[1], b[2], b[3]);
    bbox[2 * (t * kTB + w) + 1] = make_float4(b[4], b[5], 0.f, 0.f);
#pragma unroll
    for (int d = 0; d < 6; d++) tb[w][d] = b[d];
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    float v = tb[0][threadIdx.x];
    for (int k = 1; k < kTB; k++)
      v = threadIdx.x < 3 ? fminf(v, tb[k][threadIdx.x]) : fmaxf(v, tb[k][threadIdx.x]);
    reinterpret_cast<float*>(tbox + 2 * t)[threadIdx.x] = v;
  }
}

// ------------------------------------------------------------------ pair terms
// CUT = 0: the plain screened term (blocks inside the switching radius); 1: OpenMM's switching
// polynomial on the energy, S = (1-x)^3 (1 + 3x + 6x^2), x = (r - r_s)/(r_c - r_s) clamped to
// [0, 1], so that pairs beyond r_c contribute exactly 0 (opendust.py:481-485); 2: hard cutoff.
struct cut_args {
  float rho0, rc2, rs, inv_w;
  float in2;    // blocks closer than sqrt(in2) throughout take CUT = 0
  float cull2;  // blocks farther than sqrt(cull2) are skipped
  double rcd;   // hard cutoff: r_c (lambda) in FP64
};
struct cut_consts {
  od_u64 eps, rho, nl2e, one, three, six, w30, rc2;
  float invw, nrsw, rc2f, skip2, band;
};
__device__ __forceinline__ cut_consts make_consts(const cut_args& c) {
  cut_consts k;
  k.eps = p2(1e-30f, 1e-30f);
  k.rho = p2(c.rho0, c.rho0);
  k.nl2e = p2(OD_NLOG2E, OD_NLOG2E);
  k.one = p2(1.f, 1.f); k.three = p2(3.f, 3.f); k.six = p2(6.f, 6.f);
  k.w30 = p2(30.f * c.inv_w, 30.f * c.inv_w);
  k.rc2 = p2(c.rc2, c.rc2);
  k.invw = c.inv_w;
  k.nrsw = -c.rs * c.inv_w;
  k.rc2f = c.rc2;
  // (1 + 2e-5) rc^2: beyond it the clamped switching variable is 1 in FP32 and the switched term
  // exactly zero (the hard cutoff is exactly zero from rc^2 on)
  k.skip2 = c.rc2 * 1.00002f;
  // the FP32 r^2 of a pair is within 4e-7 of its exact value on the same float positions
  k.band = c.rc2 * 2e-6f;
  return k;
}
__device__ __forceinline__ float fma_sat(float a, float b, float c) {
  float r; asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r;
}

// Is the pair of float positions t, s inside the cutoff as the FP64 reference decides it:
// sqrt((dx^2 + dy^2) + dz^2) < r_c with the differences taken exactly in FP64 and every
// operation rounded once (the oracle's pair_factor).
__device__ __noinline__ bool inside_exact(float tx, float ty, float tz, float sx, float sy,
                                          float sz, double rcd) {
  const double dx = __dsub_rn((double)tx, (double)sx), dy = __dsub_rn((double)ty, (double)sy),
               dz = __dsub_rn((double)tz, (double)sz);
  const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  return __dsqrt_rn(r2) < rcd;
}

// One pack: a target (in both halves) against two sources, as od_n3.cu's pair_once with R = r and
// W = 1/(r (r + rho)). Switching, with u = exp(-r)/s: c = exp(-r) W [(1 + 1/s) S + 30 x^2 (1-x)^2
// /(r_c - r_s)] = exp(-r) W (1-x)^2 [(1 + W r)(1-x)(1 + 3x + 6x^2) + 30 x^2/(r_c - r_s)] (no
// cancellation as x -> 1; x by a saturating fma, so that neither x nor 1 - x needs a clamp). A pack
// whose 64 pairs all lie beyond the cutoff is skipped (a warp vote: 22.7 ms with it at field_chain,
// 25.5 without; a second vote that skips the switching part where no pair needs it made the
// kernel 5 % slower). Hard cutoff: pairs more than `band` inside count here, pairs within it are
// left to the exact pass; near keeps the smallest |r^2 - r_c^2|. COUNT adds the pairs inside.
template <int CUT, bool REACT, bool COUNT>
__device__ __forceinline__ void cut_pair(const cut_consts& k, od_u64 X, od_u64 Y, od_u64 Z, od_u64 QX,
                                         od_u64 QY, od_u64 QZ, od_u64& AX, od_u64& AY, od_u64& AZ,
                                         od_u64& RX, od_u64& RY, od_u64& RZ, float& near,
                                         unsigned int& cnt) {
  const od_u64 DX = sub2(X, QX), DY = sub2(Y, QY), DZ = sub2(Z, QZ);
  od_u64 R2 = fma2(DX, DX, k.eps);
  R2 = fma2(DY, DY, R2);
  R2 = fma2(DZ, DZ, R2);
  const float2 r2 = up2(R2);
  if (CUT != 0 && __all_sync(0xffffffffu, fminf(r2.x, r2.y) >= k.skip2)) return;
  const od_u64 R = p2(od_sqrt(r2.x), od_sqrt(r2.y));
  const float2 rs = up2(fma2(R, k.rho, R2));
  const od_u64 W = p2(od_rcp(rs.x), od_rcp(rs.y));
  const float2 ea = up2(mul2(R, k.nl2e));
  const od_u64 EX = p2(od_ex2(ea.x), od_ex2(ea.y));
  const od_u64 SI = mul2(W, R);
  od_u64 C;
  if (CUT == 0) {
    C = mul2(EX, fma2(W, SI, W));
  } else if (CUT == 1) {
    const float2 r = up2(R);
    const od_u64 x = p2(fma_sat(r.x, k.invw, k.nrsw), fma_sat(r.y, k.invw, k.nrsw));
    const od_u64 om = sub2(k.one, x);
    const od_u64 P = mul2(om, fma2(x, fma2(k.six, x, k.three), k.one));
    const od_u64 V = fma2(mul2(x, x), k.w30, fma2(SI, P, P));
    C = mul2(mul2(W, mul2(om, om)), mul2(EX, V));
  } else {
    const float2 c = up2(mul2(EX, fma2(W, SI, W)));
    const float2 e = up2(sub2(R2, k.rc2));
    near = fminf(near, fminf(fabsf(e.x), fabsf(e.y)));
    C = p2(e.x < -k.band ? c.x : 0.f, e.y < -k.band ? c.y : 0.f);
  }
  if (COUNT) {
    const float lim = CUT == 2 ? -k.band : 0.f;
    cnt += (REACT ? 2u : 1u) * ((unsigned)(r2.x - k.rc2f < lim && r2.x > 1e-29f) +
                                (unsigned)(r2.y - k.rc2f < lim && r2.y > 1e-29f));
  }
  AX = fma2(C, DX, AX); AY = fma2(C, DY, AY); AZ = fma2(C, DZ, AZ);
  if (REACT) { RX = fma2(C, DX, RX); RY = fma2(C, DY, RY); RZ = fma2(C, DZ, RZ); }
}

// Hard cutoff, the exact pass of half a batch: pairs whose FP32 r^2 lies within `band` of r_c^2 are
// decided as the FP64 reference decides them and added straight to the accumulators, so that both
// include the same pairs (rare: about 1 half in 50 at field_chain has such a pair).
template <bool REACT, bool COUNT>
__device__ __noinline__ void exact_pass(const float* __restrict__ xs, const float* __restrict__ ys,
                                        const float* __restrict__ zs, size_t ns,
                                        unsigned long long* __restrict__ acc, const cut_args& cut,
                                        int sg, const unsigned int* tb, int nb, int half,
                                        unsigned int& cnt) {
  const int lane = threadIdx.x & 31;
  const float band = cut.rc2 * 2e-6f;
  for (int t = 0; t < nb; t++) {
    const int ti = (int)tb[t] * kBlk + lane;
    const float px = xs[ti], py = ys[ti], pz = zs[ti];
    for (int j = 0; j < 32; j++) {  // 16 lane steps, two sources each
      const int sj = sg * 64 + 2 * (j & 16) + ((lane + 16 * half + (j & 15)) & 31);
      const float sx = xs[sj], sy = ys[sj], sz = zs[sj];
      const float dx = px - sx, dy = py - sy, dz = pz - sz;
      const float r2 = fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, 1e-30f)));
      const float e = r2 - cut.rc2;
      if (!(e < -band) && e <= band && inside_exact(px, py, pz, sx, sy, sz, cut.rcd)) {
        const float c = od_pair_c(r2, cut.rho0);
        od_fix_add1(acc + ti, c * dx); od_fix_add1(acc + ns + ti, c * dy);
        od_fix_add1(acc + 2 * ns + ti, c * dz);
        if (REACT) {
          od_fix_add1(acc + sj, -c * dx); od_fix_add1(acc + ns + sj, -c * dy);
          od_fix_add1(acc + 2 * ns + sj, -c * dz);
        }
        if (COUNT) cnt += REACT ? 2u : 1u;
      }
    }
  }
}

// MT target blocks tb[0 .. nb) (nb <= MT, the rest empty) against the 64 slots of source group sg:
// halves [h0, h1) of the 32 lane steps. Reactions are summed in FP32 over 16 lane steps and added to
// the accumulators of the sources where they stand (shorter chains than the 32 steps they could take: at 2^19 ions the median per-ion
// error is 0.8 of that and the kernel 1 % slower).
template <int MT, int CUT, bool REACT, bool COUNT, int UNROLL>
__device__ __forceinline__ void cut_batch(const cut_consts& k, const float* __restrict__ xs,
                                          const float* __restrict__ ys,
                                          const float* __restrict__ zs, size_t ns,
                                          unsigned long long* __restrict__ acc,
                                          const cut_args& cut, int sg, const unsigned int* tb,
                                          int nb, unsigned int& cnt, int h0 = 0, int h1 = 2) {
  const int lane = threadIdx.x & 31, src = (lane + 1) & 31;
  od_u64 X[MT], Y[MT], Z[MT], AX[MT], AY[MT], AZ[MT];
#pragma unroll
  for (int t = 0; t < MT; t++) {
    float x = OD_SENTINEL, y = OD_SENTINEL, z = OD_SENTINEL;
    if (t < nb) {
      const int i = (int)tb[t] * kBlk + lane;
      x = xs[i]; y = ys[i]; z = zs[i];
    }
    X[t] = p2(x, x); Y[t] = p2(y, y); Z[t] = p2(z, z);
    AX[t] = AY[t] = AZ[t] = 0ull;
  }
  const int j = sg * 64 + ((lane + 16 * h0) & 31);
  od_u64 QX = p2(xs[j], xs[j + 32]), QY = p2(ys[j], ys[j + 32]), QZ = p2(zs[j], zs[j + 32]);
#pragma unroll 1
  for (int h = h0; h < h1; h++) {
    od_u64 RX = 0ull, RY = 0ull, RZ = 0ull;
    float near = 3e38f;
#pragma unroll UNROLL
    for (int st = 0; st < 16; st++) {
#pragma unroll
      for (int t = 0; t < MT; t++)
        cut_pair<CUT, REACT, COUNT>(k, X[t], Y[t], Z[t], QX, QY, QZ, AX[t], AY[t], AZ[t], RX, RY,
                                    RZ, near, cnt);
      QX = shfl64(QX, src); QY = shfl64(QY, src); QZ = shfl64(QZ, src);
      if (REACT) { RX = shfl64(RX, src); RY = shfl64(RY, src); RZ = shfl64(RZ, src); }
    }
    if (REACT) {  // the force on the sources is minus the accumulated terms
      const float2 rx = up2(RX), ry = up2(RY), rz = up2(RZ);
      unsigned long long* a = acc + sg * 64 + ((lane + 16 * h + 16) & 31);
      od_fix_add1(a, -rx.x); od_fix_add1(a + 32, -rx.y);
      od_fix_add1(a + ns, -ry.x); od_fix_add1(a + ns + 32, -ry.y);
      od_fix_add1(a + 2 * ns, -rz.x); od_fix_add1(a + 2 * ns + 32, -rz.y);
    }
    if (CUT == 2 && __any_sync(0xffffffffu, near <= k.band))
      exact_pass<REACT, COUNT>(xs, ys, zs, ns, acc, cut, sg, tb, nb, h, cnt);
  }
#pragma unroll
  for (int t = 0; t < MT; t++)
    if (t < nb) {
      unsigned long long* a = acc + (int)tb[t] * kBlk + lane;
      od_fix_add1(a, sum2(AX[t]));
      od_fix_add1(a + ns, sum2(AY[t]));
      od_fix_add1(a + 2 * ns, sum2(AZ[t]));
    }
}

// squared nearest and farthest distance of a box from box a (min xyz, max xyz)
__device__ __forceinline__ void box_dist(const float4* __restrict__ box, int i, const float (&a)[6],
                                         float& d2, float& f2) {
  const float4 u = box[2 * i], v = box[2 * i + 1];
  const float lo[3] = {u.x, u.y, u.z}, hi[3] = {u.w, v.x, v.y};
  d2 = 0.f;
  f2 = 0.f;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const float gap = fmaxf(fmaxf(lo[d] - a[3 + d], a[d] - hi[d]), 0.f);
    const float far = fmaxf(hi[d] - a[d], a[3 + d] - lo[d]);
    d2 = fmaf(gap, gap, d2);
    f2 = fmaf(far, far, f2);
  }
}

// box of source group sg
__device__ __forceinline__ void group_box(const float4* __restrict__ bbox, int sg, float (&b)[6]) {
  const float4 p = bbox[4 * sg], q = bbox[4 * sg + 1], r = bbox[4 * sg + 2], s = bbox[4 * sg + 3];
  b[0] = fminf(p.x, r.x); b[1] = fminf(p.y, r.y); b[2] = fminf(p.z, r.z);
  b[3] = fmaxf(p.w, r.w); b[4] = fmaxf(q.x, s.x); b[5] = fmaxf(q.y, s.y);
}

// Units: source group sg (row a = sg / 8) and its c-th run of B tiles from tile a on, numbered run by
// run over the groups, c = 0 first. Units before run c: 8 (c nT - B c (c - 1) / 2).
__host__ __device__ __forceinline__ long long units_before(long long c, int nT, int B) {
  return 8 * (c * nT - B * (c * (c - 1) / 2));
}

// Registers: resident warps and unrolling. field_chain, ms per evaluation: switching 22.6 with 24 warps per
// SM and two lane steps (22.9 with 20, 22.5 with 28 and one step, 24.5 with 16), hard cutoff 20.5 with 20
// and one step (21.2 with 24 and two); 65536 ions at 2 lambda 0.594 and 0.548 ms.
template <int CUT>
struct cut_traits {
  static constexpr int WARPS = 4;  // per block; they share nothing
  static constexpr int MIN_BLOCKS = CUT == 2 ? 5 : 6;
  static constexpr int UNROLL = CUT == 2 ? 1 : 2;
};

template <int CUT, bool COUNT>
__global__ void __launch_bounds__(cut_traits<CUT>::WARPS * 32, cut_traits<CUT>::MIN_BLOCKS)
    k_pairs_cutn3(const float* __restrict__ xs, const float* __restrict__ ys,
                  const float* __restrict__ zs, int nslots, int nT, int B, long long nunits,
                  unsigned long long* __restrict__ next, unsigned long long* __restrict__ acc,
                  const __grid_constant__ cut_args cut, const float4* __restrict__ tbox,
                  const float4* __restrict__ bbox, unsigned long long* __restrict__ pair_count) {
  od_pdl_wait();
  od_pdl_trigger();
  constexpr int WARPS = cut_traits<CUT>::WARPS, UNROLL = cut_traits<CUT>::UNROLL;
  // per warp: target blocks waiting, those that need the cutoff term and the inner ones (at most 3
  // left over plus the 32 of one round)
  __shared__ unsigned int s_list[WARPS][2][40];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned int* const qo = s_list[w][0];
  unsigned int* const qi = s_list[w][1];
  const cut_consts k = make_consts(cut);
  unsigned int cnt = 0;
  for (;;) {
    unsigned long long u = 0;
    if (lane == 0) u = atomicAdd(next, 1ull);
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u >= (unsigned long long)nunits) break;
    int sg, b0, b1;
    {
      const float h = (float)nT + 0.5f * (float)B;
      int c = (int)((h - sqrtf(fmaxf(h * h - 0.25f * (float)B * (float)u, 0.f))) / (float)B);
      while (c > 0 && units_before(c, nT, B) > (long long)u) c--;
      while (units_before(c + 1, nT, B) <= (long long)u) c++;
      sg = (int)((long long)u - units_before(c, nT, B));
      b0 = (sg >> 3) + c * B;
      b1 = min(b0 + B, nT);
    }
    float sb[6];
    group_box(bbox, sg, sb);
    unsigned int tiles;
    {
      float d2 = 3e38f, f2;
      if (b0 + lane < b1) box_dist(tbox, b0 + lane, sb, d2, f2);
      tiles = __ballot_sync(0xffffffffu, d2 < cut.cull2);
    }
    if (b0 == sg >> 3) {  // the group itself: directed
      if (lane < 2) qo[lane] = 2 * sg + lane;
      __syncwarp();
      cut_batch<2, CUT, false, COUNT, 1>(k, xs, ys, zs, nslots, acc, cut, sg, qo, 2, cnt);
      __syncwarp();
    }
    int no = 0, ni = 0;
    while (tiles) {
      // two tiles a round: lanes 0-15 the blocks of the first, 16-31 of the second
      const int t1 = __ffs(tiles) - 1;
      tiles &= tiles - 1;
      const int t2 = tiles ? __ffs(tiles) - 1 : -1;
      if (tiles) tiles &= tiles - 1;
      const int tl = lane < 16 ? t1 : t2;
      const int blk = (b0 + tl) * kTB + (lane & 15);
      float d2 = 3e38f, f2 = 3e38f;
      if (tl >= 0 && blk > 2 * sg + 1) box_dist(bbox, blk, sb, d2, f2);
      const bool keep = d2 < cut.cull2, inner = keep && f2 < cut.in2;
      const unsigned int mi = __ballot_sync(0xffffffffu, inner),
                         mo = __ballot_sync(0xffffffffu, keep && !inner);
      const unsigned int below = (1u << lane) - 1u;
      if (inner) qi[ni + __popc(mi & below)] = blk;
      else if (keep) qo[no + __popc(mo & below)] = blk;
      ni += __popc(mi);
      no += __popc(mo);
      __syncwarp();
      const bool last = tiles == 0;
      if (last) {  // the inner blocks that fill no batch join the others
        const int r = ni & 3;
        if (lane < r) qo[no + lane] = qi[ni - r + lane];
        no += r;
        ni -= r;
        __syncwarp();
      }
      for (; ni >= 4; ni -= 4)
        cut_batch<4, 0, true, COUNT, UNROLL>(k, xs, ys, zs, nslots, acc, cut, sg, qi + ni - 4, 4,
                                             cnt);
      for (; no >= 4; no -= 4)
        cut_batch<4, CUT, true, COUNT, UNROLL>(k, xs, ys, zs, nslots, acc, cut, sg, qo + no - 4, 4,
                                               cnt);
      if (last && no > 2)
        cut_batch<4, CUT, true, COUNT, UNROLL>(k, xs, ys, zs, nslots, acc, cut, sg, qo, no, cnt);
      else if (last && no > 0)
        cut_batch<2, CUT, true, COUNT, 1>(k, xs, ys, zs, nslots, acc, cut, sg, qo, no, cnt);
      __syncwarp();
    }
  }
  if (COUNT) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if (lane == 0 && cnt) atomicAdd(pair_count, (unsigned long long)cnt);
  }
}

// ------------------------------------------------------------------ small systems: listed work
// Up to kListBlocks blocks the units above are too coarse: a warp gets a few batches, and the last ones
// run alone (force chain of 8192 ions at 2 lambda 0.132 ms). Here one warp per source group lists its
// target blocks first (inner ones from the front of its row, the others from the back), every block of the
// pair kernel takes the prefix over the groups, and its warps draw runs of equal length from it: half
// batches where there are fewer than six per warp (20011 ions 118.9 us per step, whole batches 121.5;
// 30000, with eight to twelve per warp, 195.0 and 193.1), else whole ones, 32 runs per warp (65536 ions 0.594 ms, 0.635
// with the units). Ending whole runs with a round of halves: 117.0 us at 20011 ions, but 588 instead of
// 585 at 65536 and 1864 instead of 1848 at 131072.
constexpr int kListBlocks = 4096;
__global__ void __launch_bounds__(256) k_cut_lists(int nsg, int nT, const cut_args cut,
                                                   const float4* __restrict__ tbox,
                                                   const float4* __restrict__ bbox,
                                                   uint16_t* __restrict__ rows,
                                                   int2* __restrict__ cnt) {
  od_pdl_wait();
  od_pdl_trigger();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int sg = blockIdx.x * 8 + w, nB = nT * kTB;
  if (sg < nsg) {
    float sb[6];
    group_box(bbox, sg, sb);
    uint16_t* const row = rows + (size_t)sg * nB;
    int ni = 0, no = 0;
    for (int b0 = sg >> 3; b0 < nT; b0 += 32) {
      float d2 = 3e38f, f2;
      if (b0 + lane < nT) box_dist(tbox, b0 + lane, sb, d2, f2);
      unsigned int tiles = __ballot_sync(0xffffffffu, d2 < cut.cull2);
      while (tiles) {
        // eight tiles a round, two at a time, so that their loads overlap (20011 ions: 10.3 us with
        // two a round)
        int blk[4];
        float near2[4], far2[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const int t1 = __ffs(tiles) - 1;  // -1: none left
          tiles &= tiles - 1;
          const int t2 = __ffs(tiles) - 1;
          tiles &= tiles - 1;
          const int tl = lane < 16 ? t1 : t2;
          blk[r] = (b0 + tl) * kTB + (lane & 15);
          near2[r] = far2[r] = 3e38f;
          if (tl >= 0 && blk[r] > 2 * sg + 1) box_dist(bbox, blk[r], sb, near2[r], far2[r]);
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const bool keep = near2[r] < cut.cull2, inner = keep && far2[r] < cut.in2;
          const unsigned int mi = __ballot_sync(0xffffffffu, inner),
                             mo = __ballot_sync(0xffffffffu, keep && !inner);
          const unsigned int below = (1u << lane) - 1u;
          if (inner) row[ni + __popc(mi & below)] = (uint16_t)blk[r];
          else if (keep) row[nB - 1 - no - __popc(mo & below)] = (uint16_t)blk[r];
          ni += __popc(mi);
          no += __popc(mo);
        }
      }
    }
    if (lane == 0) cnt[sg] = make_int2(ni, no);
  }
}

template <int CUT, bool COUNT>
__global__ void __launch_bounds__(cut_traits<CUT>::WARPS * 32, cut_traits<CUT>::MIN_BLOCKS)
    k_pairs_cutlist(const float* __restrict__ xs, const float* __restrict__ ys,
                    const float* __restrict__ zs, int nslots, unsigned long long* __restrict__ acc,
                    const __grid_constant__ cut_args cut, const uint16_t* __restrict__ rows,
                    const int2* __restrict__ counts, unsigned int* __restrict__ next,
                    unsigned long long* __restrict__ pair_count) {
  od_pdl_wait();
  od_pdl_trigger();
  constexpr int WARPS = cut_traits<CUT>::WARPS, UNROLL = cut_traits<CUT>::UNROLL;
  __shared__ int s_prefix[kListBlocks / 2 + 1];
  __shared__ unsigned int s_tb[WARPS][4];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nsg = nslots / 64, nB = nslots / kBlk;
  {  // prefix of the groups' half batches: the group itself, the inner fours, the rest
    __shared__ int s_w[WARPS];
    const int per = (nsg + WARPS * 32 - 1) / (WARPS * 32);
    const int g0 = min((int)threadIdx.x * per, nsg), g1 = min(g0 + per, nsg);
    int sum = 0;
#pragma unroll 4
    for (int g = g0; g < g1; g++) {
      const int2 c = counts[g];
      const int q = 2 * (1 + c.x / 4 + (c.y + (c.x & 3) + 3) / 4);
      s_prefix[g] = q;
      sum += q;
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_w[w] = incl;
    __syncthreads();
    int off = incl - sum;
    for (int v = 0; v < w; v++) off += s_w[v];
    for (int g = g0; g < g1; g++) {
      const int q = s_prefix[g];
      s_prefix[g] = off;
      off += q;
    }
    if (threadIdx.x == WARPS * 32 - 1) s_prefix[nsg] = off;
    __syncthreads();
  }
  unsigned int* const tb = s_tb[w];
  const cut_consts k = make_consts(cut);
  unsigned int cnt = 0;
  const int Q = s_prefix[nsg], W = gridDim.x * WARPS;
  const int run = Q < 6 * W ? 1 : max(2, (Q / (W * 32)) & ~1);
  for (;;) {
    int q = 0;
    if (lane == 0) q = (int)min(atomicAdd(next, 1u), (unsigned)Q) * run;
    q = __shfl_sync(0xffffffffu, q, 0);
    if (q >= Q) break;
    const int q1 = min(q + run, Q);
    int sg = 0;
    for (int hi = nsg; hi - sg > 1;) {  // the group whose range holds q
      const int mid = (sg + hi) >> 1;
      if (s_prefix[mid] <= q) sg = mid;
      else hi = mid;
    }
    while (q < q1) {
      while (s_prefix[sg + 1] <= q) sg++;
      const int r = q - s_prefix[sg], b = r >> 1, h0 = r & 1;
      const int h1 = min(2, h0 + q1 - q);
      const int2 c = counts[sg];
      const int fours = c.x >> 2, rest = c.x & 3;
      const uint16_t* const row = rows + (size_t)sg * nB;
      int nb = 4;
      __syncwarp();
      if (b == 0) {  // the group itself
        nb = 2;
        if (lane < 2) tb[lane] = 2 * sg + lane;
      } else if (b <= fours) {
        if (lane < 4) tb[lane] = row[4 * (b - 1) + lane];
      } else {  // the inner blocks that fill no batch, then the others
        const int at = 4 * (b - 1 - fours);
        nb = min(4, c.y + rest - at);
        if (lane < nb)
          tb[lane] = at + lane < rest ? row[4 * fours + at + lane] : row[nB - 1 - (at + lane - rest)];
      }
      __syncwarp();
      if (b == 0)
        cut_batch<2, CUT, false, COUNT, 1>(k, xs, ys, zs, nslots, acc, cut, sg, tb, 2, cnt, h0, h1);
      else if (b <= fours)
        cut_batch<4, 0, true, COUNT, UNROLL>(k, xs, ys, zs, nslots, acc, cut, sg, tb, 4, cnt, h0, h1);
      else if (nb > 2)
        cut_batch<4, CUT, true, COUNT, UNROLL>(k, xs, ys, zs, nslots, acc, cut, sg, tb, nb, cnt, h0,
                                               h1);
      else
        cut_batch<2, CUT, true, COUNT, 1>(k, xs, ys, zs, nslots, acc, cut, sg, tb, nb, cnt, h0, h1);
      q += h1 - h0;
    }
  }
  if (COUNT) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if (lane == 0 && cnt) atomicAdd(pair_count, (unsigned long long)cnt);
  }
}

// Slot accumulators -> the ions' entries of (ph, pl) as two-float sums (slot s holds ion
// perm[s], -1 for the sentinels in the tail), every slot cleared for the next evaluation.
__global__ void __launch_bounds__(256) k_slot_take(int nslots, unsigned long long* __restrict__ acc,
                                                  const int32_t* __restrict__ perm,
                                                  float4* __restrict__ ph, float4* __restrict__ pl) {
  od_pdl_wait();
  od_pdl_trigger();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nslots) return;
  float3 hi, lo;
  od_fix_take(acc + e, (size_t)nslots, hi, lo);
  const int i = perm[e];
  if (i < 0) return;
  ph[i] = make_float4(hi.x, hi.y, hi.z, 0.f);
  pl[i] = make_float4(lo.x, lo.y, lo.z, 0.f);
}

}  // namespace

od_cgrid od_cutn3_grid(int N, double R, double H) {
  od_cgrid g;
  // a domain at most 1.5 times as high as wide is one cube; a taller one a column of cubes as
  // wide as the domain, so that the cells keep their size whatever the aspect ratio
  g.nb = H <= 3.0 * R ? 1 : (int)std::ceil(H / (2.0 * R));
  g.side = (g.nb == 1 ? std::max(2.0 * R, H) : 2.0 * R) * 1.02;
  // 1.4 to 11 ions per cell of a cube: the sort's order inside a cell is arbitrary, so smaller cells give
  // tighter blocks. Against 2.8 to 22 and, before, up to 128 per cell, us per step: 20011 ions 128, 128,
  // 137; 40000 298, 298, 328; 65536 606, 616, 616; 131072 1870, 1870, 1968; 2^19 22270, 22710, 22710
  const double per = (double)N / g.nb;
  g.G = 8;
  while (g.G < 128 && (double)g.G * g.G * g.G * 8.0 * 2.0 < per * 1.4142) g.G <<= 1;
  g.ncells = g.nb * g.G * g.G * g.G;
  return g;
}

bool od_cutn3_listed(size_t nslots) { return nslots / kBlk <= kListBlocks; }
static size_t od_cutn3_list_bytes(size_t ns) {
  const size_t nsg = ns / 64, nB = ns / kBlk;
  return od_cutn3_listed(ns) ? sizeof(uint16_t) * nsg * nB + sizeof(int2) * nsg
                             : 0;
}

size_t od_cutn3_bytes(int N, int T, int ncells) {
  const size_t ns = (size_t)((N + T - 1) / T) * T, nc = (size_t)ncells;
  return sizeof(unsigned long long) * (3 * ns + 1)                    // accumulators, work counter
         + sizeof(float4) * 2 * (ns / kBlk + ns / kTile)              // boxes
         + od_cutn3_list_bytes(ns)
         + sizeof(float) * 3 * ns                                     // sorted positions
         + sizeof(int32_t) * (ns + 3 * (size_t)N + 2 * nc + 2 + nc / 4096);
}

bool od_cutn3_supported(int ipt, int T) {
  return (ipt == 2 && T == 512) || (ipt == 4 && T == 1024);
}

// resident blocks per SM of the pair kernel (the persistent grid is this times the SM count)
int od_cutn3_blocks_per_sm(bool hard) {
  int nb = 0;
  const cudaError_t e =
      hard ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_pairs_cutn3<2, false>,
                                                           cut_traits<2>::WARPS * 32, 0)
           : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_pairs_cutn3<1, false>,
                                                           cut_traits<1>::WARPS * 32, 0);
  if (e != cudaSuccess) cudaGetLastError();
  return e == cudaSuccess && nb > 0 ? nb : 5;
}

#define OD_CUTN3_FORMS()                       \
  do {                                         \
    if (sw) {                                  \
      if (pair_count) OD_CUTN3(1, true);       \
      else OD_CUTN3(1, false);                 \
    } else {                                   \
      if (pair_count) OD_CUTN3(2, true);       \
      else OD_CUTN3(2, false);                 \
    }                                          \
  } while (0)

cudaError_t od_launch_cutoff_n3(const od_cutn3& L, const float4* pos, int n, float4* part_hi,
                                float4* part_lo, float rho0, float rc, float rs, uint32_t* err,
                                unsigned long long* pair_count, cudaStream_t s) {
  // every kernel of the chain with programmatic dependent launch, the next one let in only after the
  // wait (8192 ions 72.0 -> 68.7 us per step, 20011 140 -> 137; let in before it, the waiting blocks of
  // two kernels on, the pair kernel's among them, hold the SMs: 142)
  const dim3 nb((n + 255) / 256), nt(256);
  const int nT = L.nslots / kTile;
  cudaError_t e = od_launch_pdl(k_mc_count, nb, nt, s, n, pos, L.lo, L.lo_z, L.inv_s, L.G, L.nb,
                                L.cell_of, L.rank_of, L.count, L.next);
  if (L.ncells <= kScanCells) {
    if (e == cudaSuccess)
      e = od_launch_pdl_smem(k_mc_scan_scatter, nb, nt, sizeof(int32_t) * (L.ncells + L.ncells / 16), s,
                             n, L.ncells, (const int32_t*)L.cell_of, (const int32_t*)L.rank_of,
                             (const int32_t*)L.count, L.start, L.unsorted);
  } else {
    const int sb = L.ncells / kScanBlock;
    if (e == cudaSuccess && L.ncells % kScanBlock == 0) {
      e = od_launch_pdl(k_scan_blocks, dim3(sb), dim3(1024), s, (const int32_t*)L.count, L.start,
                        L.totals);
      if (e == cudaSuccess)
        e = od_launch_pdl(k_scan_add, dim3(sb), dim3(1024), s, L.ncells, (const int32_t*)L.totals,
                          L.start);
    } else if (e == cudaSuccess) {
      e = od_launch_pdl(k_scan_excl, dim3(1), dim3(1024), s, L.ncells, (const int32_t*)L.count,
                        L.start);
    }
    if (e == cudaSuccess)
      e = od_launch_pdl(k_mc_scatter, nb, nt, s, n, (const int32_t*)L.cell_of,
                        (const int32_t*)L.rank_of, (const int32_t*)L.start, L.unsorted);
  }
  if (e == cudaSuccess)
    e = od_launch_pdl(k_mc_sort, nb, nt, s, n, (const int32_t*)L.cell_of, (const int32_t*)L.start,
                      (const int32_t*)L.unsorted, pos, L.count, L.perm, L.xs, L.ys, L.zs,
                      err);
  if (e == cudaSuccess)
    e = od_launch_pdl(k_tile_box, dim3(nT), dim3(kTile), s, n, L.xs, L.ys, L.zs, L.perm, L.bbox,
                      L.tbox);
  if (e != cudaSuccess) return e;
  const bool sw = rs < rc;
  // blocks whose farthest box distance is below the switching radius (hard cutoff: the cutoff), with a
  // relative margin of 1e-5 against rounding, skip the switching polynomial; blocks whose nearest box
  // distance is beyond the cutoff, with the same margin, are skipped
  const float rin = (sw ? rs : rc) * (1.0f - 1e-5f);
  const cut_args cut{rho0, rc * rc, rs, sw ? 1.0f / (rc - rs) : 0.0f, rin * rin,
                     rc * rc * 1.00001f, L.rc_d};
  const int grid = sw ? L.grid : L.grid_hard;
  if (L.rows) {
    const int nsg = L.nslots / 64;
    e = od_launch_pdl(k_cut_lists, dim3((nsg + 7) / 8), nt, s, nsg, nT, cut, (const float4*)L.tbox,
                      (const float4*)L.bbox, L.rows, L.counts);
    if (e != cudaSuccess) return e;
#define OD_CUTN3(CUT, CNT)                                                                       \
  e = od_launch_pdl(k_pairs_cutlist<CUT, CNT>, dim3(grid), dim3(cut_traits<CUT>::WARPS * 32), s, \
                    (const float*)L.xs, (const float*)L.ys, (const float*)L.zs, L.nslots, L.acc, \
                    cut, (const uint16_t*)L.rows, (const int2*)L.counts, (unsigned int*)L.next,  \
                    pair_count)
    OD_CUTN3_FORMS();
#undef OD_CUTN3
  } else {
    // tiles per unit: more in larger systems, so that the units, most of them empty, stay few beside
    // the work (2^19 ions: no difference from 4 to 16)
    const int B = std::min(32, std::max(1, nT / 128));
    const long long nunits = units_before((nT + B - 1) / B, nT, B);
#define OD_CUTN3(CUT, CNT)                                                                       \
  e = od_launch_pdl(k_pairs_cutn3<CUT, CNT>, dim3(grid), dim3(cut_traits<CUT>::WARPS * 32), s,   \
                    (const float*)L.xs, (const float*)L.ys, (const float*)L.zs, L.nslots, nT, B, \
                    nunits, L.next, L.acc, cut, (const float4*)L.tbox, (const float4*)L.bbox,    \
                    pair_count)
    OD_CUTN3_FORMS();
#undef OD_CUTN3
  }
  if (e != cudaSuccess) return e;
  return od_launch_pdl(k_slot_take, dim3((L.nslots + 255) / 256), nt, s, L.nslots, L.acc,
                       (const int32_t*)L.perm, part_hi, part_lo);
}
