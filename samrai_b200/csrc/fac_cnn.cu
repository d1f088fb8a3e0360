// Learned coarse-correction network: forward, backward and Adam kernels.
//
// Four 3x3x3 convolutions 1 -> 16 -> 16 -> 16 -> 1 channels, ReLU after
// the first three, no biases (so the network is positively homogeneous and
// the residual's scale passes straight through), zero padding at the edge
// of each sample.  Weights and stored activations are BF16; accumulation is
// FP32.  One sample is a patch plus a one-cell halo padded to an S^3 box
// (S = 18: patches of up to 16^3 cells).
//
// The 16 -> 16 layers run as implicit GEMMs on the 5th-generation tensor
// cores (k_conv_mid_tc: tcgen05.mma, BF16 operands in shared memory, FP32
// accumulators in tensor memory): a CTA stages slabs of z-planes of one
// sample with a zero halo in shared memory, and each 128-row tile of the
// slab's cells gets 9 MMAs, one per (y, z) tap shift, whose N holds the three
// x taps side by side (M = 128 cells, N = 3 x 16 output channels, K = 16 input
// channels); the shift is a move of the A operand's start address, the x taps
// are added from neighbouring rows when the accumulators are read.  The same
// kernel computes the backward pass with respect to
// the data (taps reversed, weights transposed, gated by the forward
// ReLU mask) and layer 4 (16 -> 1).  Weight gradients of the 16 -> 16 layers
// are 27 16 x 16 GEMMs reducing over all cells, from staged slabs
// (ldmatrix + mma.sync, three taps per warp).  The operations between one
// channel and 16 (layer 1, layer 4's data gradient, and the weight gradients
// of both) run on mma.sync with the taps as a matrix dimension: values of the
// one-channel field are gathered from a staged slab, FP32 fields as the sum of
// three BF16 numbers (split_bf16).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/samrai_fac_b200.h"
#include "fac_kernels.h"

namespace {

using samrai_b200::WaitTest;

constexpr int S = FAC_CNN_BOX;       // sample box side (patch + halo)
constexpr int S3 = S * S * S;
constexpr int C = 16;                // hidden channels
constexpr int T = 27;                // taps

__device__ __forceinline__ int tap_dx(int t) { return t % 3 - 1; }
__device__ __forceinline__ int tap_dy(int t) { return (t / 3) % 3 - 1; }
__device__ __forceinline__ int tap_dz(int t) { return t / 9 - 1; }

__device__ __forceinline__ void mma_bf16(float *d, const uint32_t *a, uint32_t b0, uint32_t b1)
{
   asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ---------------------------------------------------------------------------
// layers 2, 3, 4 (and the data gradients of 2, 3) on tcgen05.
//
// A CTA takes slabs of kTcNz output z-planes of one sample in turn.  It
// stages the slab's input planes z0-1 .. z0+kTcNz with a one-cell zero halo
// in x and y (kTcPx x kTcPx cells per plane) in shared memory, channels
// split in two planes of 8 (16 bytes per cell each): with cells as rows and
// channels as K, that is the K-major canonical layout without swizzle (8
// consecutive cells form a core matrix of 8 rows x 16 bytes; SBO = 128 bytes
// between groups of 8 cells, LBO = the distance of the two channel planes).
// Output row r (a padded cell index) needs input row r + off(tap), so a tap
// is the same descriptor with its start moved by off cells.  The three x taps
// of a (y, z) shift share one MMA: its N columns are (x tap, output channel),
// D[r][dx] holds the taps' part for the output row r - dx, and the output row
// is D[r-1][-1] + D[r][0] + D[r+1][+1], from the lanes beside; rows at the ends
// of a warp's 32 go through shared memory, one turn later.  The padded rows of
// halo positions are computed and dropped.  Accumulators: tile i of a half
// slab in tensor-memory columns N i .. of the half's 256, lane = row; warp w
// reads lanes 32 (w % 4) .. + 31.
//
// Everything is two deep: while one warp feeds the tensor cores half a slab
// (five tiles), the twenty others issue the copies of the next slab (cp.async)
// and read, gate, round and store the half before, a tile per four warps.  One
// CTA per SM.  What bounds it: the tensor cores read A from shared memory for
// every MMA, 40 cycles for 128 rows with N = 16 and 64 with N = 48 (one or five
// issuing threads alike), hence three taps per MMA; then the readers.  For 256
// samples (ncu): 80 us a 16 -> 16 convolution and 53 us layer 4, 102 us each
// with one MMA of N = 16 per tap and staging, multiplying and storing in turn
// (two CTAs per SM); one tap per MMA in the two-deep form 78 us each.
// ---------------------------------------------------------------------------
constexpr int kTcPx = S + 2;                         // padded row length
constexpr int kTcPlane = kTcPx * kTcPx;              // padded plane
constexpr int kTcNz = 3;                             // output planes per slab
constexpr int kTcSlabs = S / kTcNz;                  // slabs per sample
constexpr int kTcBox = (kTcNz + 2) * kTcPlane;       // staged cells
constexpr int kTcTiles = (kTcNz * kTcPlane + 127) / 128;
constexpr int kTcShifts = T / 3;                     // (y, z) shifts
constexpr int kTcReach = 1 + kTcPx + kTcPlane;       // largest |tap offset|
constexpr int kTcFront = 32;                         // cells before the box
constexpr int kTcSpan = kTcFront + kTcBox + 128;     // cells per channel plane
constexpr int kTcHalf = 256;                         // tensor-memory columns per half slab
constexpr int kTcHalfTiles = kTcTiles / 2;
constexpr int kTcPlaneBytes = kTcSpan * 16;
constexpr int kTcWBytes = T * 512;
constexpr int kTcRows = 128 * kTcTiles;
constexpr int kTcRuns = kTcRows / 32;                // a warp's rows
constexpr int kTcEdge = 5 * kTcRuns * 16;            // floats of the runs' end rows
constexpr int kTcReadWarps = 4 * kTcHalfTiles;       // four to a tile
constexpr int kTcReaders = 32 * kTcReadWarps;
constexpr int kTcThreads = kTcReaders + 32;
constexpr int kTcSmem = 4 * kTcPlaneBytes + kTcWBytes + 2 * 4 * kTcEdge + 2 * kTcBox + 2 * kTcRows + 32;
constexpr int kSlabCells = kTcNz * S * S;            // contiguous in a sample
constexpr unsigned short kNoCell = 0xffffu;
static_assert(S % kTcNz == 0, "whole slabs");
static_assert(kTcFront + kTcPlane - kTcReach >= 0, "front guard");
static_assert(kTcFront + kTcPlane + kTcRows + kTcReach <= kTcSpan, "back guard");
static_assert(kTcTiles % 2 == 0 && 48 * kTcHalfTiles <= kTcHalf, "accumulator columns");
static_assert(kTcPlaneBytes % 16 == 0 && (kTcPlaneBytes >> 4) < (1 << 14), "LBO field");
static_assert(kTcSmem <= 227 * 1024, "shared memory of one CTA");
static_assert(kTcBox % 4 == 0 && kTcRows % 4 == 0, "barriers aligned");
// instruction descriptor, kind::f16: FP32 accumulator (bits 4-5 = 1), BF16
// A and B (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at
// bit 24
template <unsigned N>
constexpr unsigned kTcIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) |
                              ((128u >> 4) << 24);
__device__ __forceinline__ unsigned tc_smem(const void *p)
{
   return (unsigned)__cvta_generic_to_shared(p);
}

// shared-memory matrix descriptor: start, leading and stride byte offsets
// (16-byte units), descriptor version 1, no swizzle
__device__ __forceinline__ unsigned long long tc_desc(unsigned addr, unsigned lbo, unsigned sbo)
{
   return (unsigned long long)((addr >> 4) & 0x3FFFu) |
          ((unsigned long long)((lbo >> 4) & 0x3FFFu) << 16) |
          ((unsigned long long)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ void tc_mma(unsigned d, unsigned long long a, unsigned long long b,
                                       unsigned idesc, unsigned accumulate)
{
   asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ bool tc_try_wait(unsigned bar, unsigned parity)
{
   unsigned ok;
   asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
   return ok != 0;
}

__device__ __forceinline__ void tc_ld8(unsigned taddr, unsigned *v)
{
   asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7])
      : "r"(taddr));
}

__device__ __forceinline__ void tc_ld_done()
{
   asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void copy16(unsigned dst, const void *src, bool on)
{
   asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0)
                : "memory");
}

__device__ __forceinline__ void copies_done()
{
   asm volatile("cp.async.wait_all;" ::: "memory");
}

// Cell (from the slab's first input plane, z0 - 1) of each position of the
// padded box, kNoCell for its x and y halo.
__device__ __forceinline__ void box_cells(unsigned short *tab, int tid, int nthr)
{
   for (int i = tid; i < kTcBox; i += nthr) {
      const int zz = i / kTcPlane, r = i - zz * kTcPlane;
      const int py = r / kTcPx, px = r - py * kTcPx;
      tab[i] = px >= 1 && px <= S && py >= 1 && py <= S
                  ? (unsigned short)(px - 1 + S * (py - 1 + S * zz)) : kNoCell;
   }
}

// The cell of the sample at position i of the box of slab z0, -1 outside the
// sample (planes below the first and above the last among them).
__device__ __forceinline__ int box_cell(const unsigned short *tab, int i, int z0)
{
   const int e = tab[i], cell = e + (z0 - 1) * S * S;
   return e != kNoCell && (unsigned)cell < (unsigned)S3 ? cell : -1;
}

// The box of slab z0 of sample xs (16 channels a cell) into the channel
// planes at shared addresses p0 and p1, zeros outside the sample; copies left
// in flight.
__device__ __forceinline__ void stage_slab(const __nv_bfloat16 *xs, int z0, const unsigned short *tab,
                                           unsigned p0, unsigned p1, int tid, int nthr)
{
   for (int i = tid; i < kTcBox; i += nthr) {
      const int cell = box_cell(tab, i, z0);
      const __nv_bfloat16 *src = xs + (cell >= 0 ? cell : 0) * C;
      copy16(p0 + 16u * (kTcFront + i), src, cell >= 0);
      copy16(p1 + 16u * (kTcFront + i), src + 8, cell >= 0);
   }
}

// eight output channels in FP32: ReLU, or the gate g > 0, to BF16
__device__ __forceinline__ void put_half(const float *o, __nv_bfloat16 *y, const uint4 &gg, int mode)
{
   const __nv_bfloat16 *g = reinterpret_cast<const __nv_bfloat16 *>(&gg);
   uint4 out;
   __nv_bfloat162 *ob = reinterpret_cast<__nv_bfloat162 *>(&out);
#pragma unroll
   for (int c = 0; c < 4; ++c) {
      float v0 = o[2 * c], v1 = o[2 * c + 1];
      if (mode == 0) {
         v0 = fmaxf(v0, 0.f);
         v1 = fmaxf(v1, 0.f);
      } else {
         v0 = __bfloat162float(g[2 * c]) > 0.f ? v0 : 0.f;
         v1 = __bfloat162float(g[2 * c + 1]) > 0.f ? v1 : 0.f;
      }
      ob[c] = __floats2bfloat162_rn(v0, v1);
   }
   *reinterpret_cast<uint4 *>(y) = out;
}

// wt: BF16 B operands [(y, z) shift][input-channel half][N][8 in]; N = 48,
// column (x tap, output channel), mode 0: y = relu(acc); mode 1: y = acc *
// (gate > 0).  N = 16 (layer 4): columns 0..2 the x taps of the one output
// channel, yf in FP32.  A wait that runs out sets *err and ends the CTA's work
// once the multiplications in flight are done (a second wait, bounded too).
template <int N>
__global__ void __launch_bounds__(kTcThreads, 1)
k_conv_mid_tc(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ wt,
              __nv_bfloat16 *__restrict__ y, const __nv_bfloat16 *__restrict__ gate,
              float *__restrict__ yf, long long nsamp, int mode, int *__restrict__ err,
              WaitTest wait)
{
   constexpr int NC = N == 48 ? 16 : 1;  // output channels
   extern __shared__ __align__(128) unsigned char tsm[];
   unsigned char *ws = tsm + 4 * kTcPlaneBytes;
   float *edges = reinterpret_cast<float *>(ws + kTcWBytes);
   unsigned short *tab = reinterpret_cast<unsigned short *>(edges + 2 * kTcEdge);
   unsigned short *rows = tab + kTcBox;  // cell of the slab of each output row
   unsigned long long *bar = reinterpret_cast<unsigned long long *>(rows + kTcRows);
   unsigned *tslot = reinterpret_cast<unsigned *>(bar + 3);
   const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
   for (int i = tid; i < kTcShifts * N * 2; i += kTcThreads)
      reinterpret_cast<uint4 *>(ws)[i] = reinterpret_cast<const uint4 *>(wt)[i];
   for (int i = tid; i < 4 * kTcSpan; i += kTcThreads)
      reinterpret_cast<uint4 *>(tsm)[i] = make_uint4(0u, 0u, 0u, 0u);
   box_cells(tab, tid, kTcThreads);
   if (tid == 0) {
      for (int i = 0; i < 3; ++i)  // one per half, and one that nothing completes
         asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(bar + i)) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
   }
   if (warp == 0) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                      tc_smem(tslot)),
                   "r"(2 * kTcHalf)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
   }
   asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
   __syncthreads();
   asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
   // output row r is position kTcPlane + r of the box, one input plane up
   for (int i = tid; i < kTcRows; i += kTcThreads) {
      const int e = i < kTcNz * kTcPlane ? tab[kTcPlane + i] : kNoCell;
      rows[i] = (unsigned short)(e != kNoCell ? e - S * S : kNoCell);
   }
   const unsigned tmem = *tslot;
   const unsigned sx = tc_smem(tsm), sw = tc_smem(ws), sb = tc_smem(bar);
   const long long nslab = nsamp * kTcSlabs;
   const long long first = blockIdx.x, step = gridDim.x;
   const int turns = first < nslab ? 2 * (int)((nslab - first + step - 1) / step) : 0;
   auto stage = [&](int k) {
      const long long slab = first + k * step, smp = slab / kTcSlabs;
      stage_slab(x + smp * (long long)S3 * C, (int)(slab - smp * kTcSlabs) * kTcNz, tab,
                 sx + 2u * (k & 1) * kTcPlaneBytes, sx + (2u * (k & 1) + 1u) * kTcPlaneBytes, tid,
                 kTcReaders);
   };
   if (warp < kTcReadWarps && turns) stage(0);
   // the mbarriers the readers wait on; a test's first wait is for the third's
   // first phase
   const unsigned bar_first = wait.never ? sb + 16u : sb, bar_step = wait.never ? 0u : 8u;
   bool ok = true;
   int j = 0;
   // turn j multiplies half j % 2 of the CTA's slab j / 2, reads the half
   // before, and finishes the end rows of the slab read in the two turns before
   // that; an even turn also stages the next slab
   for (; turns && j < turns + 2; ++j) {
      // the slab is staged (the tensor cores read it through the async proxy),
      // the accumulators this turn writes are read, the end rows are there
      copies_done();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      if (!__syncthreads_and(ok)) break;
      if (warp == kTcReadWarps) {
         if (lane == 0 && j < turns) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned long long bd = tc_desc(sw, 16u * N, 128u);
            const unsigned long long ad = tc_desc(
               sx + 2u * ((j >> 1) & 1) * kTcPlaneBytes +
                  16u * (unsigned)(kTcFront + kTcPlane + 128 * kTcHalfTiles * (j & 1)),
               kTcPlaneBytes, 128u);
            const unsigned d = tmem + (unsigned)(kTcHalf * (j & 1));
            // a cell is one 16-byte unit of the A address, a shift 2 N of B's
#pragma unroll
            for (int q = 0; q < kTcShifts; ++q) {
               const int off = kTcPx * (q % 3 - 1) + kTcPlane * (q / 3 - 1);
#pragma unroll
               for (int i = 0; i < kTcHalfTiles; ++i)
                  tc_mma(d + (unsigned)(N * i), ad + (long long)(off + 128 * i),
                         bd + (unsigned long long)(2 * N * q), kTcIdesc<N>, q > 0 ? 1u : 0u);
            }
            asm volatile(
               "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                  sb + 8u * (j & 1))
               : "memory");
         }
         __syncwarp();
         continue;
      }
      const bool read = j > 0 && j <= turns;
      const int kr = (j - 1) >> 1;                               // slab to read
      const int g = 4 * kTcHalfTiles * ((j - 1) & 1) + warp;     // run of 32 rows
      const unsigned at = read ? rows[32 * g + lane] : kNoCell;
      const bool put = at != kNoCell && lane > 0 && lane < 31;
      const long long cell = (first + kr * step) * kSlabCells + at;
      uint4 gg[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
      if (mode == 1 && put) {
         // the gates, loaded while the tensor cores work
         const uint4 *gp = reinterpret_cast<const uint4 *>(gate + cell * C);
         gg[0] = gp[0];
         gg[1] = gp[1];
      }
      if (read) {
         // the half before is multiplied (an mbarrier per half: one alone could be
         // a phase further already, with this turn's half)
         const long long t0 = clock64();
         while (ok && !tc_try_wait(bar_first + bar_step * ((j - 1) & 1), (unsigned)kr & 1u))
            if (clock64() - t0 > wait.limit) ok = false;
         ok = __all_sync(0xffffffffu, ok);
         if (!ok) continue;  // leaves at the barrier
      }
      if (!(j & 1) && j + 2 < turns) stage((j >> 1) + 1);
      constexpr int kArr = kTcRuns * 16;
      constexpr int NP = NC < 8 ? NC : 8;  // channels at a time
      if (read) {
         asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
         const unsigned ta = tmem + ((unsigned)(32 * (warp & 3)) << 16) +
                             (unsigned)(kTcHalf * ((j - 1) & 1) + N * (warp >> 2));
#pragma unroll
         for (int c0 = 0; c0 < NC; c0 += NP) {
            // columns of the x taps -1, 0, +1
            unsigned v0[8], v1[8], v2[8];
            tc_ld8(ta + (unsigned)c0, v0);
            if (N == 48) {
               tc_ld8(ta + 16u + (unsigned)c0, v1);
               tc_ld8(ta + 32u + (unsigned)c0, v2);
            }
            tc_ld_done();
            float o[NP], lo[NP], hi[NP];
#pragma unroll
            for (int c = 0; c < NP; ++c) {
               const float m = __uint_as_float(v0[c]), z = __uint_as_float(N == 48 ? v1[c] : v0[1]),
                           p = __uint_as_float(N == 48 ? v2[c] : v0[2]);
               lo[c] = __shfl_up_sync(0xffffffffu, m, 1) + z;
               hi[c] = __shfl_down_sync(0xffffffffu, p, 1);
               o[c] = lo[c] + hi[c];
            }
            // end rows: [0] the last row's part of the run after, [1] + [4] the
            // first row's own sum, [2] the last row's, [3] the first row's part
            // of the run before
            float *e = edges + (kr & 1) * kTcEdge + 16 * g + c0;
            if (lane == 31) {
#pragma unroll
               for (int c = 0; c < NP; ++c) {
                  e[c] = __uint_as_float(v0[c]);
                  e[2 * kArr + c] = lo[c];
               }
            } else if (lane == 0) {
#pragma unroll
               for (int c = 0; c < NP; ++c) {
                  e[kArr + c] = __uint_as_float(N == 48 ? v1[c] : v0[1]);
                  e[3 * kArr + c] = __uint_as_float(N == 48 ? v2[c] : v0[2]);
                  e[4 * kArr + c] = hi[c];
               }
            } else if (put) {
               if constexpr (N == 48) put_half(o, y + cell * C + c0, gg[c0 / 8], mode);
               else yf[cell] = o[0];
            }
         }
      }
      if ((j & 1) && j >= 3) {
         // the slab's own first and last rows are halo rows
         const int k = (j - 3) >> 1;
         const long long base = (first + k * step) * kSlabCells;
         constexpr int kParts = N == 48 ? 2 : 1;  // of 8 channels, or the one
         for (int w = tid; w < 2 * kTcRuns * kParts; w += kTcReaders) {
            const int part = w % kParts, side = w / kParts % 2, g = w / (2 * kParts);
            const unsigned at = rows[32 * g + (side ? 31 : 0)];
            if (at == kNoCell) continue;
            const long long cell = (base + at) * C + 8 * part;
            uint4 gg = make_uint4(0u, 0u, 0u, 0u);
            if (mode == 1) gg = *reinterpret_cast<const uint4 *>(gate + cell);
            const float *e = edges + (k & 1) * kTcEdge + 16 * g + 8 * part;
            float o[8];
#pragma unroll
            for (int c = 0; c < (N == 48 ? 8 : 1); ++c)
               o[c] = side ? e[2 * kArr + c] + e[3 * kArr + 16 + c]
                           : (e[c - 16] + e[kArr + c]) + e[4 * kArr + c];
            if constexpr (N == 48) put_half(o, y + cell, gg, mode);
            else yf[base + at] = o[0];
         }
      }
   }
   copies_done();
   // every accumulator read is done before the tensor memory is released
   asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
   if (!__syncthreads_and(ok) && tid == 0) {
      atomicExch(err, 1);
      // the last turn of each half may still be multiplying: its operands and
      // accumulators stay until it is done
      for (int t = j - 1; t >= 0 && t >= j - 2; --t) {
         const long long t0 = clock64();
         while (t < turns && !tc_try_wait(sb + 8u * (t & 1), (unsigned)(t >> 1) & 1u))
            if (clock64() - t0 > WaitTest().limit) break;
      }
   }
   __syncwarp();
   if (warp == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                   "r"(2 * kTcHalf)
                   : "memory");
   }
}

// Sum of the mask, in double, by the same additions every time: block sums of
// strided elements, then the last block adds the blocks in order (8 us for 256
// samples; reading the mask back and adding on the host took 4 ms).
constexpr int kSumBlocks = 256, kSumThreads = 256;

__global__ void __launch_bounds__(kSumThreads)
k_mask_sum(const float *__restrict__ mask, long long n, double *__restrict__ partial,
           unsigned *__restrict__ done, double *__restrict__ sum)
{
   __shared__ double red[kSumThreads / 32];
   __shared__ bool last;
   auto block_sum = [&](double v) {
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      __syncthreads();
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
      __syncthreads();
      v = 0.0;
      for (int w = 0; w < kSumThreads / 32; ++w) v += red[w];
      return v;
   };
   double v = 0.0;
   for (long long i = (long long)blockIdx.x * kSumThreads + threadIdx.x; i < n;
        i += (long long)kSumBlocks * kSumThreads)
      v += (double)mask[i];
   v = block_sum(v);
   if (threadIdx.x == 0) {
      partial[blockIdx.x] = v;
      __threadfence();
      last = atomicAdd(done, 1u) == kSumBlocks - 1u;
   }
   __syncthreads();
   if (!last) return;
   __threadfence();
   v = block_sum(((const volatile double *)partial)[threadIdx.x]);
   if (threadIdx.x == 0) {
      *sum = v;
      *done = 0u;
   }
}
static_assert(kSumBlocks == kSumThreads, "one block sum per thread of the last block");

// masked MSE: dy = 2/m * mask * (y - target); loss += sum(mask*(y-target)^2);
// m = *msum when given (the mask's sum on the device), else 1 / inv_m
__global__ void __launch_bounds__(256)
k_loss_grad(const float *__restrict__ y, const float *__restrict__ target,
            const float *__restrict__ mask, float inv_m, const double *__restrict__ msum,
            float *__restrict__ dy, double *__restrict__ loss, long long ncells)
{
   if (msum) inv_m = (float)(1.0 / *msum);
   double l = 0.0;
   for (long long cell = (long long)blockIdx.x * blockDim.x + threadIdx.x; cell < ncells;
        cell += (long long)gridDim.x * blockDim.x) {
      const float d = (y[cell] - target[cell]) * mask[cell];
      dy[cell] = 2.f * inv_m * d;
      l += (double)d * (double)d;
   }
   for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
   __shared__ double red[8];
   if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = l;
   __syncthreads();
   if (threadIdx.x == 0) {
      for (int w = 1; w < 8; ++w) l += red[w];
      if (l != 0.0) atomicAdd(loss, l);
   }
}

// ---------------------------------------------------------------------------
// one channel <-> 16 channels on mma.sync (m16n8k16), slab by slab of kTcNz
// z-planes.  The one-channel field is staged with a zero halo in shared memory
// as NSP BF16 numbers per cell whose sum it is: NSP = 1 rounds (layer 1's
// input), NSP = 3 holds an FP32 value whole (h = bf16(v), then the same of the
// remainder twice: 3 x 8 bits; from about 2^-110 in magnitude up, below which
// the last parts underflow), so products and sums are those of the FP32 field.  The 27 taps (padded to 32 by zero weights or dropped results) are
// the K dimension of the convolution and the N dimension of the weight
// gradient; each lane gathers its cells' tap values from the slab (16-bit
// loads).  For 256 samples (ncu): layer 1 28 us, layer 4's data gradient 57,
// the weight gradients 42 and 64; on the FP32 cores, bound by loads and
// multiply-adds, 113, 80, 326 and 326.
// ---------------------------------------------------------------------------
constexpr int kSlabSteps = (kSlabCells + 15) / 16;        // runs of 16 cells
constexpr int kSmWarps = 8;
constexpr int kSmThreads = 32 * kSmWarps;

constexpr float kBf16Max = 3.38953139e38f, kFloatMax = 3.40282347e38f;

template <int NSP>
__device__ __forceinline__ void split_bf16(float v, __nv_bfloat16 *o)
{
   if (NSP == 1) {
      o[0] = __float2bfloat16_rn(v);
      return;
   }
#pragma unroll
   for (int k = 0; k < NSP; ++k) {
      // a finite value does not round up to infinity
      const float c = fabsf(v) <= kFloatMax ? fminf(fmaxf(v, -kBf16Max), kBf16Max) : v;
      o[k] = __float2bfloat16_rn(c);
      const float h = __bfloat162float(o[k]);
      v = fabsf(h) <= kBf16Max ? v - h : 0.f;  // an infinity or NaN is its first part alone
   }
}

// padded box index of each cell of a slab (cells past the last: cell 0's)
__device__ __forceinline__ void slab_index(unsigned short *at, int tid)
{
   for (int i = tid; i < 16 * kSlabSteps; i += kSmThreads) {
      const int c = i < kSlabCells ? i : 0;
      const int z = c / (S * S), r = c - z * S * S;
      at[i] = (unsigned short)(kTcFront + (z + 1) * kTcPlane + (r / S + 1) * kTcPx + r % S + 1);
   }
}

template <int NSP>
__device__ __forceinline__ void stage_field(const float *v, int z0, const unsigned short *tab,
                                            __nv_bfloat16 (*sv)[kTcSpan], int tid)
{
   // four cells of a thread in flight
#pragma unroll 4
   for (int i = tid; i < kTcBox; i += kSmThreads) {
      const int cell = box_cell(tab, i, z0);
      __nv_bfloat16 o[NSP];
      split_bf16<NSP>(cell >= 0 ? v[cell] : 0.f, o);
#pragma unroll
      for (int k = 0; k < NSP; ++k) sv[k][kTcFront + i] = o[k];
   }
}

__device__ __forceinline__ uint32_t pair(const __nv_bfloat16 *sv, int i, int j)
{
   const unsigned short *p = reinterpret_cast<const unsigned short *>(sv);
   return (uint32_t)p[i] | ((uint32_t)p[j] << 16);
}

// out[cell][c] = sum_t w[t][c] v[cell + DIR off_t], DIR = +1: layer 1, ReLU; -1:
// the data gradient through layer 4, gated by gate > 0.  w: FP32, used rounded
// to BF16.  Column n of the two N tiles is channel 4 (n / 2) + n % 2 (+ 2 in
// the second), so a lane holds four consecutive channels of its rows.
template <int NSP, int DIR>
__global__ void __launch_bounds__(kSmThreads)
k_conv_one(const float *__restrict__ v, const float *__restrict__ w, __nv_bfloat16 *__restrict__ out,
           const __nv_bfloat16 *__restrict__ gate, long long nsamp)
{
   __shared__ __nv_bfloat16 sv[NSP][kTcSpan];
   __shared__ unsigned short at[16 * kSlabSteps], tab[kTcBox];
   const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
   for (int i = tid; i < NSP * kTcSpan; i += kSmThreads) sv[0][i] = __float2bfloat16_rn(0.f);
   slab_index(at, tid);
   box_cells(tab, tid, kSmThreads);
   // B: taps x channels, and the lane's tap offsets
   uint32_t b[2][2][2];
   int off[2][4];
#pragma unroll
   for (int ks = 0; ks < 2; ++ks)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
         const int t0 = 16 * ks + 2 * q + 8 * h;
#pragma unroll
         for (int e = 0; e < 2; ++e) {
            const int t = t0 + e;
            off[ks][2 * h + e] =
               t < T ? DIR * (tap_dx(t) + kTcPx * tap_dy(t) + kTcPlane * tap_dz(t)) : 0;
         }
#pragma unroll
         for (int j = 0; j < 2; ++j) {
            const int c = 4 * (g >> 1) + (g & 1) + 2 * j;
            const __nv_bfloat162 p = __floats2bfloat162_rn(t0 < T ? w[t0 * C + c] : 0.f,
                                                           t0 + 1 < T ? w[(t0 + 1) * C + c] : 0.f);
            b[ks][j][h] = *reinterpret_cast<const uint32_t *>(&p);
         }
      }
   // the taps from 27 on (of this lane: 24 + 2 q, 25 + 2 q) read the zero at index
   // 0: a cell's own value in their place, times the weight 0, would make an
   // infinite one a NaN
   const int in0 = 24 + 2 * q < T ? -1 : 0, in1 = 25 + 2 * q < T ? -1 : 0;
   const long long nslab = nsamp * kTcSlabs;
   for (long long slab = blockIdx.x; slab < nslab; slab += gridDim.x) {
      const long long smp = slab / kTcSlabs;
      const int z0 = (int)(slab - smp * kTcSlabs) * kTcNz;
      __syncthreads();
      stage_field<NSP>(v + smp * S3, z0, tab, sv, tid);
      __syncthreads();
      const long long base = smp * S3 + (long long)z0 * S * S;
      for (int st = warp; st < kSlabSteps; st += kSmWarps) {
         const int r0 = 16 * st + g, r1 = r0 + 8;
         const int p0 = at[r0], p1 = at[r1];
         const int q0[2][2] = {{p0, p0}, {p0 & in0, p0 & in1}};  // of the upper taps of a step
         const int q1[2][2] = {{p1, p1}, {p1 & in0, p1 & in1}};
         float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
         for (int k = 0; k < NSP; ++k)
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
               const uint32_t a[4] = {pair(sv[k], p0 + off[ks][0], p0 + off[ks][1]),
                                      pair(sv[k], p1 + off[ks][0], p1 + off[ks][1]),
                                      pair(sv[k], q0[ks][0] + off[ks][2], q0[ks][1] + off[ks][3]),
                                      pair(sv[k], q1[ks][0] + off[ks][2], q1[ks][1] + off[ks][3])};
               mma_bf16(d[0], a, b[ks][0][0], b[ks][0][1]);
               mma_bf16(d[1], a, b[ks][1][0], b[ks][1][1]);
            }
#pragma unroll
         for (int h = 0; h < 2; ++h) {
            const int r = h ? r1 : r0;
            if (r >= kSlabCells) continue;
            const long long o = (base + r) * C + 4 * q;
            float f[4] = {d[0][2 * h], d[0][2 * h + 1], d[1][2 * h], d[1][2 * h + 1]};
            if (DIR > 0) {
#pragma unroll
               for (int c = 0; c < 4; ++c) f[c] = fmaxf(f[c], 0.f);
            } else {
               const uint2 gg = *reinterpret_cast<const uint2 *>(gate + o);
               const __nv_bfloat16 *gp = reinterpret_cast<const __nv_bfloat16 *>(&gg);
#pragma unroll
               for (int c = 0; c < 4; ++c) f[c] = __bfloat162float(gp[c]) > 0.f ? f[c] : 0.f;
            }
            const __nv_bfloat162 o0 = __floats2bfloat162_rn(f[0], f[1]),
                                 o1 = __floats2bfloat162_rn(f[2], f[3]);
            *reinterpret_cast<uint2 *>(out + o) =
               make_uint2(*reinterpret_cast<const uint32_t *>(&o0), *reinterpret_cast<const uint32_t *>(&o1));
         }
      }
   }
}

__device__ __forceinline__ void ldm_x4_trans(unsigned addr, uint32_t *r)
{
   asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                : "r"(addr));
}

// the 16-channel cells of a slab, channel halves in planes of 16 bytes a cell;
// copies left in flight
__device__ __forceinline__ void stage_cells(const __nv_bfloat16 *src, unsigned p0, unsigned p1,
                                            int tid, int nthr)
{
   for (int i = tid; i < 2 * kSlabCells; i += nthr)
      copy16(((i & 1) ? p1 : p0) + 16u * (i >> 1), src + (size_t)i * 8, true);
}

// dw[t][c] += sum over cells of a[cell][c] v[cell + DIR off_t]: layer 1 (a its
// output's gradient, v the input, DIR = +1) and layer 4 (a its input, v the
// output's gradient, DIR = -1).  A = a^T (16 channels x 16 cells, ldmatrix),
// B = 16 cells x 8 taps gathered from the slab; each warp sums its runs of
// cells in registers, the block adds its warps and then once to dw.
template <int NSP>
constexpr int kOneSmem = 16 * 2 * 16 * kSlabSteps + 4 * 32 * C + 2 * (16 * kSlabSteps + kTcBox + NSP * kTcSpan);

template <int NSP, int DIR>
__global__ void __launch_bounds__(kSmThreads)
k_weight_one(const __nv_bfloat16 *__restrict__ a, const float *__restrict__ v,
             float *__restrict__ dw, long long nsamp)
{
   extern __shared__ __align__(128) unsigned char osm[];
   uint4 (*sa)[16 * kSlabSteps] = reinterpret_cast<uint4 (*)[16 * kSlabSteps]>(osm);
   float *sum = reinterpret_cast<float *>(osm + sizeof(uint4) * 2 * 16 * kSlabSteps);
   unsigned short *at = reinterpret_cast<unsigned short *>(sum + 32 * C);
   unsigned short *tab = at + 16 * kSlabSteps;
   __nv_bfloat16 (*sv)[kTcSpan] = reinterpret_cast<__nv_bfloat16 (*)[kTcSpan]>(tab + kTcBox);
   const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
   for (int i = tid; i < NSP * kTcSpan; i += kSmThreads) sv[0][i] = __float2bfloat16_rn(0.f);
   for (int i = tid; i < 2 * 16 * kSlabSteps; i += kSmThreads) sa[0][i] = make_uint4(0u, 0u, 0u, 0u);
   for (int i = tid; i < 32 * C; i += kSmThreads) sum[i] = 0.f;
   slab_index(at, tid);
   box_cells(tab, tid, kSmThreads);
   int off[4];
#pragma unroll
   for (int j = 0; j < 4; ++j) {
      const int t = 8 * j + g;
      off[j] = t < T ? DIR * (tap_dx(t) + kTcPx * tap_dy(t) + kTcPlane * tap_dz(t)) : 0;
   }
   const unsigned a0 = tc_smem(sa[0]), a1 = tc_smem(sa[1]);
   const int mrow = lane & 7, mj = lane >> 3;
   float acc[4][4];
#pragma unroll
   for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[j][c] = 0.f;
   const long long nslab = nsamp * kTcSlabs;
   for (long long slab = blockIdx.x; slab < nslab; slab += gridDim.x) {
      const long long smp = slab / kTcSlabs;
      const int z0 = (int)(slab - smp * kTcSlabs) * kTcNz;
      __syncthreads();
      stage_cells(a + (smp * S3 + (long long)z0 * S * S) * C, a0, a1, tid, kSmThreads);
      stage_field<NSP>(v + smp * S3, z0, tab, sv, tid);
      copies_done();
      __syncthreads();
      for (int st = warp; st < kSlabSteps; st += kSmWarps) {
         // matrices (c 0-7, cells +0), (c 8-15, +0), (c 0-7, +8), (c 8-15, +8)
         uint32_t av[4];
         ldm_x4_trans(((mj & 1) ? a1 : a0) + 16u * (unsigned)(16 * st + 8 * (mj >> 1) + mrow), av);
         const unsigned short *ap = at + 16 * st + 2 * q;
         const int c0 = ap[0], c1 = ap[1], c2 = ap[8], c3 = ap[9];
#pragma unroll
         for (int k = 0; k < NSP; ++k)
#pragma unroll
            for (int j = 0; j < 4; ++j)
               mma_bf16(acc[j], av, pair(sv[k], c0 + off[j], c1 + off[j]),
                        pair(sv[k], c2 + off[j], c3 + off[j]));
      }
   }
   // rows g, g + 8 are channels, columns 2q, 2q + 1 taps
#pragma unroll
   for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c)
         atomicAdd(&sum[(8 * j + 2 * q + (c & 1)) * C + g + 8 * (c >> 1)], acc[j][c]);
   __syncthreads();
   for (int i = tid; i < T * C; i += kSmThreads) atomicAdd(&dw[i], sum[i]);
}

// weight gradient of a 16 -> 16 layer: dw[t][ci][co] += sum over cells of
// x[cell + off_t][ci] * dy[cell][co].  The slab's input box (zero halo) and
// its gradient cells are staged in shared memory in channel planes of 16 bytes
// per cell; warp w owns taps 3w .. 3w + 2 (one x-row of taps) and multiplies
// A = x^T (16 in-channels x 16 cells, ldmatrix.trans at the tap's shifted
// rows) by B = dy (16 cells x 8 out-channels, ldmatrix.trans) with
// mma.sync m16n8k16 over every 16 cells of the slab.  The tensor cores'
// tcgen05 form needs M >= 64 output rows, and with 16 x 16 outputs per tap
// and the tap as a row shift no operand layout gives that.  Each CTA sums
// its slabs in registers and adds them once.  Bound by the latency of
// ldmatrix (36 per 16 cells over the nine warps): 104 us for 256 samples, 118
// with the halo positions among the 16-cell steps and copies through registers.
constexpr int kWgWarps = T / 3;                      // 9 warps, 3 taps each
constexpr int kWgThreads = 32 * kWgWarps;
constexpr int kWgSmem = 2 * kTcPlaneBytes + 2 * 16 * kSlabSteps * 16 + 16 * kSlabSteps * 2 + kTcBox * 2;
static_assert(T % 3 == 0, "three taps per warp");
static_assert(2 * kWgSmem <= 227 * 1024, "two CTAs per SM");

__global__ void __launch_bounds__(kWgThreads)
k_bwd_weight_mid(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ dy,
                 float *__restrict__ dw, long long nsamp)
{
   extern __shared__ __align__(128) unsigned char wsm[];
   const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
   constexpr int kFirst = 2 * kTcPlaneBytes, kCells = 16 * kSlabSteps;
   for (int i = tid; i < (kFirst + 2 * kCells * 16) / 16; i += kWgThreads)
      reinterpret_cast<uint4 *>(wsm)[i] = make_uint4(0u, 0u, 0u, 0u);
   unsigned short *at = reinterpret_cast<unsigned short *>(wsm + kFirst + 2 * kCells * 16);
   if (tid < kSmThreads) slab_index(at, tid);
   unsigned short *tab = at + kCells;
   box_cells(tab, tid, kWgThreads);
   const unsigned sx0 = tc_smem(wsm), sx1 = sx0 + kTcPlaneBytes;
   const unsigned sg0 = sx0 + kFirst, sg1 = sg0 + 16u * kCells;
   // ldmatrix.x4: lanes 8j .. 8j + 7 give the rows of matrix j
   const int mrow = lane & 7, mj = lane >> 3;
   float acc[3][2][4];
#pragma unroll
   for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
         for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.f;
   int off[3];
#pragma unroll
   for (int a = 0; a < 3; ++a) {
      const int t = 3 * warp + a;
      off[a] = 16 * (tap_dx(t) + kTcPx * tap_dy(t) + kTcPlane * tap_dz(t));
   }
   const unsigned sxm = (mj & 1) ? sx1 : sx0, sgm = (mj >> 1) ? sg1 : sg0;
   const long long nslab = nsamp * kTcSlabs;
   for (long long slab = blockIdx.x; slab < nslab; slab += gridDim.x) {
      const long long smp = slab / kTcSlabs;
      const int z0 = (int)(slab - smp * kTcSlabs) * kTcNz;
      __syncthreads();  // the previous slab's reads are done
      stage_slab(x + smp * (long long)S3 * C, z0, tab, sx0, sx1, tid, kWgThreads);
      stage_cells(dy + (smp * S3 + (long long)z0 * S * S) * C, sg0, sg1, tid, kWgThreads);
      copies_done();
      __syncthreads();
#pragma unroll 2
      for (int k0 = 0; k0 < kCells; k0 += 16) {
         // B: dy cells k0 .. k0 + 15; matrices (co 0-7, cells +0), (co 0-7,
         // +8), (co 8-15, +0), (co 8-15, +8)
         uint32_t b[4];
         ldm_x4_trans(sgm + 16u * (unsigned)(k0 + 8 * (mj & 1) + mrow), b);
         const unsigned row = sxm + 16u * at[k0 + 8 * (mj >> 1) + mrow];
#pragma unroll
         for (int a = 0; a < 3; ++a) {
            // A = x^T at the tap's rows: matrices (ci 0-7, cells +0),
            // (ci 8-15, +0), (ci 0-7, +8), (ci 8-15, +8)
            uint32_t av[4];
            ldm_x4_trans(row + off[a], av);
            mma_bf16(acc[a][0], av, b[0], b[1]);
            mma_bf16(acc[a][1], av, b[2], b[3]);
         }
      }
   }
   const int g = lane >> 2, q = lane & 3;
#pragma unroll
   for (int a = 0; a < 3; ++a) {
      const int t = 3 * warp + a;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
         const int co = 8 * j + 2 * q;
         atomicAdd(&dw[(t * C + g) * C + co], acc[a][j][0]);
         atomicAdd(&dw[(t * C + g) * C + co + 1], acc[a][j][1]);
         atomicAdd(&dw[(t * C + g + 8) * C + co], acc[a][j][2]);
         atomicAdd(&dw[(t * C + g + 8) * C + co + 1], acc[a][j][3]);
      }
   }
}

// BF16 B operands of k_conv_mid_tc, [(y, z) shift][input-channel half][N][8]:
// 16 -> 16 weights (N = 48, column 16 x-tap + output channel), forward and
// for the data gradient (taps reversed, channels exchanged)
__global__ void k_pack_mid(const float *__restrict__ w, __nv_bfloat16 *__restrict__ wf,
                           __nv_bfloat16 *__restrict__ wd)
{
   const int i = blockIdx.x * blockDim.x + threadIdx.x;
   if (i >= T * C * C) return;
   const int t = i / (C * C), ci = (i / C) % C, co = i % C;
   const __nv_bfloat16 v = __float2bfloat16_rn(w[i]);
   auto at = [](int tap, int in, int out) {
      return (((tap / 3) * 2 + in / 8) * 48 + 16 * (tap % 3) + out) * 8 + in % 8;
   };
   wf[at(t, ci, co)] = v;
   wd[at(T - 1 - t, co, ci)] = v;
}

// the 16 -> 1 weights as such operands with N = 16: column = x tap, columns 3
// and up zero
__global__ void k_pack_out(const float *__restrict__ w4, __nv_bfloat16 *__restrict__ wo)
{
   const int i = blockIdx.x * blockDim.x + threadIdx.x;
   if (i >= kTcShifts * C * C) return;
   const int q = i / (C * C), half = (i / (8 * C)) % 2, n = (i / 8) % C, j = i % 8;
   wo[i] = __float2bfloat16_rn(n < 3 ? w4[(3 * q + n) * C + 8 * half + j] : 0.f);
}

__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2)
{
   const int i = blockIdx.x * blockDim.x + threadIdx.x;
   if (i >= n) return;
   const float gi = g[i];
   const float mi = b1 * m[i] + (1.f - b1) * gi;
   const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
   m[i] = mi;
   v[i] = vi;
   w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

thread_local std::string t_cnn_error;

}  // namespace

// ---------------------------------------------------------------------------
// network object
// ---------------------------------------------------------------------------

struct fac_cnn {
   int device = 0;
   int max_batch = 0;
   cudaStream_t stream = nullptr;
   // FP32 masters, Adam moments and gradients: w1 [27*16], w2, w3 [27*16*16], w4 [27*16]
   float *w[4] = {nullptr}, *gw[4] = {nullptr}, *m[4] = {nullptr}, *v[4] = {nullptr};
   // gradients, loss and mask sum lie in one block, read back by one copy;
   // the error flag follows them
   float *grads = nullptr;
   unsigned char *host = nullptr;        // pinned, as large
   __nv_bfloat16 *wf[2] = {nullptr}, *wd[2] = {nullptr};  // layers 2, 3
   __nv_bfloat16 *wo = nullptr;          // layer 4
   __nv_bfloat16 *a[3] = {nullptr}, *d[3] = {nullptr};
   float *y = nullptr, *dy = nullptr;
   double *loss = nullptr, *msum = nullptr;
   int *kerr = nullptr;                  // set by a tensor-core wait that ran out
   double *partial = nullptr;            // block sums of k_mask_sum
   unsigned *done = nullptr;
   WaitTest wait_test;
   int sms = 0;
   int steps = 0;
   std::vector<void *> allocs;
};

namespace {

const int kSizes[4] = {T * C, T * C * C, T * C * C, T * C};
constexpr size_t kGradFloats = 2 * T * C + 2 * T * C * C;
constexpr size_t kGradBytes = kGradFloats * 4 + 2 * sizeof(double);  // with loss and mask sum
constexpr size_t kBackBytes = kGradBytes + sizeof(int);
static_assert(kGradFloats % 2 == 0, "loss aligned");

#define CNN_CHECK(x)                                                                \
   do {                                                                             \
      cudaError_t _e = (x);                                                         \
      if (_e != cudaSuccess) {                                                      \
         t_cnn_error = std::string(#x) + ": " + cudaGetErrorString(_e);             \
         return FAC_ERR_CUDA;                                                       \
      }                                                                             \
   } while (0)

template <class P>
int dalloc(fac_cnn *n, P **p, size_t bytes)
{
   cudaError_t e = cudaMalloc((void **)p, bytes);
   if (e != cudaSuccess) {
      t_cnn_error = std::string("cudaMalloc: ") + cudaGetErrorString(e);
      return FAC_ERR_NOMEM;
   }
   n->allocs.push_back((void *)*p);
   return FAC_OK;
}

int pack(fac_cnn *n)
{
   for (int l = 0; l < 2; ++l) {
      k_pack_mid<<<(T * C * C + 255) / 256, 256, 0, n->stream>>>(n->w[l + 1], n->wf[l], n->wd[l]);
   }
   k_pack_out<<<(kTcShifts * C * C + 255) / 256, 256, 0, n->stream>>>(n->w[3], n->wo);
   samrai_b200::add_kernel_launches(3);
   CNN_CHECK(cudaGetLastError());
   return FAC_OK;
}

unsigned slab_grid(const fac_cnn *n, long long nsamp, int per_sm)
{
   return (unsigned)std::min<long long>(nsamp * kTcSlabs, (long long)per_sm * n->sms);
}

void conv_mid(fac_cnn *n, const __nv_bfloat16 *x, const __nv_bfloat16 *wt, __nv_bfloat16 *y,
              const __nv_bfloat16 *gate, long long nsamp, int mode, cudaStream_t st)
{
   k_conv_mid_tc<48><<<slab_grid(n, nsamp, 1), kTcThreads, kTcSmem, st>>>(x, wt, y, gate, nullptr,
                                                                         nsamp, mode, n->kerr, n->wait_test);
}

void weight_mid(fac_cnn *n, const __nv_bfloat16 *x, const __nv_bfloat16 *dy, float *dw,
                long long nsamp)
{
   k_bwd_weight_mid<<<slab_grid(n, nsamp, 2), kWgThreads, kWgSmem, n->stream>>>(x, dy, dw, nsamp);
}

// the block's first `bytes` and the device error flag, after the stream has
// drained
int read_back(fac_cnn *n, bool all)
{
   const size_t from = all ? 0 : kGradBytes;
   CNN_CHECK(cudaMemcpyAsync(n->host + from, reinterpret_cast<unsigned char *>(n->grads) + from,
                             kBackBytes - from, cudaMemcpyDeviceToHost, n->stream));
   CNN_CHECK(cudaStreamSynchronize(n->stream));
   int e = 0;
   std::memcpy(&e, n->host + kGradBytes, sizeof(int));
   if (e) {
      t_cnn_error = "a tensor-core wait ran out (k_conv_mid_tc)";
      return FAC_ERR_DEVICE;
   }
   return FAC_OK;
}

int forward_on(fac_cnn *n, const float *x, long long nsamp, cudaStream_t st, float *y)
{
   k_conv_one<1, 1><<<slab_grid(n, nsamp, 4), kSmThreads, 0, st>>>(x, n->w[0], n->a[0], nullptr,
                                                                   nsamp);
   conv_mid(n, n->a[0], n->wf[0], n->a[1], nullptr, nsamp, 0, st);
   conv_mid(n, n->a[1], n->wf[1], n->a[2], nullptr, nsamp, 0, st);
   k_conv_mid_tc<16><<<slab_grid(n, nsamp, 1), kTcThreads, kTcSmem, st>>>(
      n->a[2], n->wo, nullptr, nullptr, y, nsamp, 2, n->kerr, n->wait_test);
   samrai_b200::add_kernel_launches(4);
   CNN_CHECK(cudaGetLastError());
   return FAC_OK;
}

int forward(fac_cnn *n, const float *x, long long nsamp, float *y)
{
   return forward_on(n, x, nsamp, n->stream, y);
}

// mask_sum > 0: the mask's sum; else it is formed on the device
int backward(fac_cnn *n, const float *x, const float *target, const float *mask, long long nsamp,
             double mask_sum)
{
   const long long cells = nsamp * S3;
   CNN_CHECK(cudaMemsetAsync(n->grads, 0, kGradBytes, n->stream));
   const bool sum_here = !(mask_sum > 0);
   if (sum_here)
      k_mask_sum<<<kSumBlocks, kSumThreads, 0, n->stream>>>(mask, cells, n->partial, n->done, n->msum);
   const unsigned lb = (unsigned)std::min<long long>((cells + 255) / 256, 8LL * n->sms);
   k_loss_grad<<<lb, 256, 0, n->stream>>>(n->y, target, mask,
                                          sum_here ? 0.f : (float)(1.0 / mask_sum),
                                          sum_here ? n->msum : nullptr, n->dy, n->loss, cells);
   const unsigned sg = slab_grid(n, nsamp, 2);
   k_weight_one<3, -1><<<sg, kSmThreads, kOneSmem<3>, n->stream>>>(n->a[2], n->dy, n->gw[3], nsamp);
   k_conv_one<3, -1><<<slab_grid(n, nsamp, 4), kSmThreads, 0, n->stream>>>(n->dy, n->w[3], n->d[2],
                                                                           n->a[2], nsamp);
   weight_mid(n, n->a[1], n->d[2], n->gw[2], nsamp);
   conv_mid(n, n->d[2], n->wd[1], n->d[1], n->a[1], nsamp, 1, n->stream);
   weight_mid(n, n->a[0], n->d[1], n->gw[1], nsamp);
   conv_mid(n, n->d[1], n->wd[0], n->d[0], n->a[0], nsamp, 1, n->stream);
   k_weight_one<1, 1><<<sg, kSmThreads, kOneSmem<1>, n->stream>>>(n->d[0], x, n->gw[0], nsamp);
   samrai_b200::add_kernel_launches(8 + (sum_here ? 1 : 0));
   CNN_CHECK(cudaGetLastError());
   return FAC_OK;
}

int check_batch(fac_cnn *n, long long nsamp)
{
   if (!n) {
      t_cnn_error = "null network";
      return FAC_ERR_ARG;
   }
   if (nsamp < 1 || nsamp > n->max_batch) {
      t_cnn_error = "batch size out of range";
      return FAC_ERR_ARG;
   }
   return FAC_OK;
}

}  // namespace

namespace samrai_b200 {
// Forward pass on the caller's stream (used inside the FAC cycle); *y points
// at the network's output buffer (nsamp * S^3 floats).
int cnn_forward_on_stream(fac_cnn *n, const float *x, long long nsamp, cudaStream_t st,
                          const float **y)
{
   int rc = check_batch(n, nsamp);
   if (rc) return rc;
   rc = forward_on(n, x, nsamp, st, n->y);
   if (y) *y = n->y;
   return rc;
}
int cnn_max_batch(const fac_cnn *n) { return n ? n->max_batch : 0; }
int cnn_device(const fac_cnn *n) { return n ? n->device : -1; }
}  // namespace samrai_b200

extern "C" {

const char *fac_cnn_last_error(void) { return t_cnn_error.c_str(); }

int fac_cnn_create(fac_cnn **out, int device, int max_batch, unsigned long long seed)
{
   if (!out || max_batch < 1) {
      t_cnn_error = "bad arguments";
      return FAC_ERR_ARG;
   }
   CNN_CHECK(cudaSetDevice(device));
   fac_cnn *n = new fac_cnn();
   n->device = device;
   n->max_batch = max_batch;
   int rc = FAC_OK;
   auto fail = [&](int r) {
      for (void *p : n->allocs) cudaFree(p);
      if (n->host) cudaFreeHost(n->host);
      delete n;
      return r;
   };
   if (cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking) != cudaSuccess)
      return fail(FAC_ERR_CUDA);
   const long long cells = (long long)max_batch * S3;
   for (int l = 0; l < 4; ++l) {
      if ((rc = dalloc(n, &n->w[l], kSizes[l] * sizeof(float))) ||
          (rc = dalloc(n, &n->m[l], kSizes[l] * sizeof(float))) ||
          (rc = dalloc(n, &n->v[l], kSizes[l] * sizeof(float))))
         return fail(rc);
   }
   if ((rc = dalloc(n, &n->wo, kTcShifts * C * C * 2)) || (rc = dalloc(n, &n->grads, kBackBytes)) ||
       (rc = dalloc(n, &n->partial, kSumBlocks * sizeof(double))) ||
       (rc = dalloc(n, &n->done, sizeof(unsigned))))
      return fail(rc);
   if (samrai_b200::pinned_alloc((void **)&n->host, kBackBytes) != cudaSuccess) {
      n->host = nullptr;
      t_cnn_error = "no page-locked host memory";
      return fail(FAC_ERR_NOMEM);
   }
   for (size_t l = 0, at = 0; l < 4; at += kSizes[l++]) n->gw[l] = n->grads + at;
   n->loss = reinterpret_cast<double *>(n->grads + kGradFloats);
   n->msum = n->loss + 1;
   n->kerr = reinterpret_cast<int *>(n->msum + 1);
   for (int l = 0; l < 2; ++l)
      if ((rc = dalloc(n, &n->wf[l], T * C * C * 2)) || (rc = dalloc(n, &n->wd[l], T * C * C * 2)))
         return fail(rc);
   for (int l = 0; l < 3; ++l)
      if ((rc = dalloc(n, &n->a[l], cells * C * 2)) || (rc = dalloc(n, &n->d[l], cells * C * 2)))
         return fail(rc);
   if ((rc = dalloc(n, &n->y, cells * 4)) || (rc = dalloc(n, &n->dy, cells * 4))) return fail(rc);
   if (cudaDeviceGetAttribute(&n->sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
       cudaFuncSetAttribute(k_conv_mid_tc<48>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            kTcSmem) != cudaSuccess ||
       cudaFuncSetAttribute(k_conv_mid_tc<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            kTcSmem) != cudaSuccess ||
       cudaFuncSetAttribute(k_weight_one<3, -1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            kOneSmem<3>) != cudaSuccess ||
       cudaFuncSetAttribute(k_bwd_weight_mid, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            kWgSmem) != cudaSuccess)
      return fail(FAC_ERR_CUDA);
   if (cudaMemsetAsync(n->kerr, 0, sizeof(int), n->stream) != cudaSuccess ||
       cudaMemsetAsync(n->done, 0, sizeof(unsigned), n->stream) != cudaSuccess)
      return fail(FAC_ERR_CUDA);
   // He initialisation from a seeded host generator (splitmix64 + Box-Muller)
   unsigned long long st = seed * 0x9E3779B97F4A7C15ull + 1;
   auto next = [&]() {
      st += 0x9E3779B97F4A7C15ull;
      unsigned long long z = st;
      z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
      z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
      return ((z ^ (z >> 31)) >> 11) * (1.0 / 9007199254740992.0);
   };
   const int fan_in[4] = {T, T * C, T * C, T * C};
   for (int l = 0; l < 4; ++l) {
      std::vector<float> h(kSizes[l]);
      const double sd = std::sqrt(2.0 / fan_in[l]);
      for (auto &x : h) {
         const double u1 = next() + 1e-300, u2 = next();
         x = (float)(sd * std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2));
      }
      if (l == 3)
         for (auto &x : h) x *= 0.1f;  // start close to a zero correction
      CNN_CHECK(cudaMemcpyAsync(n->w[l], h.data(), kSizes[l] * 4, cudaMemcpyHostToDevice,
                                n->stream));
      CNN_CHECK(cudaMemsetAsync(n->m[l], 0, kSizes[l] * 4, n->stream));
      CNN_CHECK(cudaMemsetAsync(n->v[l], 0, kSizes[l] * 4, n->stream));
   }
   if ((rc = pack(n))) return fail(rc);
   CNN_CHECK(cudaStreamSynchronize(n->stream));
   *out = n;
   return FAC_OK;
}

int fac_cnn_destroy(fac_cnn *n)
{
   if (!n) return FAC_OK;
   cudaSetDevice(n->device);
   cudaStreamSynchronize(n->stream);
   for (void *p : n->allocs) cudaFree(p);
   cudaFreeHost(n->host);
   cudaStreamDestroy(n->stream);
   delete n;
   return FAC_OK;
}

int fac_cnn_set_wait_test(fac_cnn *n, long long limit_cycles, int never)
{
   if (!n || limit_cycles < 1 || never < 0 || never > 1) {
      t_cnn_error = "bad wait test";
      return FAC_ERR_ARG;
   }
   n->wait_test.limit = limit_cycles;
   n->wait_test.never = never;
   CNN_CHECK(cudaMemsetAsync(n->kerr, 0, sizeof(int), n->stream));
   CNN_CHECK(cudaStreamSynchronize(n->stream));
   return FAC_OK;
}

int fac_cnn_set_weights(fac_cnn *n, const float *w1, const float *w2, const float *w3,
                        const float *w4)
{
   if (!n || !w1 || !w2 || !w3 || !w4) {
      t_cnn_error = "null argument";
      return FAC_ERR_ARG;
   }
   const float *src[4] = {w1, w2, w3, w4};
   for (int l = 0; l < 4; ++l)
      CNN_CHECK(cudaMemcpyAsync(n->w[l], src[l], kSizes[l] * 4, cudaMemcpyHostToDevice,
                                n->stream));
   int rc = pack(n);
   if (rc) return rc;
   CNN_CHECK(cudaStreamSynchronize(n->stream));
   return FAC_OK;
}

int fac_cnn_get_weights(fac_cnn *n, float *w1, float *w2, float *w3, float *w4)
{
   if (!n || !w1 || !w2 || !w3 || !w4) {
      t_cnn_error = "null argument";
      return FAC_ERR_ARG;
   }
   float *dst[4] = {w1, w2, w3, w4};
   for (int l = 0; l < 4; ++l)
      CNN_CHECK(cudaMemcpyAsync(dst[l], n->w[l], kSizes[l] * 4, cudaMemcpyDeviceToHost,
                                n->stream));
   CNN_CHECK(cudaStreamSynchronize(n->stream));
   return FAC_OK;
}

int fac_cnn_forward(fac_cnn *n, const float *x, long long nsamp, float *y)
{
   int rc = check_batch(n, nsamp);
   if (rc) return rc;
   if (!x || !y) {
      t_cnn_error = "null argument";
      return FAC_ERR_ARG;
   }
   if ((rc = forward(n, x, nsamp, y))) return rc;
   return read_back(n, false);
}

int fac_cnn_gradients(fac_cnn *n, const float *x, const float *target, const float *mask,
                      long long nsamp, double *loss, float *g1, float *g2, float *g3, float *g4)
{
   int rc = check_batch(n, nsamp);
   if (rc) return rc;
   if (!x || !target || !mask) {
      t_cnn_error = "null argument";
      return FAC_ERR_ARG;
   }
   if ((rc = forward(n, x, nsamp, n->y))) return rc;
   if ((rc = backward(n, x, target, mask, nsamp, 0.0))) return rc;
   if ((rc = read_back(n, true))) return rc;
   double l[2];  // loss sum and mask sum
   std::memcpy(l, n->host + kGradFloats * 4, sizeof(l));
   if (l[1] <= 0) {
      t_cnn_error = "empty mask";
      return FAC_ERR_ARG;
   }
   float *dst[4] = {g1, g2, g3, g4};
   size_t at = 0;
   for (int k = 0; k < 4; at += kSizes[k++] * sizeof(float))
      if (dst[k]) std::memcpy(dst[k], n->host + at, kSizes[k] * sizeof(float));
   if (loss) *loss = l[0] / l[1];
   return FAC_OK;
}

int fac_cnn_train_step(fac_cnn *n, const float *x, const float *target, const float *mask,
                       long long nsamp, double mask_sum, float lr, double *loss)
{
   int rc = check_batch(n, nsamp);
   if (rc) return rc;
   if (!x || !target || !mask || !(mask_sum > 0)) {
      t_cnn_error = "bad arguments";
      return FAC_ERR_ARG;
   }
   if ((rc = forward(n, x, nsamp, n->y))) return rc;
   if ((rc = backward(n, x, target, mask, nsamp, mask_sum))) return rc;
   n->steps += 1;
   const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
   const float c1 = 1.f - std::pow(b1, (float)n->steps), c2 = 1.f - std::pow(b2, (float)n->steps);
   for (int l = 0; l < 4; ++l)
      k_adam<<<(kSizes[l] + 255) / 256, 256, 0, n->stream>>>(n->w[l], n->gw[l], n->m[l], n->v[l],
                                                              kSizes[l], lr, b1, b2, eps, c1, c2);
   samrai_b200::add_kernel_launches(4);
   if ((rc = pack(n))) return rc;
   if (loss) {
      if ((rc = read_back(n, true))) return rc;
      double l = 0;
      std::memcpy(&l, n->host + kGradFloats * 4, sizeof(l));
      *loss = l / mask_sum;
   }
   return FAC_OK;
}

}  // extern "C"
