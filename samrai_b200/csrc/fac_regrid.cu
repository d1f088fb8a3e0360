// The regrid step on the device: tagging by the FAC_adaptive adaption
// estimate and the tag histograms (signatures) of Berger-Rigoutsos
// clustering.  The clustering's decisions (bounding box, efficiency,
// zero-swath and inflection cuts, recombination) are host logic over the
// histograms, in fac_host.cu (fac_cluster_tags).
#include <cuda_runtime.h>

#include "fac_device.h"
#include "fac_internal.h"
#include "fac_kernels.h"

namespace samrai_b200 {

namespace {

using namespace dev;

// AdaptivePoisson::computeAdaptionEstimate (source/test/FAC_adaptive/
// AdaptivePoisson.C:622-720) and the threshold test of
// applyGradientDetector (:517-527): the largest |(u(+) + u(-)) - 2 u(0)|
// along the axes and half of it along the face diagonals; tag where it
// exceeds the threshold.  The maxima are taken in the reference's order
// (max is exact, the order only matters for NaN).
template <int DIM>
__global__ void __launch_bounds__(kThreads)
k_adaption_tags(const PatchDesc *__restrict__ patches, const Chunk *__restrict__ chunks,
                int nwork, const double *__restrict__ u, double threshold,
                unsigned char *__restrict__ tags, unsigned long long *__restrict__ counts,
                const int *__restrict__ run)
{
   pdl_begin();
   __shared__ unsigned cnt[kThreads / 32];
   WORK_LOOP(ch) {
      const PatchDesc &p = patches[ch.patch];
      if (run && !run[p.prob]) continue;
      const int nx = p.hi[0] - p.lo[0] + 1;
      const int ny = p.hi[1] - p.lo[1] + 1;
      const int gx = nx + 2, gxy = (nx + 2) * (ny + 2);
      const double *up = u + p.off1;
      unsigned mine = 0;
      for (int t = threadIdx.x; t < ch.count; t += blockDim.x) {
         const int lin = ch.begin + t;
         int li, lj, lk;
         patch_cell(p, lin, nx, ny, li, lj, lk);
         const int c = (li + 1) + gx * (lj + 1) + (DIM == 3 ? gxy * (lk + 1) : 0);
         const double u0 = up[c];
         auto d2 = [&](int o) { return fabs((up[c + o] + up[c - o]) - 2 * u0); };
         double est;
         if (DIM == 2) {
            const double est0 = d2(1);
            const double est1 = d2(gx);
            const double est2 = 0.5 * d2(1 + gx);
            const double est3 = 0.5 * fabs((up[c + 1 - gx] + up[c - 1 + gx]) - 2 * u0);
            est = fmax(fmax(est0, est1), fmax(est2, est3));
         } else {
            const double est0 = d2(1);
            const double est1 = d2(gx);
            const double est2 = d2(gxy);
            const double est3 = 0.5 * d2(gx + gxy);
            const double est4 = 0.5 * fabs((up[c + gx - gxy] + up[c - gx + gxy]) - 2 * u0);
            const double est5 = 0.5 * d2(1 + gxy);
            const double est6 = 0.5 * fabs((up[c + 1 - gxy] + up[c - 1 + gxy]) - 2 * u0);
            const double est7 = 0.5 * d2(1 + gx);
            const double est8 = 0.5 * fabs((up[c + 1 - gx] + up[c - 1 + gx]) - 2 * u0);
            const double esta = fmax(est0, est1), estb = fmax(est2, est3);
            const double estc = fmax(est4, est5), estd = fmax(est6, est7);
            est = fmax(fmax(fmax(esta, estb), fmax(estc, estd)), est8);
         }
         const bool tag = est > threshold;
         tags[p.off0 + lin] = tag ? 1 : 0;
         mine += tag ? 1u : 0u;
      }
      for (int o = 16; o > 0; o >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, o);
      if ((threadIdx.x & 31) == 0) cnt[threadIdx.x >> 5] = mine;
      __syncthreads();
      if (threadIdx.x == 0) {
         unsigned long long s = 0;
         for (int w = 0; w < kThreads / 32; ++w) s += cnt[w];
         if (s) atomicAdd(counts + p.prob, s);
      }
      __syncthreads();
   }
}

// The tags of one problem's patches of a level placed into a dense array
// over the box [lo, lo + n) (x fastest); the array is zeroed before.
template <int DIM>
__global__ void __launch_bounds__(kThreads)
k_tags_dense(const PatchDesc *__restrict__ patches, const Chunk *__restrict__ chunks, int nwork,
             const unsigned char *__restrict__ tags, int prob, int3 lo, int3 n,
             unsigned char *__restrict__ dense)
{
   pdl_begin();
   WORK_LOOP(ch) {
      const PatchDesc &p = patches[ch.patch];
      if (p.prob != prob) continue;
      const int nx = p.hi[0] - p.lo[0] + 1;
      const int ny = p.hi[1] - p.lo[1] + 1;
      for (int t = threadIdx.x; t < ch.count; t += blockDim.x) {
         const int lin = ch.begin + t;
         int li, lj, lk;
         patch_cell(p, lin, nx, ny, li, lj, lk);
         const long long x = p.lo[0] + li - lo.x, y = p.lo[1] + lj - lo.y;
         const long long z = DIM == 3 ? p.lo[2] + lk - lo.z : 0;
         dense[x + (long long)n.x * (y + (long long)n.y * z)] = tags[p.off0 + lin];
      }
   }
}

// Tag histograms of Berger-Rigoutsos nodes (makeLocalTagHistogram,
// mesh/BergerRigoutsosNode.C:1186-1241): per node, the number of tags in
// each index plane normal to each axis.  One block per work item (a run of
// rows of one node box; a row runs along x).  A row is read in words of four
// tags (the dense arrays' rows are whole words, so a node's x positions keep
// their byte in every row); a row of up to 128 tags takes as many lanes as it
// has words, so a warp reads several short rows at once.  A lane adds its words
// up bytewise (at most 255 rows), rows' totals are reduced among their lanes;
// both are gathered in shared memory and added to the node's counts once per
// block.  Integer atomics: the result does not depend on the order.
//
// Bound by the latency of the tag loads, four rows of a lane in flight.  Eight
// problems of 10.4 million cells, their finest levels: 12.6 us a tree depth on
// average, 300 with a block of byte loads and two barriers per row; the whole
// regrid step 7.3 ms and 2.2.
__global__ void __launch_bounds__(kBrThreads)
k_br_histogram(const BrItem *__restrict__ items, const BrNode *__restrict__ nodes,
               const unsigned char *__restrict__ dense_all, int *__restrict__ hist)
{
   pdl_begin();
   __shared__ int xs[kBrMaxX], rows[kBrMaxRows];
   const BrItem it = items[blockIdx.x];
   const BrNode nd = nodes[it.node];
   const int ex = nd.hi[0] - nd.lo[0] + 1, ey = nd.hi[1] - nd.lo[1] + 1;
   int *hx = hist + nd.hoff, *hy = hx + ex, *hz = hy + ey;
   const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
   for (int i = threadIdx.x; i < ex; i += kBrThreads) xs[i] = 0;
   for (int i = threadIdx.x; i < it.nrows; i += kBrThreads) rows[i] = 0;
   __syncthreads();
   const int x0 = nd.lo[0] - nd.dlo[0];
   const int shift = x0 & 3;                    // tags of the first word before the node
   const int words = (shift + ex + 3) >> 2;
   int lanes = 1;                               // per row
   while (lanes < words && lanes < 32) lanes *= 2;
   const int wl = lane & (lanes - 1), per = 32 / lanes;
   const int first = wid * per + lane / lanes, step = kBrThreads / 32 * per;
   const long long pitch = nd.dn[0], plane = pitch * nd.dn[1];
   const unsigned char *base = dense_all + nd.doff + (x0 - shift) +
                               pitch * (nd.lo[1] - nd.dlo[1]) + plane * (nd.lo[2] - nd.dlo[2]);
   for (int w0 = 0; w0 < words; w0 += lanes) {
      const int w = w0 + wl;
      // bytes of this lane's word inside the node
      unsigned mask = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
         const int x = 4 * w + q - shift;
         if (x >= 0 && x < ex) mask |= 1u << (8 * q);
      }
      unsigned sum = 0;  // four counts
      for (int r0 = 0; r0 < it.nrows; r0 += 4 * step) {
         unsigned v[4];
#pragma unroll
         for (int q = 0; q < 4; ++q) {
            const int r = r0 + first + q * step, g = it.row0 + r;
            v[q] = 0;
            if (r < it.nrows && mask)
               v[q] = *reinterpret_cast<const unsigned *>(base + 4 * w + pitch * (g % ey) +
                                                          plane * (g / ey)) & mask;
         }
#pragma unroll
         for (int q = 0; q < 4; ++q) {
            const int r = r0 + first + q * step;
            sum += v[q];
            int c = __popc(v[q]);
            for (int o = lanes / 2; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
            if (wl == 0 && r < it.nrows && c) rows[r] += c;  // this lane's row alone
         }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
         const int c = (int)((sum >> (8 * q)) & 0xffu);
         if (c) atomicAdd(&xs[4 * w + q - shift], c);
      }
   }
   __syncthreads();
   for (int i = threadIdx.x; i < ex; i += kBrThreads)
      if (xs[i]) atomicAdd(hx + i, xs[i]);
   for (int i = threadIdx.x; i < it.nrows; i += kBrThreads)
      if (rows[i]) {
         const int g = it.row0 + i;
         atomicAdd(hy + g % ey, rows[i]);
         atomicAdd(hz + g / ey, rows[i]);
      }
}

}  // namespace

void launch_adaption_tags(cudaStream_t s, int dim, int nchunks, const PatchDesc *patches,
                          const Chunk *chunks, const double *u, double threshold,
                          unsigned char *tags, unsigned long long *counts, const int *run)
{
   if (nchunks <= 0) return;
   add_kernel_launches(1);
   if (dim == 2)
      launch_after(k_adaption_tags<2>, work_grid(k_adaption_tags<2>, nchunks), kThreads, 0, s, patches, chunks, nchunks, u, threshold, tags, counts, run);
   else
      launch_after(k_adaption_tags<3>, work_grid(k_adaption_tags<3>, nchunks), kThreads, 0, s, patches, chunks, nchunks, u, threshold, tags, counts, run);
}

void launch_tags_dense(cudaStream_t s, int dim, int nchunks, const PatchDesc *patches,
                       const Chunk *chunks, const unsigned char *tags, int prob, const int *lo,
                       const int *n, unsigned char *dense)
{
   if (nchunks <= 0) return;
   add_kernel_launches(1);
   const int3 l = make_int3(lo[0], lo[1], lo[2]), e = make_int3(n[0], n[1], n[2]);
   if (dim == 2)
      launch_after(k_tags_dense<2>, work_grid(k_tags_dense<2>, nchunks), kThreads, 0, s, patches, chunks, nchunks, tags, prob, l, e, dense);
   else
      launch_after(k_tags_dense<3>, work_grid(k_tags_dense<3>, nchunks), kThreads, 0, s, patches, chunks, nchunks, tags, prob, l, e, dense);
}

void launch_br_histogram(cudaStream_t s, int nitems, const BrItem *items, const BrNode *nodes,
                         const unsigned char *dense, int *hist)
{
   if (nitems <= 0) return;
   add_kernel_launches(1);
   launch_after(k_br_histogram, nitems, kBrThreads, 0, s, items, nodes, dense, hist);
}

}  // namespace samrai_b200
