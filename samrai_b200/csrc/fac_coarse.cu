// Coarsest-level solve: every red-black sweep of a smoothing to a tolerance
// in one launch, one thread-block cluster per problem (sm_100a).
//
// The cells of a problem's coarsest level -- all its patches, in patch and
// storage order -- are cut into equal runs, one per CTA of the cluster
// (tables built by build_coarse_solve).  A thread owns up to SP cells of
// each colour for the whole launch: their values, right-hand sides, C, the
// products (1/dx) D of their faces and the reciprocal of the diagonal stay in
// registers, formed once with the expressions of rb_point, so that a pass is
// only the fluxes, the residual and the update, in the order and rounding of
// k_rbgs (the same bits).  The values sit in shared memory, colour by colour
// (a row's neighbours of the other colour are consecutive words), where the
// neighbours read them.
//
// Between CTAs a pass needs no barrier: a cell on the cut sends its new value
// into the neighbour CTA's copy with st.async, which counts the bytes on that
// CTA's mbarrier of the colour, and a CTA goes on once its own threads have
// met and its copies of the colour have come in.  A CTA cannot run ahead into
// a copy that is still read: the value it sends next needs the values of the
// cells that read it.  Nor can a colour's phase complete while a thread still
// waits for the one before: it is armed behind the block barrier after those
// waits.  The sweep check goes round the cluster behind the
// sweep: the CTAs of the checked patch store the outcome in every CTA, all
// arrive at the cluster barrier after the black pass, and wait for it after
// the next red pass, which is undone (each thread keeps its old red values)
// if the sweep before it was the last.
//
// A thread whose wait runs out sets the device error flag and goes on without
// waiting, so that every CTA still sends, and arrives at the cluster barrier,
// as often as the others; the sweep's outcome carries the stop to all of them.
// Thread 0, which arms the phases, then waits for the values still on their way
// before its CTA exits.  (The cluster barrier itself is the hardware's, between
// CTAs that are resident together: it opens because every thread arrives.)
//
// The homogeneous Robin values behind physical faces are a list of their own,
// renewed while the copies are on their way, one division per thread.
//
// What bounds it: the latency of a pass.  Measured per pass (B200, FP64, the
// sweep check on; in brackets one block per problem on shared copies of all
// arrays, thread per cell, with the coefficients and the diagonal's division
// formed anew in every pass): 64^2 constant D 0.65 us on 8 CTAs [3.0], 57 x 76
// variable D and C 0.66 us on 8 [3.5], 8^3 variable D 0.37 us on one CTA
// [2.2], 16^3 variable D 0.74 us on 8 and 0.81 us on 4 [6.2]; 32^3 in eight
// patches 1.43 us on 16 [14, a launch per pass].  A CTA alone takes 0.3 us for
// the chain of shared loads, ten dependent FP64 operations and the barrier;
// the way to another CTA adds 0.3 us whatever their number, so a level is
// spread until a thread has one cell of a colour (coarse_pass_us).
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <tuple>

#include "fac_device.h"
#include "fac_internal.h"
#include "fac_kernels.h"

namespace samrai_b200 {

namespace {

using namespace dev;

__device__ __forceinline__ unsigned shared_addr(const void *p)
{
   return (unsigned)__cvta_generic_to_shared(p);
}

// the address of local shared address a in CTA rank r of the cluster
__device__ __forceinline__ unsigned map_rank(unsigned a, unsigned r)
{
   unsigned o;
   asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(a), "r"(r));
   return o;
}

__device__ __forceinline__ void store_remote(unsigned a, int v)
{
   asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// v to address a of a CTA of the cluster, its 8 bytes counted on mbarrier bar there
__device__ __forceinline__ void send(unsigned a, double v, unsigned bar)
{
   asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
                "l"(__double_as_longlong(v)), "r"(bar)
                : "memory");
}

__device__ __forceinline__ void expect_bytes(unsigned bar, unsigned bytes)
{
   asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                : "memory");
}

// Wait for a phase of an mbarrier whose bytes come from other CTAs; gives up
// after `limit` SM clock cycles.
__device__ __forceinline__ bool wait_bytes(unsigned bar, unsigned parity, long long limit)
{
   unsigned ok = 0;
   long long t0 = 0;
   for (int n = 0;; ++n) {
      asm volatile(
         "{\n"
         " .reg .pred p;\n"
         " mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
         " selp.u32 %0, 1, 0, p;\n"
         "}\n"
         : "=r"(ok)
         : "r"(bar), "r"(parity)
         : "memory");
      if (ok) return true;
      if (n == 0) t0 = clock64();
      else if (clock64() - t0 > limit) return false;
   }
}

__device__ __forceinline__ void cluster_arrive()
{
   asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}

__device__ __forceinline__ void cluster_wait()
{
   asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// One thread's cells of one colour.
template <int DIM, bool DVAR, int CKIND, int SP>
struct CoarseCells {
   double uc[SP], fv[SP], dudr[SP], sc[CKIND == 2 ? SP : 1];
   double ad[DVAR ? SP : 1][2 * DIM];  // (1/dx) D of the low and high face per axis
   unsigned nb[SP][DIM];               // shared values of the low | high << 16 neighbour
   unsigned push[SP];                  // first push entry | entries << 24 | checked patch << 31
};

template <int DIM, bool DVAR, int CKIND, int SP>
__global__ void __launch_bounds__(kCoarseThreads, 1)
k_coarse_solve(const CoarseCta *__restrict__ ctas, const CoarseCell *__restrict__ cells,
               const long long *__restrict__ halo, const unsigned *__restrict__ push,
               const unsigned *__restrict__ ghost, const PatchDesc *__restrict__ patches,
               double *__restrict__ u, const double *__restrict__ f,
               const double *__restrict__ dside, const double *__restrict__ cfield,
               double dconst, double cconst, BcCoefs bc, int ncta, int nsweeps, double tol,
               int *__restrict__ run, long long *__restrict__ sweeps, int *__restrict__ err,
               WaitTest wt)
{
   extern __shared__ __align__(16) double su[];
   __shared__ unsigned long long bars[3];  // per colour, and one that nothing completes
   __shared__ double bnum[6], bden[6], binv[6];
   // the outcome of a sweep, by its parity: {some residual above tol, a wait ran out}
   __shared__ __align__(8) int2 flag[2];
   pdl_begin();
   const CoarseCta ct = ctas[blockIdx.x];
   if (!run[ct.prob]) return;  // the whole cluster
   const int tid = threadIdx.x;
   const int nown = ct.ncol[0] + ct.ncol[1];
   const int ghost0 = nown + ct.nhalo, nghost = ct.nghost[0] + ct.nghost[1];
   uint2 *spush = reinterpret_cast<uint2 *>(su + ghost0 + nghost);
   unsigned *sghost = reinterpret_cast<unsigned *>(spush + ct.npush);
   const unsigned su0 = shared_addr(su), bar0 = shared_addr(bars), flag0 = shared_addr(flag);
   for (int q = tid; q < ct.npush; q += kCoarseThreads) {
      const unsigned t = push[ct.push0 + q];
      spush[q] = make_uint2(map_rank(su0, t >> 16) + 8u * (t & 0xffffu), map_rank(bar0, t >> 16));
   }
   for (int q = tid; q < ct.nhalo; q += kCoarseThreads) su[nown + q] = u[halo[ct.halo0 + q]];
   for (int q = tid; q < nghost; q += kCoarseThreads) sghost[q] = ghost[ct.ghost0 + q];
   double dxi, dyi, dzi;
   {
      const PatchDesc &p = patches[ct.patch0];
      dxi = 1.0 / p.dx[0];
      dyi = 1.0 / p.dx[1];
      dzi = DIM == 3 ? 1.0 / p.dx[2] : 0.0;
      if (tid < 2 * DIM) {
         // robin_abg, homogeneous: u (b - h a / 2) / (b + h a / 2)
         const double t = 0.5 * p.dx[tid >> 1] * bc.a[tid];
         const double den = bc.b[tid] + t;
         bnum[tid] = bc.b[tid] - t;
         bden[tid] = den;
         // dividing by a power of two is multiplying by its reciprocal, exactly
         const unsigned long long m = (unsigned long long)__double_as_longlong(den);
         const unsigned ex = (unsigned)(m >> 52) & 0x7ffu;
         binv[tid] = (m << 12) == 0ull && ex > 2u && ex < 2044u ? 1.0 / den : 0.0;
      }
   }
   if (tid == 0) {
      flag[0] = flag[1] = make_int2(0, 0);
      for (int k = 0; k < 3; ++k)
         asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8u * k) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      for (int k = 0; k < 2; ++k)
         if (ct.nin[k]) expect_bytes(bar0 + 8u * k, 8u * ct.nin[k]);
   }
   const double adc[3] = {dxi * dconst, dyi * dconst, dzi * dconst};
   CoarseCells<DIM, DVAR, CKIND, SP> cs[2];
   double ured[SP];  // red values before the latest red pass
   // renew the ghost values of the cells of a colour; the list from the last
   // thread down, where threads without cells are
   auto ghosts = [&](int col) {
      const int e = col ? nghost : ct.nghost[0];
      for (int q = (col ? ct.nghost[0] : 0) + kCoarseThreads - 1 - tid; q < e; q += kCoarseThreads) {
         const unsigned g = sghost[q];
         const int fc = (int)(g >> 16);
         const double x = su[g & 0xffffu] * bnum[fc];
         const double inv = binv[fc];
         su[ghost0 + q] = inv != 0.0 ? x * inv : x / bden[fc];
      }
   };
#pragma unroll
   for (int col = 0; col < 2; ++col) {
      CoarseCells<DIM, DVAR, CKIND, SP> &c = cs[col];
      const int self0 = col ? ct.ncol[0] : 0;
#pragma unroll
      for (int s = 0; s < SP; ++s) {
         const int q = tid + s * kCoarseThreads;
         if (q >= ct.ncol[col]) continue;
         const CoarseCell ce = cells[ct.cell0 + self0 + q];
         const PatchDesc &p = patches[ce.patch];
         int li, lj, lk;
         patch_cell(p, ce.lin, p.hi[0] - p.lo[0] + 1, p.hi[1] - p.lo[1] + 1, li, lj, lk);
         const int i = p.lo[0] + li, j = p.lo[1] + lj, k = DIM == 3 ? p.lo[2] + lk : 0;
         c.uc[s] = u[cidx<DIM>(p, p.off1, 1, i, j, k)];
         su[self0 + q] = c.uc[s];
         c.fv[s] = f[p.off0 + ce.lin];
         const double scv = CKIND == 2 ? cfield[p.off0 + ce.lin] : (CKIND == 1 ? cconst : 0.0);
         if (CKIND == 2) c.sc[s] = scv;
         double d[6] = {dconst, dconst, dconst, dconst, dconst, dconst};
         if (DVAR) {
            d[0] = dside[sidx(p, 0, i, j, k)];
            d[1] = dside[sidx(p, 0, i + 1, j, k)];
            d[2] = dside[sidx(p, 1, i, j, k)];
            d[3] = dside[sidx(p, 1, i, j + 1, k)];
            if (DIM == 3) {
               d[4] = dside[sidx(p, 2, i, j, k)];
               d[5] = dside[sidx(p, 2, i, j, k + 1)];
            }
            c.ad[s][0] = dxi * d[0];
            c.ad[s][1] = dxi * d[1];
            c.ad[s][2] = dyi * d[2];
            c.ad[s][3] = dyi * d[3];
            if (DIM == 3) {
               c.ad[s][2 * DIM - 2] = dzi * d[4];
               c.ad[s][2 * DIM - 1] = dzi * d[5];
            }
         }
         if (DIM == 2) {
            c.dudr[s] = 1.0 / ((dxi * dxi * (d[1] + d[0]) + dyi * dyi * (d[3] + d[2])) - scv);
         } else {
            const double dxi2 = dxi * dxi, dyi2 = dyi * dyi, dzi2 = dzi * dzi;
            c.dudr[s] = 1.0 / ((dxi2 * (d[1] + d[0]) + dyi2 * (d[3] + d[2]) + dzi2 * (d[5] + d[4])) -
                               scv);
         }
#pragma unroll
         for (int a = 0; a < DIM; ++a)
            c.nb[s][a] = (unsigned)ce.nb[2 * a] | ((unsigned)ce.nb[2 * a + 1] << 16);
         c.push[s] = (unsigned)ce.push0 | ((unsigned)ce.npush << 24) | ((unsigned)ce.last << 31);
      }
   }
   // every CTA's shared memory and mbarriers are set before the first send
   cluster_arrive();
   cluster_wait();
   ghosts(0);
   ghosts(1);
   __syncthreads();
   // the test of the bounded wait: in problems of even number the last thread
   // of the first CTA waits for what nothing completes, in the others every
   // thread does
   const bool never = wt.never && ((ct.prob & 1) || (ct.rank == 0 && tid == kCoarseThreads - 1));
   bool going = true;
   int dead = 0;  // 1 + 2 sweep + colour of this thread's wait that ran out
   auto outcome = [&](int s) {
      const long long v = *(volatile long long *)&flag[s & 1];
      return (tol < 0.0 || (int)v != 0) && (int)(v >> 32) == 0;
   };
   int sw = 0;
   for (; sw < nsweeps; ++sw) {
      bool any = false;
#pragma unroll
      for (int col = 0; col < 2; ++col) {
         CoarseCells<DIM, DVAR, CKIND, SP> &c = cs[col];
         const int self0 = col ? ct.ncol[0] : 0;
#pragma unroll
         for (int s = 0; s < SP; ++s) {
            const int q = tid + s * kCoarseThreads;
            if (q >= ct.ncol[col]) continue;
            const double uc = c.uc[s];
            if (col == 0) ured[s] = uc;
            const double *ad = DVAR ? c.ad[s] : nullptr;
            const double nxl = su[c.nb[s][0] & 0xffffu], nxh = su[c.nb[s][0] >> 16];
            const double nyl = su[c.nb[s][1] & 0xffffu], nyh = su[c.nb[s][1] >> 16];
            const double fxl = (DVAR ? ad[0] : adc[0]) * (uc - nxl);
            const double fxh = (DVAR ? ad[1] : adc[0]) * (nxh - uc);
            const double fyl = (DVAR ? ad[2] : adc[1]) * (uc - nyl);
            const double fyh = (DVAR ? ad[3] : adc[1]) * (nyh - uc);
            const double scv = CKIND == 2 ? c.sc[s] : (CKIND == 1 ? cconst : 0.0);
            double residual;
            if (DIM == 2) {
               residual = c.fv[s] - (dxi * (fxh - fxl) + dyi * (fyh - fyl)) - scv * uc;
            } else {
               const double nzl = su[c.nb[s][DIM - 1] & 0xffffu], nzh = su[c.nb[s][DIM - 1] >> 16];
               const double fzl = (DVAR ? ad[2 * DIM - 2] : adc[2]) * (uc - nzl);
               const double fzh = (DVAR ? ad[2 * DIM - 1] : adc[2]) * (nzh - uc);
               residual = c.fv[s] -
                          (dxi * (fxh - fxl) + dyi * (fyh - fyl) + dzi * (fzh - fzl)) - scv * uc;
            }
            const double v = uc + -residual * c.dudr[s];
            c.uc[s] = v;
            su[self0 + q] = v;
            any = any || ((c.push[s] >> 31) && fabs(residual) > tol);
            const unsigned p0 = c.push[s] & 0xffffffu, pe = p0 + ((c.push[s] >> 24) & 0x7fu);
            for (unsigned e = p0; e < pe; ++e) {
               const uint2 t = spush[e];
               send(t.x, v, t.y + 8u * col);
            }
         }
         // this CTA's values of the colour are in place; after the black pass
         // also the sweep check of smoothErrorByRedBlack: the problem stops
         // once no |residual| of its last patch exceeded the tolerance in
         // either pass (the reference's maximum is that patch's; a NaN never
         // exceeds it)
         int hit = 0;
         if (col == 1 && tol >= 0.0 && ct.last) hit = __syncthreads_or(any);
         else __syncthreads();
         // Every thread has left its wait for the other colour's copies, so that
         // colour's next phase may complete from here on: its bytes are expected
         // now (early ones are counted already).  Expected any sooner, a thread that
         // is late at its wait, one without a cell on the cut among them, could
         // find the phase after the one it waits for complete, and wait for good:
         // the other CTAs need nothing of it to send again.
         if (tid == 0 && !dead && ct.nin[1 - col] && (col == 1 || sw > 0))
            expect_bytes(bar0 + 8u * (1 - col), 8u * ct.nin[1 - col]);
         if (ncta == 1) {
            ghosts(col);
            if (col == 1) going = tol < 0.0 || hit;
            continue;
         }
         if (col == 1) {
            // the last sweep's outcome was read by all after the red pass; no
            // CTA stores into its place again before it has seen this arrival
            if (tid == 0 && sw > 0) flag[(sw - 1) & 1] = make_int2(0, 0);
            if (hit && tid < ncta) store_remote(map_rank(flag0 + 8u * (sw & 1), tid), 1);
            if (dead)
               for (int r = 0; r < ncta; ++r) store_remote(map_rank(flag0 + 8u * (sw & 1) + 4u, r), 1);
            cluster_arrive();
         }
         ghosts(col);
         if (ct.nin[col] && !dead &&
             !wait_bytes(never ? bar0 + 16u : bar0 + 8u * col, never ? 0u : sw & 1, wt.limit)) {
            // on with the passes, without waiting: every CTA keeps sending and
            // arriving until the outcome of a sweep stops them all together
            dead = 1 + 2 * sw + col;
            atomicExch(err, 1);
         }
         if (col == 0 && sw > 0) {
            cluster_wait();
            going = outcome(sw - 1);
            if (!going) {
               // the sweep before was the last: take this red pass back
#pragma unroll
               for (int s = 0; s < SP; ++s) cs[0].uc[s] = ured[s];
               break;
            }
         }
      }
      if (ncta == 1) {
         if (!going) {
            ++sw;
            break;
         }
         continue;
      }
      if (!going) break;
   }
   // passes of each colour all CTAs have made: a stop comes after a red one
   const int made[2] = {sw < nsweeps ? sw + 1 : sw, sw};
   if (ncta > 1 && going && sw > 0) {
      cluster_wait();
      going = outcome(sw - 1);
   }
   // Values on their way into this CTA's shared memory land before it exits.
   // Thread 0 has seen every phase of both colours complete or, where its own
   // wait ran out, goes through those since then now; the first of them is armed.
   if (dead && tid == 0) {
      const int gsw = (dead - 1) >> 1, gcol = (dead - 1) & 1;
      for (int col = 0; col < 2; ++col) {
         const int first = col < gcol ? gsw + 1 : gsw;
         for (int q = first; ct.nin[col] && q < made[col]; ++q) {
            if (q > first) expect_bytes(bar0 + 8u * col, 8u * ct.nin[col]);
            if (!wait_bytes(bar0 + 8u * col, q & 1, WaitTest().limit)) break;
         }
      }
   }
#pragma unroll
   for (int col = 0; col < 2; ++col) {
      const int self0 = col ? ct.ncol[0] : 0;
#pragma unroll
      for (int s = 0; s < SP; ++s) {
         const int q = tid + s * kCoarseThreads;
         if (q >= ct.ncol[col]) continue;
         const CoarseCell ce = cells[ct.cell0 + self0 + q];
         const PatchDesc &p = patches[ce.patch];
         int li, lj, lk;
         patch_cell(p, ce.lin, p.hi[0] - p.lo[0] + 1, p.hi[1] - p.lo[1] + 1, li, lj, lk);
         u[cidx<DIM>(p, p.off1, 1, p.lo[0] + li, p.lo[1] + lj, DIM == 3 ? p.lo[2] + lk : 0)] =
            cs[col].uc[s];
      }
   }
   if (tid == 0 && ct.rank == 0) {
      sweeps[ct.prob] += sw;
      run[ct.prob] = going ? 1 : 0;
   }
}

using CoarseFn = void (*)(const CoarseCta *, const CoarseCell *, const long long *,
                          const unsigned *, const unsigned *, const PatchDesc *, double *,
                          const double *, const double *, const double *, double, double, BcCoefs,
                          int, int, double, int *, long long *, int *, WaitTest);

template <int DIM, bool DVAR, int CKIND>
CoarseFn pick_sp(int sp)
{
   return sp == 1 ? k_coarse_solve<DIM, DVAR, CKIND, 1>
                  : (sp == 2 ? k_coarse_solve<DIM, DVAR, CKIND, 2>
                             : k_coarse_solve<DIM, DVAR, CKIND, 4>);
}

template <int DIM, bool DVAR>
CoarseFn pick_c(int ckind, int sp)
{
   return ckind == 2 ? pick_sp<DIM, DVAR, 2>(sp)
                     : (ckind == 1 ? pick_sp<DIM, DVAR, 1>(sp) : pick_sp<DIM, DVAR, 0>(sp));
}

CoarseFn pick(int dim, const PoissonSpec &spec, int sp)
{
   if (dim == 2) return spec.d_variable ? pick_c<2, true>(spec.c_kind, sp) : pick_c<2, false>(spec.c_kind, sp);
   return spec.d_variable ? pick_c<3, true>(spec.c_kind, sp) : pick_c<3, false>(spec.c_kind, sp);
}

cudaLaunchConfig_t launch_config(int blocks, int ncta, size_t smem, cudaStream_t s,
                                 cudaLaunchAttribute *attr)
{
   cudaLaunchConfig_t cfg = {};
   cfg.gridDim = dim3((unsigned)blocks);
   cfg.blockDim = dim3(kCoarseThreads);
   cfg.dynamicSmemBytes = smem;
   cfg.stream = s;
   attr->id = cudaLaunchAttributeClusterDimension;
   attr->val.clusterDim.x = (unsigned)ncta;
   attr->val.clusterDim.y = 1;
   attr->val.clusterDim.z = 1;
   attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
   attr[1].val.programmaticStreamSerializationAllowed = 1;
   cfg.attrs = attr;
   cfg.numAttrs = 2;
   return cfg;
}

}  // namespace

int coarse_solve_clusters(int dim, const PoissonSpec &spec, int ncta, int sp)
{
   // queried once per device, kernel and cluster size
   static std::mutex mutex;
   static std::map<std::tuple<int, CoarseFn, int>, int> known;
   CoarseFn fn = pick(dim, spec, sp);
   int device = 0;
   if (cudaGetDevice(&device) != cudaSuccess) {
      (void)cudaGetLastError();
      return 0;
   }
   std::lock_guard<std::mutex> lock(mutex);
   const auto at = known.find({device, fn, ncta});
   if (at != known.end()) return at->second;
   int &answer = known[{device, fn, ncta}];
   if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSolveSmemMax) !=
          cudaSuccess ||
       (ncta > 8 && cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
                       cudaSuccess)) {
      (void)cudaGetLastError();
      return 0;
   }
   cudaLaunchAttribute attr[2];
   const cudaLaunchConfig_t cfg = launch_config(ncta, ncta, kSolveSmemMax, nullptr, attr);
   int clusters = 0;
   if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      return 0;
   }
   answer = clusters;
   return clusters;
}

cudaError_t launch_coarse_solve(cudaStream_t s, int dim, const PoissonSpec &spec, int nprob,
                                int ncta, int sp, int smem, const CoarseCta *ctas,
                                const CoarseCell *cells, const long long *halo,
                                const unsigned *push, const unsigned *ghost,
                                const PatchDesc *patches, double *u, const double *f,
                                const double *dside, const double *cfield, const BcCoefs &bc,
                                int nsweeps, double tol, int *run, long long *sweeps, int *err,
                                const WaitTest &wt)
{
   if (nprob <= 0 || nsweeps <= 0) return cudaSuccess;
   cudaLaunchAttribute attr[2];
   const cudaLaunchConfig_t cfg = launch_config(nprob * ncta, ncta, smem, s, attr);
   add_kernel_launches(1);
   return cudaLaunchKernelEx(&cfg, pick(dim, spec, sp), ctas, cells, halo, push, ghost, patches,
                             u, f, dside, cfield, spec.d_const, spec.c_const, bc, ncta, nsweeps,
                             tol, run, sweeps, err, wt);
}

}  // namespace samrai_b200
