// pm_stream_kernel.cuh -- the streamed inversion kernel template of one pixel per
// warp and its launcher, shared by the translation units that instantiate it:
// pm_stream.cu (FP64 of normal Zeeman triplets; their FP32 form holds two pixels per
// warp, pm_pair_kernel.cuh) and pm_stream_zm.cu (Zeeman multiplets).  Everything
// here has internal linkage; each unit compiles its own instances.
#pragma once
#include "pm_device.cuh"

namespace {
// ---------------------------------------------------------------------------
// Streamed inversion: a persistent kernel fed while it runs.  Pixels are
// tickets; the host publishes tickets in stream order after the data they cover
// has been copied (a copy engine writes PmStreamQ::avail), and appends scans
// ("jobs": a run of tickets with its own buffers and wavelength grid) to a ring
// of descriptors.  A warp takes the next ticket with one atomicAdd and owns it:
// if it is not yet published, the warp waits for its publication, so a ticket
// is never handed out twice nor lost.  The kernel ends when the host closes the
// queue (PmStreamQ::closed, written after the last publication): warps holding
// tickets beyond the final count exit.  Waits are bounded: a waiting warp that sees no
// publication for wait_limit_ns sets PMQ_ERR_WAIT and exits.  (The limit does not
// count from the warp's own ticket: a slow producer may take longer to reach it.)
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ long long global_ns() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Next ticket, or -1 when the kernel should exit.
__device__ long long next_ticket(PmStreamQ* q, long long limit_ns) {
  const unsigned long long t = atomicAdd(&q->next, 1ull);
  long long since = -1;
  unsigned long long avail = 0;
  unsigned sleep = 32;
  while (true) {
    const unsigned long long seen = ld_acquire(&q->avail);
    if (t < seen) return (long long)t;
    if (seen != avail) since = -1;
    avail = seen;
    if (ld_acquire(&q->closed)) {
      // closed is written after the last publication: one more look
      return t < ld_acquire(&q->avail) ? (long long)t : -1;
    }
    const long long now = global_ns();
    if (since < 0) since = now;
    if (now - since > limit_ns) {
      atomicExch(&q->err, (unsigned long long)PMQ_ERR_WAIT);
      return -1;
    }
    __nanosleep(sleep);
    sleep = sleep < 2048 ? 2 * sleep : 2048;
  }
}


// The grids a launch serves, by value: all PMK_MAX_GRIDS slots for a server's
// mixed launch, one slot otherwise (a 7 KB rather than 28 KB parameter block).
template <int NG>
struct GridParams {
  int ngrids;
  int pad_;
  PmParams g[NG];
};

// The warp's pixel is finished: count it on its job and, when it was the job's
// last pixel, raise the job's host flag (the server's completion signal).
template <typename SM>
__device__ __forceinline__ void job_pixel_done(SM& sm, int lane) {
  const PmJob* jp = *reinterpret_cast<const PmJob* const volatile*>(&sm.job);
  unsigned long long* done = ld_ptr(&jp->done);
  if (done) {
    __threadfence();  // every lane: its part of this pixel's results before the count
    __syncwarp();
    if (lane == 0) {
      int* flag = ld_ptr(&jp->host_flag);
      const unsigned long long np = __ldcg(reinterpret_cast<const unsigned long long*>(&jp->npix));
      if (atomicAdd(done, 1ull) + 1 == np && flag) {
        __threadfence_system();
        *reinterpret_cast<volatile int*>(flag) = 1;
      }
    }
  }
  __syncwarp();
}

template <typename R, int KT, int MINB, bool MULTI, bool MAC, bool PIXGRID, bool ZM = false>
__global__ void __launch_bounds__(128, MINB) invert_stream_kernel(
    const __grid_constant__ GridParams<MULTI ? PMK_MAX_GRIDS : 1> GS, const PmStreamIO sio) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NG = MULTI ? PMK_MAX_GRIDS : 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  BlockSmem<R>* bs = reinterpret_cast<BlockSmem<R>*>(smem_raw);
  using SM = WarpSmem<R, MAC || ZM>;
  SM& sm = reinterpret_cast<SM*>(smem_raw + NG * sizeof(BlockSmem<R>))[warp];
#pragma unroll 1
  for (int g = 0; g < NG && g < GS.ngrids; ++g) load_taps<R>(GS.g[g], bs[g]);
  __syncthreads();
  if (lane == 0) {
    sm.job_k = sio.first_job;
    sm.grid_cur = -1;  // grid of the previous pixel: the padded rows are re-zeroed on a change
  }
  __syncwarp();
  while (true) {
    long long t = 0;
    if (lane == 0) t = next_ticket(sio.q, sio.wait_limit_ns);
    t = __shfl_sync(kFull, t, 0);
    if (t < 0) break;
    // the job of ticket t: jobs are appended in ticket order, so it is at or
    // after this warp's previous one
    const PmJob* jp = nullptr;
    unsigned long long t0 = 0;
    long long k = sm.job_k;
    for (int guard = 0; guard <= sio.jobs_cap; ++guard, ++k) {
      const PmJob* c = sio.jobs + (k % sio.jobs_cap);
      const unsigned long long c0 = __ldcg(&c->t0);
      const unsigned long long cn = __ldcg(reinterpret_cast<const unsigned long long*>(&c->npix));
      if ((unsigned long long)t >= c0 && (unsigned long long)t < c0 + cn) {
        jp = c;
        t0 = c0;
        break;
      }
    }
    if (!jp) {
      if (lane == 0) atomicExch(&sio.q->err, (unsigned long long)PMQ_ERR_JOB);
      break;
    }
    const int gi = MULTI ? __ldcg(&jp->grid) : 0;
    const PmParams& P = GS.g[gi];
    if (gi != sm.grid_cur) {
      for (int e = lane; e < 4 * XSR; e += 32) (&sm.xs[0][0])[e] = R(0);
      __syncwarp();
      if (lane == 0) {
        sm.grid_cur = gi;
        sm.xs_dirty = 0;
      }
    }
    if (lane == 0) {
      sm.job_k = k;
      sm.job = jp;
      sm.pix = (unsigned long long)t - t0;
    }
    __syncwarp();
    invert_pixel<R, KT, MAC, PIXGRID, ZM>(P, bs[gi], sm, lane, sio.q->ctr);
    job_pixel_done(sm, lane);
  }
}


template <typename R, int KT, int MINB, bool MULTI, bool MAC, bool PIXGRID = false, bool ZM = false>
int launch_invert_stream(const PmGridSet& GS, const PmStreamIO& sio, cudaStream_t st, int num_sms,
                         size_t* smem_out, int wpb, int reserve) {
  if (wpb > 4) wpb = 4;  // at most 4 warps per block
  const int threads = 32 * wpb;
  const size_t smem = (MULTI ? PMK_MAX_GRIDS : 1) * sizeof(BlockSmem<R>) + sizeof(WarpSmem<R, MAC || ZM>) * (threads / 32);
  if (smem_out) *smem_out = smem;
  auto kern = invert_stream_kernel<R, KT, MINB, MULTI, MAC, PIXGRID, ZM>;
  constexpr int NG = MULTI ? PMK_MAX_GRIDS : 1;
  GridParams<NG> gp;  // copied into the launch
  gp.ngrids = GS.ngrids < NG ? GS.ngrids : NG;
  for (int g = 0; g < gp.ngrids; ++g) gp.g[g] = GS.g[g];
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess) return snprintf(pmk_g_err, sizeof pmk_g_err, "%s", cudaGetErrorString(e)), PM_EIO;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  if (e != cudaSuccess || per_sm < 1) return snprintf(pmk_g_err, sizeof pmk_g_err, "occupancy: %s", cudaGetErrorString(e)), PM_EIO;
  const int blocks = per_sm * num_sms - reserve > 1 ? per_sm * num_sms - reserve : 1;
  kern<<<unsigned(blocks), threads, smem, st>>>(gp, sio);
  e = cudaGetLastError();
  if (e != cudaSuccess) return snprintf(pmk_g_err, sizeof pmk_g_err, "stream launch: %s", cudaGetErrorString(e)), PM_EIO;
  return PM_OK;
}

}  // namespace
