// Whole runs of whole-box systems in one launch: k_run_box advances each system
// of an engine any number of steps inside one thread-block cluster.
//
// A step of such a system (a few thousand particles) is a few microseconds of
// arithmetic on one cluster; as separate kernels it is bound by launches, the
// graph's conditional node and a dozen dependent round trips to L2 (39 us at
// N = 1000).  Here a cluster of C blocks holds the system for the whole call:
//
//   * every block stages all positions in its shared memory (FP32: 32-bit fixed
//     point, FP64: doubles) and owns a run of slots, whose state stays in its
//     shared memory where that fits (else in L2);
//   * kick/drift: each block moves its slots, writes the new positions as staged
//     to memory and its largest displacement into every block (distributed
//     shared memory); cluster barrier; every block takes the same rebuild
//     decision and reads all positions (1400 cycles at N = 1000 and 3000 at N =
//     4000, FP64, where storing them into the other 15 blocks took 2000 and 6400:
//     one read is wide and coalesced, the remote stores are neither);
//   * forces from the lists (kept in shared memory where they fit), second half
//     kick, sums per 32 slots stored into every block; cluster barrier; every
//     block adds them up in the same order and runs the thermostat chain.
//
// Two cluster barriers and one exchange through L2 a step, where the state is
// resident.  Clusters are co-scheduled by the hardware and wait on nothing
// but their own barrier, so systems are independent: a batch runs one cluster
// per system, largest first, and no system waits for another's rebuild.  A list
// rebuild happens inside the cluster: every block sorts the system by cell (a
// stable counting sort over original indices, which gives the reference's
// InCell order) and by list sub-cell in its shared memory, so it takes two more
// cluster barriers (a third where a list overflows).
//
// What bounds it: the latency of a step's dependent phases for a lone system
// (16 of 148 SMs busy), the issue rate of the pair terms for a batch.  Measured
// on B200 against the kernel-by-kernel graphs it replaced, in calls of 64 steps of
// a system just off the lattice: N = 1000 FP64 39.0 -> 14.3 us a step, N = 4000
// FP64 60 -> 36, 256 FP32 replicas 400 -> 245; of settled systems N = 1000 13.5 us
// (FP32 11.5), N = 4000 25.7 (20.0).  What it does worse than the kernels: a call
// of a few steps of many systems, whose length is that of the slowest list rebuild
// (such calls take the kernels).
//
// Sums, lists and particle order are those of the kernel-by-kernel step, so a
// system's results are the same bits whichever path, cluster size or residency
// it runs with.
#pragma once
#include <cooperative_groups.h>

#include "acg_kernels.cuh"

namespace acg {
namespace cg = cooperative_groups;

constexpr int RUN_MAX_CLUSTER = 16;
constexpr int RUN_STATE_BYTES = 32 + 12 * 8 + 2 * 4;  // position, u, v, F, o, id, act
constexpr size_t RUN_SMEM_MAX = 219 * 1024;           // dynamic; the static arrays take 7 KB of the 227

__host__ __device__ __forceinline__ size_t run_align(size_t x) { return (x + 15) & ~(size_t)15; }

// shared-memory plan of one system on a cluster of C blocks of nw warps (byte offsets)
struct RunPlan {
  int nseg, nloc;       // 32-slot segments; slots per block
  size_t seg8, nn, state;  // this block's sums per 8 slots, list lengths and slots' state (none when not resident)
  size_t pool;          // staging and list cache, or the rebuild's scratch
  size_t stage_bytes, scratch_bytes, perm_bytes;
  size_t lists_at;      // in the scratch: the sorts' arrays, then the list buffers
  // the least dynamic shared memory
  __host__ __device__ size_t least() const {
    return pool + (stage_bytes > scratch_bytes ? stage_bytes : scratch_bytes) + perm_bytes;
  }
};
__host__ __device__ __forceinline__ RunPlan run_plan(int n, int ncell, int msub, int prec, int C, bool resident, int nw) {
  RunPlan p;
  p.nseg = (n + 31) / 32;
  p.nloc = 32 * ((p.nseg + C - 1) / C);
  p.seg8 = run_align(32 * (size_t)p.nseg);
  p.nn = p.seg8 + 4 * (size_t)p.nloc;
  p.state = p.nn + 4 * (size_t)p.nloc;
  p.pool = p.state + (resident ? run_align((size_t)RUN_STATE_BYTES * p.nloc) : 0);
  p.stage_bytes = run_align((size_t)n * (prec ? 12 : 24));
  const size_t m3 = (size_t)msub * msub * msub, hist = 64 * (size_t)ncell, xs = 16 * (size_t)n;
  // the sorted candidates (or the cell sort's per-warp counts and cell starts)
  // and the sub-cell starts; then the sorts' keys, orders and counts or, once
  // those are done, the list buffers of as many warps as there is room for (at
  // least half of them)
  const size_t sort = 2 * run_align(2 * (size_t)n) + run_align(4 * m3), lists = sizeof(BrickScratch) * (nw / 2);
  p.lists_at = run_align(xs > hist + 4 * (size_t)ncell ? xs : hist + 4 * (size_t)ncell) + run_align(4 * (m3 + 1));
  p.scratch_bytes = p.lists_at + (sort > lists ? sort : lists);
  p.perm_bytes = run_align(2 * (size_t)n);
  return p;
}

// the per-slot state arrays of a system's run, in global memory (index: slot of
// the engine) or in a block's shared memory (index: slot of the block)
struct RunState {
  double4 *pos;
  double *ux, *uy, *uz, *vx, *vy, *vz, *fx, *fy, *fz, *ox, *oy, *oz;
  int *id, *act;
  const char4 *kdir;
};
// in shared memory: built from the shared array alone (a copy of the kernel's
// View with pointers replaced does not do: the compiler takes the pointers of
// a by-value kernel parameter to be global ones)
__device__ __forceinline__ RunState run_resident(unsigned char *sm, int nloc, const char4 *kdir) {
  RunState w;
  w.pos = reinterpret_cast<double4 *>(sm);
  double *f = reinterpret_cast<double *>(sm + 32 * (size_t)nloc);
  w.ux = f, w.uy = f + nloc, w.uz = f + 2 * nloc;
  w.vx = f + 3 * nloc, w.vy = f + 4 * nloc, w.vz = f + 5 * nloc;
  w.fx = f + 6 * nloc, w.fy = f + 7 * nloc, w.fz = f + 8 * nloc;
  w.ox = f + 9 * nloc, w.oy = f + 10 * nloc, w.oz = f + 11 * nloc;
  w.id = reinterpret_cast<int *>(f + 12 * nloc);
  w.act = w.id + nloc;
  w.kdir = kdir;
  return w;
}
__device__ __forceinline__ RunState run_global(const View &v) {
  return RunState{v.pos, v.ux, v.uy, v.uz, v.vx, v.vy, v.vz, v.fx, v.fy, v.fz, v.ox, v.oy, v.oz, v.id, v.act, v.kdir};
}
// the permuted state of a rebuild, beside the present one (no ox, oy, oz)
__device__ __forceinline__ RunState run_scratch(const View &v) {
  return RunState{v.pos_s, v.ux_s, v.uy_s, v.uz_s, v.vx_s, v.vy_s, v.vz_s, v.fx_s, v.fy_s, v.fz_s,
                  nullptr, nullptr, nullptr, v.id_s, v.act_s, v.kdir};
}

// slot i of `to` = slot j of `from`
__device__ __forceinline__ void run_copy_slot(const RunState &to, int i, const RunState &from, int j) {
  to.pos[i] = from.pos[j];
  to.ux[i] = from.ux[j];
  to.uy[i] = from.uy[j];
  to.uz[i] = from.uz[j];
  to.vx[i] = from.vx[j];
  to.vy[i] = from.vy[j];
  to.vz[i] = from.vz[j];
  to.fx[i] = from.fx[j];
  to.fy[i] = from.fy[j];
  to.fz[i] = from.fz[j];
  to.id[i] = from.id[j];
  to.act[i] = from.act[j];
}
// the position at the last rebuild: of another state, or the present one
__device__ __forceinline__ void run_copy_old(const RunState &to, int i, const RunState &from, int j) {
  to.ox[i] = from.ox[j];
  to.oy[i] = from.oy[j];
  to.oz[i] = from.oz[j];
}
__device__ __forceinline__ void run_fresh_old(const RunState &w, int i) {
  w.ox[i] = w.ux[i];
  w.oy[i] = w.uy[i];
  w.oz[i] = w.uz[i];
}

template <int PREC>
__device__ __forceinline__ void run_stage(unsigned char *stg, int n, int s, const double4 &p) {
  if (PREC == 1) {
    int *q = reinterpret_cast<int *>(stg);
    q[s] = fixed32(p.x);
    q[n + s] = fixed32(p.y);
    q[2 * n + s] = fixed32(p.z);
  } else {
    double *q = reinterpret_cast<double *>(stg);
    q[s] = p.x;
    q[n + s] = p.y;
    q[2 * n + s] = p.z;
  }
}

// perm[new slot] = old slot, by cell and inside a cell by original index (the
// order of k_cells_order), by all threads of the block.  Every warp takes a run
// of original indices and counts its particles per cell, the counts are
// scanned over (cell, warp), and every warp places its run in index order.
// key, inv [n], hist [warps][ncell] and base [ncell] are scratch; `publish`:
// store the cells' starts and counts for the other kernels.
__device__ __forceinline__ void run_sort_cells(const View &v, const SysDesc &d, uint16_t *perm, uint16_t *key,
                                               uint16_t *inv, uint16_t *hist, int *base, bool publish) {
  const int n = d.n, nc = d.nc, ncell = d.ncell;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int k = threadIdx.x; k < ncell * nw; k += blockDim.x) hist[k] = 0;
  for (int s = threadIdx.x; s < n; s += blockDim.x) {
    const double4 p = v.pos[d.poff + s];
    key[s] = (uint16_t)(cell_coord(p.x, d.inv_cell, nc) + cell_coord(p.y, d.inv_cell, nc) * nc +
                        cell_coord(p.z, d.inv_cell, nc) * nc * nc);
    inv[v.id[d.poff + s]] = (uint16_t)s;
  }
  __syncthreads();
  const int run = (((n + 31) / 32 + nw - 1) / nw) * 32, k0 = warp * run, k1 = min(n, k0 + run);
  uint16_t *h = hist + (size_t)warp * ncell;
  for (int q = k0; q < k1; q += 32) {
    const bool valid = q + lane < k1;
    const int c = valid ? key[inv[q + lane]] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, c);
    if (valid && lane == __ffs(same) - 1) h[c] += (uint16_t)__popc(same);
    __syncwarp();
  }
  __syncthreads();
  for (int c = threadIdx.x; c < ncell; c += blockDim.x) {
    int m = 0;
    for (int w = 0; w < nw; w++) m += hist[(size_t)w * ncell + c];
    base[c] = m;
  }
  __syncthreads();
  if (warp == 0) {  // exclusive scan of the cells' counts
    int before = 0;
    for (int c0 = 0; c0 < ncell; c0 += 32) {
      const int c = c0 + lane, m = c < ncell ? base[c] : 0;
      int x = m;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (c < ncell) {
        base[c] = before + x - m;
        if (publish) {
          v.cstart[d.coff + c] = before + x - m;
          v.ccount[d.coff + c] = m;
        }
      }
      before += __shfl_sync(0xffffffffu, x, 31);
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < ncell; c += blockDim.x) {
    int at = base[c];
    for (int w = 0; w < nw; w++) {
      const int m = hist[(size_t)w * ncell + c];
      hist[(size_t)w * ncell + c] = (uint16_t)at;
      at += m;
    }
  }
  __syncthreads();
  for (int q = k0; q < k1; q += 32) {
    const bool valid = q + lane < k1;
    const int s = valid ? inv[q + lane] : 0;
    const int c = valid ? key[s] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, c);
    if (valid) perm[h[c] + __popc(same & ((1u << lane) - 1u))] = (uint16_t)s;
    __syncwarp();
    if (valid && lane == __ffs(same) - 1) h[c] += (uint16_t)__popc(same);
    __syncwarp();
  }
  __syncthreads();
}

template <int TPP, int PREC, int NT, bool RES>
__global__ void __launch_bounds__(NT, 1) k_run_box(View v, const int *order, int nsteps, unsigned smem_bytes) {
  extern __shared__ __align__(16) unsigned char rsm[];
  __shared__ SysState ss;
  __shared__ SysDesc sd;
  __shared__ double s_wmax[32], s_cmax[RUN_MAX_CLUSTER];
  __shared__ double s_obs[OBS_EMAX][OBS_NV];
  __shared__ NhcHalf s_half;
  __shared__ int s_nnmax, s_brick;
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int r = order[blockIdx.x / C];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = NT / 32;
  auto bar = [&]() {
    if (C > 1) cl.sync();
    else __syncthreads();
  };
  copy_struct(&ss, &v.st[r]);
  copy_struct(&sd, &v.desc[r]);
  __syncthreads();
  const int n = sd.n, poff = sd.poff;
  const RunPlan P = run_plan(n, sd.ncell, sd.msub, PREC, C, RES, NW);
  const int lo = rank * P.nloc, hi = max(lo, min(n, lo + P.nloc)), own = hi - lo;
  const int lo_seg = rank * (P.nloc / 32), nseg_own = max(0, min(P.nseg - lo_seg, P.nloc / 32));
  double4 *seg = reinterpret_cast<double4 *>(rsm), *seg8 = reinterpret_cast<double4 *>(rsm + P.seg8);
  int *nn_own = reinterpret_cast<int *>(rsm + P.nn);
  unsigned char *stg = rsm + P.pool;
  uint16_t *perm = reinterpret_cast<uint16_t *>(rsm + smem_bytes - P.perm_bytes);
  uint2 *cache = reinterpret_cast<uint2 *>(stg + P.stage_bytes);
  const size_t cache_bytes = smem_bytes - P.perm_bytes - P.pool - P.stage_bytes;
  // the block's state: w with index k + wb for slot k of the system
  const RunState g = run_global(v), w = RES ? run_resident(rsm + P.state, P.nloc, v.kdir) : g;
  const int wb = RES ? -lo : poff;
  const uint2 *lists = reinterpret_cast<const uint2 *>(box_list(v, sd));
  // the step's new positions as staged, for the other blocks (the download
  // buffer, free while the system steps)
  unsigned char *shared_pos = reinterpret_cast<unsigned char *>(v.stage_f + 3 * (size_t)poff);
  bool cached = false;

  // list lengths of the block's slots, and their lists where they fit in the cache
  auto take_lists = [&]() {
    if (tid == 0) s_nnmax = 0;
    __syncthreads();
    int most = 0;
    for (int k = tid; k < own; k += NT) {
      const int nn = v.nbn[poff + lo + k];
      nn_own[k] = nn;
      most = max(most, nn);
    }
    for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
    if (lane == 0 && most > 0) atomicMax(&s_nnmax, most);
    __syncthreads();
    const int nch = (s_nnmax + 3) >> 2;
    cached = (size_t)nch * own * sizeof(uint2) <= cache_bytes;
    if (cached)
      for (int q = tid; q < nch * own; q += NT) cache[q] = lists[(size_t)(q / own) * n + lo + q % own];
    __syncthreads();
  };

  if (RES)
    for (int k = lo + tid; k < hi; k += NT) {
      run_copy_slot(w, wb + k, g, poff + k);
      run_copy_old(w, wb + k, g, poff + k);
    }
  for (int s = tid; s < n; s += NT) run_stage<PREC>(stg, n, s, v.pos[poff + s]);
  take_lists();

  // the same in every thread of the cluster: step counter and schedules,
  // list overflow (then every block keeps its positions in global memory too)
  long long ramp = ss.ramp_left;
  const int tau = (sd.shuffle == 1 && sd.nact > 0 && sd.tau_p > 0) ? sd.tau_p : 0;
  int shuf_at = tau ? (int)(ss.step % tau) : 0, drift_at = sd.drift_every > 0 ? (int)(ss.step % sd.drift_every) : 0;
  int ovf = ss.overflow, forced = ss.force_rebuild;
  const ObsDesc &ob = v.obs[r];
  long long obs_next = 0;  // thread 0: step of the next observable event
  if (tid == 0) obs_next = ss.obs_cur < ob.n_events ? ob.ev_step[ss.obs_cur] : 0x7fffffffffffffffll;
  bar();  // every block of the cluster runs and is staged

  for (int it = 0; it < nsteps; it++) {
    const bool shuf = tau && ramp == 0 && shuf_at == 0;
    // ---- kick and drift of the block's slots
    if (tid == 0) {
      ss.shuf = shuf;
      ss.drift = sd.drift_every > 0 && ramp == 0 && drift_at == 0;
      ss.obs_lo = ss.obs_hi = 0;
      if (ramp == 0 && ss.step >= obs_next) {
        obs_due(ob, ss);
        obs_next = ss.obs_cur < ob.n_events ? ob.ev_step[ss.obs_cur] : 0x7fffffffffffffffll;
      }
    }
    double far = 0.0;
    for (int k = lo + tid; k < hi; k += NT) {
      far = fmax(far, kick_drift_one(w, sd, ss, wb + k));
      const double4 p = w.pos[wb + k];
      run_stage<PREC>(C > 1 ? shared_pos : stg, n, k, p);
      if (ovf && RES) v.pos[poff + k] = p;
    }
    for (int o = 16; o > 0; o >>= 1) far = fmax(far, __shfl_xor_sync(0xffffffffu, far, o));
    if (lane == 0) s_wmax[warp] = far;
    __syncthreads();
    // the largest displacement to every block
    if (warp == 0) {
      far = lane < NW ? s_wmax[lane] : 0.0;
      for (int o = 16; o > 0; o >>= 1) far = fmax(far, __shfl_xor_sync(0xffffffffu, far, o));
      if (lane < C) *cl.map_shared_rank(&s_cmax[rank], lane) = far;
    }
    bar();
    // ---- rebuild decision (rebuild_decision's), the same in every thread
    far = (lane & 15) < C ? s_cmax[lane & 15] : 0.0;
    for (int o = 8; o > 0; o >>= 1) far = fmax(far, __shfl_xor_sync(0xffffffffu, far, o));
    const double m2 = __dmul_rn(__dmul_rn(far, sd.L), sd.L);
    const bool rebuild = (__dmul_rn(sd.rebuild_factor, m2) > sd.skin2) || forced;
    forced = 0;
    if (tid == 0) {
      ss.maxD_last = m2;
      ss.rebuild = rebuild;
      ss.force_rebuild = 0;
    }
    if (!rebuild && C > 1) {  // every block's new positions
      const uint4 *from = reinterpret_cast<const uint4 *>(shared_pos);
      uint4 *to = reinterpret_cast<uint4 *>(stg);
      const int words = 3 * n * (PREC ? 4 : 8) / 4;
      for (int q = tid; q < words / 4; q += NT) to[q] = __ldcg(from + q);
      if (tid < words % 4)
        reinterpret_cast<unsigned *>(stg)[words / 4 * 4 + tid] =
            __ldcg(reinterpret_cast<const unsigned *>(shared_pos) + words / 4 * 4 + tid);
      __syncthreads();
    }
    if (rebuild) {
      const int m3 = sd.msub * sd.msub * sd.msub;
      float4 *xs = reinterpret_cast<float4 *>(stg);
      uint16_t *hist = reinterpret_cast<uint16_t *>(stg);
      int *sst = reinterpret_cast<int *>(stg + P.lists_at - run_align(4 * (size_t)(m3 + 1)));
      uint16_t *key = reinterpret_cast<uint16_t *>(stg + P.lists_at);
      uint16_t *ord = reinterpret_cast<uint16_t *>(stg + P.lists_at + run_align(2 * (size_t)n));
      int *fill = reinterpret_cast<int *>(stg + P.lists_at + 2 * run_align(2 * (size_t)n));
      BrickScratch *buf = reinterpret_cast<BrickScratch *>(stg + P.lists_at);
      if (RES) {  // the state in global memory, for the blocks that take over its slots
        for (int k = lo + tid; k < hi; k += NT) run_copy_slot(g, poff + k, w, wb + k);
      }
      if (tid == 0) {
        ss.rebuilds += 1;
        s_brick = 0;
        if (rank == 0) v.st[r].overflow = 0;
      }
      bar();
      run_sort_cells(v, sd, perm, key, ord, hist, reinterpret_cast<int *>(hist + (size_t)NW * sd.ncell), rank == 0);
      if (RES) {
        for (int k = lo + tid; k < hi; k += NT) {
          run_copy_slot(w, wb + k, g, poff + perm[k]);
          run_fresh_old(w, wb + k);
        }
      } else {
        const RunState t = run_scratch(v);
        for (int k = lo + tid; k < hi; k += NT) run_copy_slot(t, poff + k, g, poff + perm[k]);
      }
      sort_sub_cells(n, sd.msub, [&](int s) { return v.pos[poff + perm[s]]; }, fill, sst, key, ord, xs);
      __syncthreads();
      // lists, one brick of sub-cells a warp: the smaller ones where the cluster
      // has warps to spare, else as many lanes of a sweep in use as fit
      const int bx = C > 1 ? 2 : sd.bx_wide, nb = bricks_of(sd, bx, sd.bz);
      const int lw = min(NW, (int)((smem_bytes - P.perm_bytes - P.pool - P.lists_at) / sizeof(BrickScratch)));
      if (C > 1) {
        if (warp < lw)
          for (int q = warp * C + rank; q < nb; q += C * lw)
            box_list_brick(v, sd, r, xs, sst, q, bx, sd.bz, lane, buf[warp]);
      } else if (warp < lw) {  // several bricks a warp: handed out as warps come free
        for (int q = warp_next(s_brick); q < nb; q = warp_next(s_brick))
          box_list_brick(v, sd, r, xs, sst, q, bx, sd.bz, lane, buf[warp]);
      }
      __syncthreads();
      for (int s = tid; s < n; s += NT) run_stage<PREC>(stg, n, s, v.pos[poff + perm[s]]);
      bar();
      if (!RES)
        for (int k = lo + tid; k < hi; k += NT) copy_back(v, poff + k);
      ovf = *reinterpret_cast<volatile int *>(&v.st[r].overflow);
      if (ovf && RES)
        for (int k = lo + tid; k < hi; k += NT) v.pos[poff + k] = w.pos[wb + k];
      take_lists();
      if (ovf) bar();
    }
    // ---- direction shuffle and observables
    if (shuf) {
      unsigned int *mt = v.mt + (size_t)r * 2 * MT_WORDS;
      for (int c = 0; c < 3; c++)
        if (c % C == rank) {
          shuffle_ref_component(v, r, c, mt + (size_t)ss.mt_cur * MT_WORDS, mt + (size_t)(ss.mt_cur ^ 1) * MT_WORDS,
                                reinterpret_cast<signed char *>(rsm), P.seg8);
          __syncthreads();
        }
    }
    const int ob_lo = ss.obs_lo, ob_hi = ss.obs_hi;
    double *part = v.stage_d + 9 * (size_t)poff;  // [segment][event][sum], free while the system steps
    for (int e = ob_lo; e < ob_hi; e++) {
      const int info = ob.ev_info[e];
      for (int q = warp; q < nseg_own; q += NW) {
        const int k = lo + 32 * q + lane;
        double val[OBS_NV] = {0.0, 0.0, 0.0, 0.0, 0.0};
        if (k < n) {
          const int i = wb + k;
          obs_particle(ob, n, info, w.id[i], w.ux[i], w.uy[i], w.uz[i], sd.L, val);
        }
        if ((info & 1) == 0) {
#pragma unroll
          for (int c = 0; c < OBS_NV; c++) {
            double x = val[c];
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            if (lane == 0) part[((size_t)(lo_seg + q) * OBS_EMAX + (e - ob_lo)) * OBS_NV + c] = x;
          }
        }
      }
    }
    if (shuf || ob_hi > ob_lo) bar();
    if (ob_hi > ob_lo && rank == 0) {
      // the order of k_observe: 32 slots, eight of those to a tile, the tiles
      const int nev = ob_hi - ob_lo;
      if (tid < nev * OBS_NV && (ob.ev_info[ob_lo + tid / OBS_NV] & 1) == 0) {
        double sum = 0.0;
        for (int b = 0; b < P.nseg; b += 8) {
          double x = 0.0;
          for (int q = b; q < min(b + 8, P.nseg); q++)
            x += part[((size_t)q * OBS_EMAX + tid / OBS_NV) * OBS_NV + tid % OBS_NV];
          sum += x;
        }
        s_obs[tid / OBS_NV][tid % OBS_NV] = sum;
      }
      __syncthreads();
      if (tid < nev && (ob.ev_info[ob_lo + tid] & 1) == 0) obs_accumulate(ob, n, ob.ev_info[ob_lo + tid], s_obs[tid]);
    }
    // ---- forces, second half kick, sums per 8 and per 32 slots
    const bool nose = sd.thermostat == 1 && ramp == 0 && ss.loaded;
    if (nose && tid == NT - 32) s_half = nhc_before(ss.p_eta_cur, sd.rq, sd.T, sd.dt);
    for (int b = warp * (32 / TPP); b < 32 * nseg_own; b += NT / TPP) {
      const int k = b + lane / TPP;
      const bool valid = k < own;
      const int sl = lo + (valid ? k : 0);
      const PairAcc a = box_pairs<TPP, PREC>(v, sd, stg, cached ? cache + (sl - lo) : lists + sl,
                                             (size_t)(cached ? own : n), valid ? nn_own[k] : 0, valid, sl, poff + sl,
                                             valid ? (int)w.pos[wb + sl].w : 0, lane % TPP);
      double4 q = make_double4(0.0, 0.0, 0.0, 0.0);
      if (valid && lane % TPP == 0) particle_epilogue(w, sd, ss, wb + sl, 0, a, q.x, q.y, q.z, q.w);
#pragma unroll
      for (int o = TPP; o < 8 * TPP; o <<= 1) q = xor4(q, o);
      if (lane % (8 * TPP) == 0) seg8[k >> 3] = q;
    }
    __syncthreads();
    for (int q = tid; q < nseg_own * C; q += NT) {
      const double4 *s8 = seg8 + 4 * (q % nseg_own);
      *cl.map_shared_rank(&seg[lo_seg + q % nseg_own], q / nseg_own) = add4(add4(s8[0], s8[1]), add4(s8[2], s8[3]));
    }
    bar();
    // ---- system sums and thermostat, the same in every block.  A Nose-Hoover
    // step's chain, the longest chain of dependent operations of a small system's
    // step, is one warp's, the part of it that needs no sums computed beforehand
    // by another; a third adds up the energies (finalize_sums' operations)
    if (nose) {
      if (warp == 0) {
        double k2 = 0.0;
        for (int q = lane; q < P.nseg; q += 32) k2 += seg[q].z;
        for (int o = 16; o > 0; o >>= 1) k2 += __shfl_xor_sync(0xffffffffu, k2, o);
        if (lane == 0) {
          double eta[NHC_M], pet[NHC_M];
          for (int k = 0; k < NHC_M; k++) {
            eta[k] = ss.eta_cur[k];
            pet[k] = ss.p_eta_cur[k];
          }
          const double s2 = nhc_after(s_half, eta, pet, sd.rq, sd.T, sd.dof, sd.dt, k2);
          const double kb = (s2 * s2) * k2;
          for (int k = 0; k < NHC_M; k++) {
            ss.eta_end[k] = eta[k];
            ss.p_eta_end[k] = pet[k];
          }
          ss.s1 = nhc_half(eta, pet, sd.rq, sd.T, sd.dof, sd.dt, kb);
          ss.s2 = s2;
          for (int k = 0; k < NHC_M; k++) {
            ss.eta_cur[k] = eta[k];
            ss.p_eta_cur[k] = pet[k];
          }
          ss.ke_end = kb * 0.5;
          if (!(k2 == k2) || k2 > 1.0e300) ss.status = 1;
        }
      } else if (warp == 1) {
        double4 t = total_of_segments(seg, P.nseg);
        if (lane == 0) {
          ss.pe = 0.5 * t.x;
          ss.virial = (0.5 * t.y) / 3.0;
          ss.vir_act = t.w;
          ss.step += 1;
          if (shuf) {
            ss.mt_cur ^= 1;
            ss.shuf = 0;
          }
          ss.prime = 0;
        }
      }
    } else if (warp == 0) {
      const double4 t = total_of_segments(seg, P.nseg);
      if (lane == 0) finalize_sums(sd, ss, sd, 0, t.x, t.y, t.z, t.w);
    }
    __syncthreads();
    if (ramp > 0) {
      ramp--;
    } else {
      if (++shuf_at >= tau) shuf_at = 0;
      if (++drift_at >= sd.drift_every) drift_at = 0;
    }
  }
  if (RES)
    for (int k = lo + tid; k < hi; k += NT) {
      run_copy_slot(g, poff + k, w, wb + k);
      run_copy_old(g, poff + k, w, wb + k);
    }
  if (rank == 0) {
    if (tid == 0) ss.overflow = ovf;
    __syncthreads();
    copy_struct(&v.st[r], &ss);
  }
}

}  // namespace acg
