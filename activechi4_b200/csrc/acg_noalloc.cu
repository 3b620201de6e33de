// Allocation-free force evaluation: acg_forces_noalloc (include/activechi4.h).
//
// Some callers cannot call cudaMalloc: code that runs inside a framework that
// owns all device memory through its own pool, hosts that forbid allocation
// after start-up (real-time or latency-bounded loops), and plug-ins that only
// receive device pointers from their host.  For them this entry point
// evaluates the pair + active forces of one system from device arrays the
// caller owns, keeping every intermediate (cell of each particle, cell counts,
// starts and fill cursors, cell-ordered particle indices, per-block partial
// sums, the last-block counter) in one fixed file-scope device array,
// acg_noalloc_scratch, instead of allocating.  Every GPU that loads the
// library holds that array (ACG_NOALLOC_SCRATCH_BYTES) until the process
// exits.
//
// All calls share the array and it keeps the last call's contents; whatever
// must start at zero is cleared at the start of each call.  Calls whose work
// overlaps on the GPU (different streams, or different host threads on one
// device) race on the array and must be serialised by the caller.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <string>

#include "../../include/activechi4.h"
#include "acg_device.cuh"

namespace acg {
int set_last_error(int code, const std::string &msg);  // acg_engine.cu: the text acg_last_error returns
}

namespace {

constexpr int NA_BLOCK = 256;
constexpr int NA_WARPS = NA_BLOCK / 32;
constexpr int NA_MAX_BLOCKS = 8192;  // force blocks (each takes every NA_MAX_BLOCKS-th cell)
// candidates of a cell's neighbourhood staged in shared memory at a time: at
// density 1.2 a neighbourhood of 27 cells holds 750 to 2000 (most where few
// cells share a box not much under one cell more per side); with 40 bytes each
// four blocks of eight warps share an SM
constexpr int NA_CAP = 1280;
constexpr int NA_FILL = 592;  // blocks that fill the 148 SMs
// below this many particles a cell, on grids of at least this many cells, the
// forces go particle by particle (us a call, by cells / by particles: 14 to 17
// cells per side 89 / 49 at one particle a cell, 57 / 50 at 2.4, 80 / 68 at 4.1,
// 74 / 74 at 4.9; 12 per side, all of whose cells fit on the chip in three waves,
// 37 / 41 at 1.2; the larger grids lie between: 27 per side 161 / 59 at one, 234 /
// 235 at 5.1)
constexpr int NA_SPARSE = 4, NA_SPARSE_CELLS = 14 * 14 * 14;
constexpr size_t NA_SMEM = (size_t)NA_CAP * (sizeof(float4) + 3 * sizeof(double));

// scratch layout (bytes): cell_of[N] order[N] ccount[C] cstart[C] cfill[C]
// partials[B][4] counter
constexpr size_t OFF_CELL = 0;
constexpr size_t OFF_ORDER = OFF_CELL + 4ull * ACG_NOALLOC_MAX_N;
constexpr size_t OFF_COUNT = OFF_ORDER + 4ull * ACG_NOALLOC_MAX_N;
constexpr size_t OFF_START = OFF_COUNT + 4ull * ACG_NOALLOC_MAX_CELLS;
constexpr size_t OFF_FILL = OFF_START + 4ull * ACG_NOALLOC_MAX_CELLS;
constexpr size_t OFF_PART = (OFF_FILL + 4ull * ACG_NOALLOC_MAX_CELLS + 255) / 256 * 256;
constexpr size_t OFF_CTR = OFF_PART + 32ull * NA_MAX_BLOCKS;
constexpr size_t SCRATCH_BYTES = (OFF_CTR + 256 + 255) / 256 * 256;
static_assert(SCRATCH_BYTES <= ACG_NOALLOC_SCRATCH_BYTES, "scratch layout exceeds the stated size");

}  // namespace

static __device__ __align__(256) unsigned char acg_noalloc_scratch[ACG_NOALLOC_SCRATCH_BYTES];

namespace {

std::mutex na_mu;
void *na_ptr[256];  // device address of the scratch array, per device

int na_fail(int code, const std::string &m) { return acg::set_last_error(code, m); }

struct NaArgs {
  const double *x, *xu;
  const int *type, *act, *k;
  double *F, *out;
  unsigned char *scr;
  int n, nact, nc;
  double L, inv_cell, f0;
};

__device__ __forceinline__ int *na_i(const NaArgs &a, size_t off) { return (int *)(a.scr + off); }

__global__ void k_na_clear(NaArgs a) {
  const int ncell = a.nc * a.nc * a.nc;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += gridDim.x * blockDim.x) {
    na_i(a, OFF_COUNT)[c] = 0;
    na_i(a, OFF_FILL)[c] = 0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *(unsigned int *)(a.scr + OFF_CTR) = 0u;
}

__global__ void k_na_count(NaArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const int cx = acg::cell_coord(a.x[3 * i], a.inv_cell, a.nc);
  const int cy = acg::cell_coord(a.x[3 * i + 1], a.inv_cell, a.nc);
  const int cz = acg::cell_coord(a.x[3 * i + 2], a.inv_cell, a.nc);
  const int c = cx + cy * a.nc + cz * a.nc * a.nc;
  na_i(a, OFF_CELL)[i] = c;
  atomicAdd(&na_i(a, OFF_COUNT)[c], 1);
}

__global__ void k_na_scan(NaArgs a) {
  __shared__ int sh[1024];
  const int ncell = a.nc * a.nc * a.nc, B = blockDim.x;
  const int chunk = (ncell + B - 1) / B;
  const int beg = min((int)threadIdx.x * chunk, ncell), end = min(beg + chunk, ncell);
  int sum = 0;
  for (int c = beg; c < end; c++) sum += na_i(a, OFF_COUNT)[c];
  sh[threadIdx.x] = sum;
  __syncthreads();
  for (int o = 1; o < B; o <<= 1) {
    int v = threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
    __syncthreads();
    sh[threadIdx.x] += v;
    __syncthreads();
  }
  int run = sh[threadIdx.x] - sum;
  for (int c = beg; c < end; c++) {
    na_i(a, OFF_START)[c] = run;
    run += na_i(a, OFF_COUNT)[c];
  }
}

__global__ void k_na_scatter(NaArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const int c = na_i(a, OFF_CELL)[i];
  const int slot = na_i(a, OFF_START)[c] + atomicAdd(&na_i(a, OFF_FILL)[c], 1);
  na_i(a, OFF_ORDER)[slot] = i;
}

// the block's sums (pe, virial, active virial; one triple a warp, from lane 0)
// stored as its partial sums; the last block to finish adds up all blocks' and
// writes the scalars
__device__ __forceinline__ void na_finish(const NaArgs &a, const double sum[3]) {
  __shared__ double sh[3][NA_WARPS];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
    for (int q = 0; q < 3; q++) sh[q][warp] = sum[q];
  __syncthreads();
  double *part = (double *)(a.scr + OFF_PART);
  if (threadIdx.x == 0) {
    for (int q = 0; q < 3; q++) {
      double t = 0.0;
      for (int ww = 0; ww < NA_WARPS; ww++) t += sh[q][ww];
      part[4 * blockIdx.x + q] = t;
    }
    __threadfence();
    s_last = atomicAdd((unsigned int *)(a.scr + OFF_CTR), 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double t[3] = {0.0, 0.0, 0.0};
  for (unsigned int b = threadIdx.x; b < gridDim.x; b += NA_BLOCK)
    for (int q = 0; q < 3; q++) t[q] += __ldcg(&part[4 * b + q]);
  for (int q = 0; q < 3; q++) {
    for (int o = 16; o > 0; o >>= 1) t[q] += __shfl_down_sync(0xffffffffu, t[q], o);
    if (lane == 0) sh[q][warp] = t[q];
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int q = 0; q < 3; q++) {
    t[q] = 0.0;
    for (int ww = 0; ww < NA_WARPS; ww++) t[q] += sh[q][ww];
  }
  a.out[0] = 0.5 * t[0];
  a.out[1] = (0.5 * t[1]) / 3.0;
  a.out[2] = t[2];
  *(unsigned int *)(a.scr + OFF_CTR) = 0u;
}

// the active force of particle i (MDcode/cell_list+forces.c:207-218) added to
// its pair force; returns its active virial
__device__ __forceinline__ double na_active(const NaArgs &a, int i, acg::PairAcc &acc) {
  const int t = a.act[i];
  if (t < 0 || t >= a.nact) return 0.0;
  const double kx = (double)a.k[t], ky = (double)a.k[a.nact + t], kz = (double)a.k[2 * a.nact + t];
  const double *u = a.xu ? a.xu : a.x;
  acc.fx += a.f0 * kx;
  acc.fy += a.f0 * ky;
  acc.fz += a.f0 * kz;
  return a.f0 * (kx * u[3 * i] + ky * u[3 * i + 1] + kz * u[3 * i + 2]);
}

// Forces by cells: one block stages a cell's 27 neighbour cells (8 at two cells
// per side) -- FP32 reduced coordinates with index and type for the distance
// test, FP64 ones for the pair terms -- and its warps take the cell's particles
// one at a time: the lanes test 32 candidates a step in FP32 against the pair's
// own cut widened by 1e-4 (the coordinates' rounding is below 2e-5 of it at the
// largest box), the accepted ones queue up, and every 32 of them are evaluated by
// a full warp in FP64 (masked by the exact cut).  About one candidate in twelve is
// within the cut, so the FP64 terms, which bounded a version that evaluated
// each candidate under a branch, run on full warps.  What bounds it now: issue
// (about 50 instructions per 32 candidates tested).  N = 20000: 260 -> 101 us a
// call with the cell build.
//
// A neighbourhood of more than NA_CAP candidates is taken in pieces of that many,
// each particle's force carried from one piece to the next in F (evaluated straight
// from memory such a cell made a call of N = 2000 take 597 us against 155 for the
// version of four threads a particle; in pieces 54).  A cell of a grid of few
// cells is shared by `split` blocks that stage the same neighbourhood: N = 700 78
// -> 30 us, N = 5000 76 -> 56.
// Coordinates outside [0, 1] get the minimum image in the test (the cells' images
// say nothing about them).
__global__ void __launch_bounds__(NA_BLOCK, 4) k_na_force(NaArgs a, int split) {
  extern __shared__ __align__(16) unsigned char na_sm[];
  float4 *cf = reinterpret_cast<float4 *>(na_sm);
  double *cx = reinterpret_cast<double *>(na_sm + NA_CAP * sizeof(float4)), *cy = cx + NA_CAP, *cz = cy + NA_CAP;
  __shared__ int s_pre[28], s_start[27];
  __shared__ uint16_t queue[NA_WARPS][96];
  __shared__ signed char s_img[3][27];  // image of each neighbour cell (3 and more cells per side)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nc = a.nc, ncell = nc * nc * nc;
  const int lo = acg::stencil_lo(nc), wd = acg::stencil_hi(nc) - lo + 1, ns = wd * wd * wd;
  const int own = nc >= 3 ? 13 : 0;  // the cell itself among its neighbours
  const double L = a.L;
  const int *order = na_i(a, OFF_ORDER);
  float cut[3];  // the test's cuts by type sum, reduced units
  for (int k = 0; k < 3; k++) cut[k] = (float)(acg::KA_RC2 * (1.0 + 1e-4) / (acg::ka_is2(k) * L * L));
  auto outside = [](double x, double y, double z) {
    return !(x >= 0.0 && x <= 1.0 && y >= 0.0 && y <= 1.0 && z >= 0.0 && z <= 1.0);
  };
  double sum[3] = {0.0, 0.0, 0.0};  // pe, virial, active virial of this warp's particles (lane 0)
  for (int b = blockIdx.x; b < ncell * split; b += gridDim.x) {
    const int c = b / split, part = b - c * split;
    if (warp == 0) {
      int m = 0;
      if (lane < ns) {
        const int cc[3] = {c % nc + lane % wd + lo, (c / nc) % nc + (lane / wd) % wd + lo,
                           c / (nc * nc) + lane / (wd * wd) + lo};
        int c2 = 0, mul = 1;
        for (int k = 0; k < 3; k++, mul *= nc) {
          c2 += acg::wrap_cell(cc[k], nc) * mul;
          s_img[k][lane] = (signed char)(nc < 3 ? 0 : (cc[k] < 0 ? -1 : (cc[k] >= nc ? 1 : 0)));
        }
        s_start[lane] = na_i(a, OFF_START)[c2];
        m = na_i(a, OFF_COUNT)[c2];
      }
      int x = m;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane < ns) s_pre[lane + 1] = x;
      if (lane == 0) s_pre[0] = 0;
    }
    __syncthreads();
    const int mc = s_pre[own + 1] - s_pre[own], Q = part * NA_WARPS < mc ? s_pre[ns] : 0;
    for (int p0 = 0; p0 < Q; p0 += NA_CAP) {
      const int np = min(Q - p0, NA_CAP);
      bool out = false;
      for (int q = threadIdx.x; q < np; q += NA_BLOCK) {
        const int u = acg::union_of(s_pre, ns, p0 + q);
        const int j = order[s_start[u] + (p0 + q - s_pre[u])];
        const double x = a.x[3 * j], y = a.x[3 * j + 1], z = a.x[3 * j + 2];
        out |= outside(x, y, z);
        cf[q] = make_float4((float)(x + s_img[0][u]), (float)(y + s_img[1][u]), (float)(z + s_img[2][u]),
                            __int_as_float(j | (a.type[j] << 30)));
        cx[q] = x;
        cy[q] = y;
        cz[q] = z;
      }
      const bool far = __syncthreads_or(out);
      if (far) {
        for (int q = threadIdx.x; q < np; q += NA_BLOCK)
          cf[q] = make_float4((float)acg::min_image(cx[q]), (float)acg::min_image(cy[q]),
                              (float)acg::min_image(cz[q]), cf[q].w);
        __syncthreads();
      }
      for (int w = part * NA_WARPS + warp; w < mc; w += NA_WARPS * split) {
        const int i = order[s_start[own] + w];
        const int ti = a.type[i];
        const acg::PairParamsD P(ti, L);
        acg::PairAcc acc = {0.0, 0.0, 0.0, 0.0, 0.0};
        const int qi = s_pre[own] + w - p0;  // the particle itself among the piece's
        const bool here = qi >= 0 && qi < np;
        const double xi = here ? cx[qi] : a.x[3 * i], yi = here ? cy[qi] : a.x[3 * i + 1],
                     zi = here ? cz[qi] : a.x[3 * i + 2];
        const bool fold = far || outside(xi, yi, zi);
        // (at two cells per side every cell neighbours every other under two images)
        const bool image = fold || nc < 3;
        const float fx = (float)(fold ? acg::min_image(xi) : xi), fy = (float)(fold ? acg::min_image(yi) : yi),
                    fz = (float)(fold ? acg::min_image(zi) : zi);
        const float c0 = ti == 0 ? cut[0] : cut[1], c1 = ti == 0 ? cut[1] : cut[2];
        uint16_t *qu = queue[warp];
        int cnt = 0;
        auto pairs = [&](int k) {  // the last k <= 32 of the queue
          __syncwarp();
          cnt -= k;
          const int q = qu[cnt + (lane < k ? lane : 0)];
          acg::pair_f64(acc, acg::min_image(xi - cx[q]), acg::min_image(yi - cy[q]), acg::min_image(zi - cz[q]), P,
                        (__float_as_int(cf[q].w) >> 30) & 1, lane < k);
          __syncwarp();
        };
        auto test = [&](int q) {
          if (q >= np) return false;
          const float4 fj = cf[q];
          float dx = fx - fj.x, dy = fy - fj.y, dz = fz - fj.z;
          if (image) {
            dx -= rintf(dx);
            dy -= rintf(dy);
            dz -= rintf(dz);
          }
          return fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < (((__float_as_int(fj.w) >> 30) & 1) ? c1 : c0) && q != qi;
        };
        const unsigned below = (1u << lane) - 1u;
        for (int q0 = lane; q0 - lane < np; q0 += 64) {
          const bool ok0 = test(q0), ok1 = test(q0 + 32);
          const unsigned b0 = __ballot_sync(0xffffffffu, ok0), b1 = __ballot_sync(0xffffffffu, ok1);
          if (ok0) qu[cnt + __popc(b0 & below)] = (uint16_t)q0;
          cnt += __popc(b0);
          if (ok1) qu[cnt + __popc(b1 & below)] = (uint16_t)(q0 + 32);
          cnt += __popc(b1);
          while (cnt >= 32) pairs(32);
        }
        if (cnt > 0) pairs(cnt);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          acc.fx += __shfl_xor_sync(0xffffffffu, acc.fx, o);
          acc.fy += __shfl_xor_sync(0xffffffffu, acc.fy, o);
          acc.fz += __shfl_xor_sync(0xffffffffu, acc.fz, o);
          acc.pe += __shfl_xor_sync(0xffffffffu, acc.pe, o);
          acc.vir += __shfl_xor_sync(0xffffffffu, acc.vir, o);
        }
        if (lane == 0) {
          acg::pair_scale(acc, L);
          if (p0 == 0) {
            sum[2] += na_active(a, i, acc);
          } else {
            acc.fx += a.F[3 * i];
            acc.fy += a.F[3 * i + 1];
            acc.fz += a.F[3 * i + 2];
          }
          a.F[3 * i] = acc.fx;
          a.F[3 * i + 1] = acc.fy;
          a.F[3 * i + 2] = acc.fz;
          sum[0] += acc.pe;
          sum[1] += acc.vir;
        }
      }
      __syncthreads();
    }
    __syncthreads();
  }
  na_finish(a, sum);
}

// Forces by particles, for large grids of few particles a cell: four threads take a particle's neighbour cells one after another,
// straight from memory.  Staging a neighbourhood of a few dozen candidates costs
// k_na_force a block and its barriers for a particle or two.
constexpr int NA_TPP = 4;
__global__ void __launch_bounds__(NA_BLOCK) k_na_force_sparse(NaArgs a) {
  const int i = (blockIdx.x * NA_BLOCK + threadIdx.x) / NA_TPP, lane = threadIdx.x % NA_TPP;
  const double L = a.L;
  acg::PairAcc acc = {0.0, 0.0, 0.0, 0.0, 0.0};
  double va = 0.0;
  if (i < a.n) {
    const double xi = a.x[3 * i], yi = a.x[3 * i + 1], zi = a.x[3 * i + 2];
    const acg::PairParamsD P(a.type[i], L);
    const int nc = a.nc, c = na_i(a, OFF_CELL)[i];
    const int cx = c % nc, cy = (c / nc) % nc, cz = c / (nc * nc);
    const int lo = acg::stencil_lo(nc), hi = acg::stencil_hi(nc);
    for (int oz = lo; oz <= hi; oz++)
      for (int oy = lo; oy <= hi; oy++)
        for (int ox = lo; ox <= hi; ox++) {
          const int c2 = acg::wrap_cell(cx + ox, nc) + acg::wrap_cell(cy + oy, nc) * nc +
                         acg::wrap_cell(cz + oz, nc) * nc * nc;
          const int s0 = na_i(a, OFF_START)[c2], m = na_i(a, OFF_COUNT)[c2];
          for (int q = lane; q < m; q += NA_TPP) {
            const int j = na_i(a, OFF_ORDER)[s0 + q];
            if (j == i) continue;
            const double dx = acg::min_image(xi - a.x[3 * j]), dy = acg::min_image(yi - a.x[3 * j + 1]),
                         dz = acg::min_image(zi - a.x[3 * j + 2]);
            const bool tj = a.type[j] != 0;
            if (fma(dx, dx, fma(dy, dy, dz * dz)) * P.is2[tj] < acg::KA_RC2)
              acg::pair_f64(acc, dx, dy, dz, P, tj, true);
          }
        }
  }
#pragma unroll
  for (int o = NA_TPP / 2; o > 0; o >>= 1) {
    acc.fx += __shfl_xor_sync(0xffffffffu, acc.fx, o);
    acc.fy += __shfl_xor_sync(0xffffffffu, acc.fy, o);
    acc.fz += __shfl_xor_sync(0xffffffffu, acc.fz, o);
    acc.pe += __shfl_xor_sync(0xffffffffu, acc.pe, o);
    acc.vir += __shfl_xor_sync(0xffffffffu, acc.vir, o);
  }
  const bool mine = i < a.n && lane == 0;
  if (mine) {
    acg::pair_scale(acc, L);
    va = na_active(a, i, acc);
    a.F[3 * i] = acc.fx;
    a.F[3 * i + 1] = acc.fy;
    a.F[3 * i + 2] = acc.fz;
  }
  double sum[3] = {mine ? acc.pe : 0.0, mine ? acc.vir : 0.0, va};
  for (int q = 0; q < 3; q++)
    for (int o = 16; o > 0; o >>= 1) sum[q] += __shfl_down_sync(0xffffffffu, sum[q], o);
  na_finish(a, sum);
}

}  // namespace

extern "C" int acg_forces_noalloc(const double *x, const double *xu, const int *type, const int *act_tag,
                                  const int *k, int n, int nact, double L, double f0, double *F,
                                  double *scalars, void *stream) {
  if (!x || !type || !act_tag || !F || !scalars || (nact > 0 && !k))
    return na_fail(ACG_ERR_INVALID, "acg_forces_noalloc: null device pointer");
  if (n < 2 || n > ACG_NOALLOC_MAX_N)
    return na_fail(ACG_ERR_INVALID, "acg_forces_noalloc: n must be in [2, " +
                                        std::to_string(ACG_NOALLOC_MAX_N) + "], got " + std::to_string(n));
  if (nact < 0 || nact > n) return na_fail(ACG_ERR_INVALID, "acg_forces_noalloc: nact must be in [0, n]");
  if (!(L > 0) || L > 1e6) return na_fail(ACG_ERR_INVALID, "acg_forces_noalloc: bad box length");
  // cell geometry of MDcode/Parallel.c:72-78 (cells no smaller than 2.85)
  const int nc = (int)((double)(int)L / 2.85);
  if (nc < 2) return na_fail(ACG_ERR_INVALID, "acg_forces_noalloc: box smaller than 2 cells of 2.85 per side");
  if ((long long)nc * nc * nc > ACG_NOALLOC_MAX_CELLS)
    return na_fail(ACG_ERR_INVALID, "acg_forces_noalloc: " + std::to_string((long long)nc * nc * nc) +
                                        " cells exceed ACG_NOALLOC_MAX_CELLS (" +
                                        std::to_string(ACG_NOALLOC_MAX_CELLS) + ")");
  int dev = 0;
  cudaError_t ce = cudaGetDevice(&dev);
  if (ce != cudaSuccess || dev < 0 || dev >= 256)
    return na_fail(ACG_ERR_CUDA, std::string("acg_forces_noalloc: cudaGetDevice: ") + cudaGetErrorString(ce));
  void *scr = nullptr;
  {
    // once per device, with that device current: the host-side name of the
    // array is not a device address; ask the runtime for the address
    std::lock_guard<std::mutex> lk(na_mu);
    if (!na_ptr[dev]) {
      void *p = nullptr;
      ce = cudaGetSymbolAddress(&p, acg_noalloc_scratch);
      if (ce != cudaSuccess || !p)
        return na_fail(ACG_ERR_CUDA,
                       std::string("acg_forces_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(ce));
      // the force kernel's staging is above the default limit
      ce = cudaFuncSetAttribute(k_na_force, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)NA_SMEM);
      if (ce != cudaSuccess)
        return na_fail(ACG_ERR_CUDA,
                       std::string("acg_forces_noalloc: cudaFuncSetAttribute: ") + cudaGetErrorString(ce));
      na_ptr[dev] = p;
    }
    scr = na_ptr[dev];
  }
  NaArgs a;
  a.x = x;
  a.xu = xu;
  a.type = type;
  a.act = act_tag;
  a.k = k;
  a.F = F;
  a.out = scalars;
  a.scr = (unsigned char *)scr;
  a.n = n;
  a.nact = nact;
  a.nc = nc;
  a.L = L;
  a.inv_cell = L / (L / (double)nc);
  a.f0 = f0;
  cudaStream_t s = (cudaStream_t)stream;
  const int ncell = nc * nc * nc;
  k_na_clear<<<(ncell + 255) / 256, 256, 0, s>>>(a);
  k_na_count<<<(n + 255) / 256, 256, 0, s>>>(a);
  k_na_scan<<<1, 1024, 0, s>>>(a);
  k_na_scatter<<<(n + 255) / 256, 256, 0, s>>>(a);
  if (ncell >= NA_SPARSE_CELLS && n < NA_SPARSE * ncell) {
    k_na_force_sparse<<<(n * NA_TPP + NA_BLOCK - 1) / NA_BLOCK, NA_BLOCK, 0, s>>>(a);
  } else {
    // blocks sharing a cell: as many as fill the chip, with a particle for each
    // warp on average
    const int split = std::max(1, std::min(NA_FILL / ncell, (n + NA_WARPS * ncell - 1) / (NA_WARPS * ncell)));
    k_na_force<<<std::min(ncell * split, NA_MAX_BLOCKS), NA_BLOCK, NA_SMEM, s>>>(a, split);
  }
  ce = cudaGetLastError();
  if (ce != cudaSuccess)
    return na_fail(ACG_ERR_CUDA, std::string("acg_forces_noalloc: launch: ") + cudaGetErrorString(ce));
  return ACG_OK;
}
