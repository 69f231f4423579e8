// The multigrid PCG loop in one cooperative launch, for volumes whose passes are latency.
//
// In the loop graph an iteration is seventeen kernels or so, and 4 us of each is its launch boundary, the gate, and the
// chain of loads before its first sum, when the passes' work is a third of that.  Here a grid of CTAs, one to an SM,
// stays for the whole loop, the passes are separated by grid meetings (GridTeam: 1.3 us on 148 CTAs, 2.1 with a sum), and
// the scalars are on chip.  The fine passes are the paired march's (fd3_zmarch2.cuh) with three teams of 256 threads per
// CTA, each taking chunks of a tile in turn; the levels run one cell per thread, their warps spread over the CTAs; the
// levels of at most TAIL_REG_THREADS cells run in the first CTA, its rows kept in shared memory for the whole loop.
//
// Every cell value is that of the separate kernels; the f64 sums have a part per chunk, added in the order of the chunks,
// so the result is the same on any number of CTAs, and a volume beside others takes fewer (fd3_volume::mg_ctas).  Whole
// projections alone, separate kernels and one launch (B200): 64^3 1.04 and 0.94 ms, 48^3 1.00 and 0.89, 32^3 0.77 and 0.70,
// 32 x 16 x 24 0.61 and 0.58.
#pragma once

#include "fd3_persist.cuh"
#include "fd3_zmarch2.cuh"

namespace fd3 {

constexpr int MG_TEAMS = 3;
constexpr int MG_THREADS = MG_TEAMS * Z2T;  // one CTA per SM, 80 registers
constexpr int MG_LEVELS = 8;                // levels above the tail
constexpr int MG_LEAST_SHARE = 8;           // CTAs beside many other volumes (sixteen 64^3 at once, ms: 3.7 on 8, 5.9 on 4)

struct MgLoop {
  Geo g;
  const unsigned short* codes;
  const float* prec;
  float *p, *r, *dir[2], *q;
  void *z, *z2;
  Lev lev[MG_LEVELS];
  int nlev;    // levels above the tail
  Lev tail[TAIL_REG_LEVELS];
  int ntail;
  Air air;     // of level 0 (sh = 1)
  Scalars* S;
  GridSlots* slots;
};

struct MgShared {
  ZPlanes2 sbuf[MG_TEAMS][2];
  ZResid2 tr[MG_TEAMS][2];
  TailShared tail;
  GridShared grid;
  // The loop's scalars, the same for every thread (thread 0 writes them).  In registers they would be spilled in the passes,
  // and a spilled register is read from L2 after each meeting: 150 bytes of spills less, 1% of a 64^3 projection.
  double rr, rz, rn, tolb2, phys;
  unsigned max_iters;
  float vk, vinv;
};

struct TeamSync {
  int id;
  __device__ __forceinline__ void operator()() const {
    asm volatile("barrier.sync %0, %1;" ::"r"(id), "r"(Z2T) : "memory");
  }
};

// Layers of a chunk: the even number that makes the longest team's march shortest, a chunk of K layers counting K + 2
// (its halo layers) and GRID_PARTS teams taking the chunks that hold water in turn; at most GRID_PARTS chunks up to the
// highest water (top).  It does not depend on the grid, nor do the sums, whose parts are the chunks.
__device__ __forceinline__ int mg_pick_chunk(const Geo& g, int* cost, int& top) {
  const int ntx = (g.nx + Z2X - 1) / Z2X, nty = (g.ny + Z2Y - 1) / Z2Y;
  if (threadIdx.x < 9) cost[threadIdx.x] = 0;
  __syncthreads();
  for (int q = threadIdx.x; q < 8 * ntx * nty; q += MG_THREADS) {
    const int k = 2 + 2 * (q & 7), t = q >> 3;
    const int high = ztile2_at(g, t % ntx, t / ntx, 0, g.nz, 0, 0).k1;
    if (high > 0) atomicAdd(cost + (q & 7), (high + k - 1) / k);
    if (high > 0 && (q & 7) == 0) atomicMax(cost + 8, high);
  }
  __syncthreads();
  int best = 2, least = 0x7fffffff;
  for (int q = 0; q < 8; ++q) {
    const int k = 2 + 2 * q, c = (cost[q] + GRID_PARTS - 1) / GRID_PARTS * (k + 2);
    if (c < least) { least = c; best = k; }
  }
  top = cost[8];
  const int high = GRID_PARTS / (ntx * nty);  // chunks of a tile, at least one (mg_fits)
  return max(best, 2 * (((top + high - 1) / high + 1) / 2));
}

inline bool mg_fits(int nx, int ny) { return ((nx + Z2X - 1) / Z2X) * ((ny + Z2Y - 1) / Z2Y) <= GRID_PARTS; }

template <class T>
__global__ void __launch_bounds__(MG_THREADS, 1) k_mg_loop(const __grid_constant__ MgLoop a) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // no early start of the next kernel: its CTAs find no room
  Scalars* S = a.S;
  if (!S->active) return;
  extern __shared__ float4 mg_smem4[];
  MgShared& sh = *reinterpret_cast<MgShared*>(mg_smem4);
  const Geo& g = a.g;
  GridTeam<MG_THREADS> grid(a.slots, sh.grid);
  const int tid = threadIdx.x, team = tid / Z2T, tx = tid & 31, ty = (tid >> 5) & 7, teams = gridDim.x * MG_TEAMS;
  const int ntx = (g.nx + Z2X - 1) / Z2X, nty = (g.ny + Z2Y - 1) / Z2Y, tiles = ntx * nty;
  int top;
  const int K = mg_pick_chunk(g, reinterpret_cast<int*>(sh.grid.warp), top);
  __syncthreads();
  const int chunks = tiles * max((top + K - 1) / K, 1);
  const bool first_cta = blockIdx.x == 0;
  if (first_cta && a.ntail > 0) tail_rows(a.tail, a.ntail, sh.tail);
  T* z = static_cast<T*>(a.z);
  T* z2 = static_cast<T*>(a.z2);
  const TeamSync sync{6 + team};
  // f(march) over the chunks of this thread's team: the chunks in order of height, dealt to the CTAs first
  auto march_at = [&](int q) {
    const int tile = q % tiles;
    return March2<TeamSync>{g,  a.codes,       ztile2_at(g, tile % ntx, tile / ntx, q / tiles * K, K, tx, ty), tx,
                            ty, sh.sbuf[team], sh.tr[team], sync};
  };
  auto each_chunk = [&](auto f) {
    for (int q = team * gridDim.x + blockIdx.x; q < chunks; q += teams) {
      f(march_at(q));
      sync();  // the planes are free for the next chunk
    }
  };
  // the same with the sum of what f(march) returns over every thread and chunk, a part per chunk; a meeting
  auto sum_chunks = [&](bool& met, auto f) -> double {
    int half = 0;
    for (int q = team * gridDim.x + blockIdx.x; q < chunks; q += teams, half ^= 1) {
      double acc = f(march_at(q));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (tx == 0) sh.grid.warp[0][tid >> 5][half] = acc;
      sync();
      if (tx == 0 && ty == 0) {  // the other half is written meanwhile, this one after the next chunk's sync
        double part = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) part += sh.grid.warp[0][(tid >> 5) + w][half];
        __stcg(grid.next_parts() + q, part);
      }
    }
    return grid.sum_parts(chunks, met);
  };
  // f(i) for i = 0 .. n - 1 (a multiple of 32 rounded up), whole warps, spread over the SMs warp by warp
  auto each_warp = [&](int n, auto f) {
    for (int w = (tid >> 5) * gridDim.x + blockIdx.x; 32 * w < n; w += gridDim.x * (MG_THREADS / 32)) f(32 * w + (tid & 31));
  };
  auto air = [&](int l) { return Air{l < 3 ? a.air.ztop : nullptr, l + 1, a.air.ntx}; };

  // z = M^-1 r with r.z in rz (v_cycle3); false when a meeting failed
  auto vcycle = [&](double& rz) -> bool {
    const float rs = Store<T>::half ? sh.vinv : 1.f;
    const bool levels = a.nlev + a.ntail > 0;
    each_chunk([&](const auto& m) { march_pre(m, a.prec, a.r, z, rs); });
    if (!grid.meet()) return false;
    const Lev& L0 = a.nlev > 0 ? a.lev[0] : a.tail[0];
    if (levels) {
      each_chunk([&](const auto& m) { march_restrict(m, a.r, (const T*)z, L0, rs); });
      if (!grid.meet()) return false;
      const int last = a.nlev - 1;
#pragma unroll 1
      for (int l = 0; l < a.nlev; ++l) {
        const Lev& L = a.lev[l];
        if (l == last && a.ntail == 0) {  // a large coarsest level: its eight sweeps
#pragma unroll 1
          for (int s = 0; s < 8; ++s) {
            each_warp(L.n, [&](int c) {
              if (c < L.n) level_sweep_at<T>(L, (s & 1) ? L.x2 : L.x, (s & 1) ? L.x : L.x2, s == 0, c);
            });
            if (!grid.meet()) return false;
          }
        } else {
          const Lev& C = l < last ? a.lev[l + 1] : a.tail[0];
          each_warp(L.n, [&](int c) {
            if (c < L.n) level_pre_at<T>(L, air(l), c);
          });
          if (!grid.meet()) return false;
          each_warp(8 * C.n, [&](int q8) { level_restrict8_at<T>(L, C, air(l + 1), q8); });
          if (!grid.meet()) return false;
        }
      }
      if (a.ntail > 0) {
        if (first_cta) {
          const Lev& L = a.tail[0];
          if (tid < L.n) sh.tail.R[tid] = Store<T>::ld(as<T>(L.r), tid);
          __syncthreads();
          tail_cycle(a.tail, a.ntail, sh.tail);
          if (tid < L.n) Store<T>::st(as<T>(L.x), tid, sh.tail.XF[tid]);
        }
        if (!grid.meet()) return false;
      }
      // up: level l's second post-sweep is part of level l - 1's first (level_post21_at)
      const int top = a.ntail > 0 ? last : last - 1;
#pragma unroll 1
      for (int l = top; l >= 0; --l) {
        const Lev& L = a.lev[l];
        const Lev& C = l < last ? a.lev[l + 1] : a.tail[0];
        if (l < top) each_warp(8 * C.n, [&](int q8) { level_post21_at<T>(L, C, air(l + 1), q8); });
        else each_warp(L.n, [&](int c) {
          if (c < L.n) level_post1_at<T>(L, C, air(l), c);
        });
        if (!grid.meet()) return false;
      }
      if (top >= 0) {
        const Lev& L = a.lev[0];
        each_warp(L.n, [&](int c) {
          if (c < L.n) level_post2_at<T>(L, air(0), c);
        });
        if (!grid.meet()) return false;
      }
    }
    each_chunk([&](const auto& m) { march_post1(m, a.prec, a.r, (const T*)z, L0, levels ? 1 : 0, z2, rs); });
    if (!grid.meet()) return false;
    bool met;
    rz = sum_chunks(met, [&](const auto& m) {
      double acc = 0.0;
      march_post2(m, a.prec, a.r, (const T*)z2, z, rs, acc);
      return acc;
    });
    return met;
  };

  if (tid == 0) {
    sh.rr = S->rr;
    sh.rz = 0.0;
    sh.tolb2 = S->tolb2;
    sh.phys = S->phys;
    sh.max_iters = S->max_iters;
    sh.vk = S->vk;
    sh.vinv = S->vinv;
  }
  __syncthreads();
  unsigned it = S->it;
  int status = 0, brk = 0, mode = 0;
  float beta = 0.f;
  // the prime (mode 0), then iterations: each ends with a V-cycle
#pragma unroll 1
  for (;;) {
    double zn = 0.0;
    if (!vcycle(zn)) { status = 100; break; }
    if (!isfinite(zn)) { status = 2; break; }
    if (mode) {  // FIN_RZ_ITER
      beta = (float)(zn / sh.rz);
      if (tid == 0) sh.rr = sh.rn;
      ++it;
    }
    __syncthreads();
    if (tid == 0) sh.rz = zn;
    const float* din = a.dir[it & 1];
    float* dout = a.dir[(it & 1) ^ 1];
    bool met;
    const double dq = sum_chunks(met, [&](const auto& m) {
      double acc = 0.0;
      march_dir(m, (const T*)z, din, dout, a.q, mode, beta, acc);
      return acc;
    });
    if (!met) { status = 100; break; }
    if (!(dq > 0.0)) { brk = 1; break; }  // FIN_DQ
    const float alpha = (float)(sh.rz / dq);
    const double rn = sum_chunks(met, [&](const auto& m) {
      double acc = 0.0;
      chunk_update(g, m.t, alpha, a.p, a.r, dout, a.q, acc);
      return acc;
    });
    if (!met) { status = 100; break; }
    if (!isfinite(rn)) { status = 2; break; }  // FIN_RN
    if (tid == 0 && sh.vk > 0.f && rn > 0.0) sh.vinv = (float)((double)sh.vk / sqrt(rn));
    if (Store<T>::half) __syncthreads();  // vinv, before the next V-cycle reads it
    if (!((rn > sh.tolb2 || rn > sh.phys) && it + 1 < sh.max_iters)) {
      if (tid == 0) sh.rr = rn;
      ++it;
      break;
    }
    if (tid == 0) sh.rn = rn;
    mode = 1;
  }
  if (tid == 0 && (first_cta || status == 100)) {
    S->rr = sh.rr;
    S->rz = sh.rz;
    S->it = it;
    S->brk = brk;
    S->vinv = sh.vinv;
    if (status) S->status = status;
    S->active = 0;
  }
}

}  // namespace fd3
