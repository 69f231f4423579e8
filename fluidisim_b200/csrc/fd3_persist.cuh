// The inner CG loop in one cooperative launch, for volumes without the multigrid (Jacobi-PCG and the
// linear path's CG).
//
// Without the multigrid an iteration is four short passes, and as separate kernels each pays a launch
// boundary, a chain of dependent loads (gate, codes, operands) and the last block's merge of the
// partials: 26 us per iteration at 215k cells, 19 at 65k, where the passes' bytes take 1 us from L2.
// Here CTAs, one to an SM, keep their cells' p, r, diagonal and row on chip for the whole loop, and the
// iteration has two grid-wide meetings, each a reduction and a barrier at once (GridTeam::sum).
// Between them a cell exchanges with its neighbours only z and the last direction, through L2.
//
// Measured (B200, whole calls): a projection of 75 x 61 x 47 cells (260 iterations) 7.22 -> 1.97 ms, the linear
// step of 64 x 32 x 32 (244 iterations) 5.04 -> 1.57 ms: 6 us per iteration, of which the two meetings take 4.3.
#pragma once

#include "fd3_fast.cuh"

namespace fd3 {

constexpr int GRID_THREADS = 512;   // one CTA per SM: the meetings cost less with fewer CTAs and warps
constexpr int GRID_MAX_CTAS = 160;  // slots
constexpr int GRID_MAX_CELLS = 12;  // cells of a thread (k_cg_loop's largest instance)
constexpr size_t cg_smem(int cells) { return (size_t)cells * 7 * GRID_THREADS * sizeof(float); }
// Polls before a CTA gives up: a meeting that never completes ends the kernel with status 100 (reported with its reason)
// instead of hanging the GPU.  They are polls, not time, so that a grid suspended meanwhile does not give up; 2^20 take
// 0.23 s.
constexpr unsigned GRID_POLLS = 1u << 22;

// The CTAs of a cooperative grid as one team, meeting at a counter that is 0 at the launch and never
// reset.  A meeting is one release-add and an acquire-poll by one thread per CTA (1.3 us on 148 CTAs); a sum
// adds the CTAs' partials in its slots (2.1 us).  Polling the slots themselves, one number per CTA beside its
// partial, took 5.6 us (148 x 148 polls of the same lines), and mailboxes per reader 2.6 us.  The slots
// alternate between two sets: a CTA writes a set again only after a later meeting, which every CTA has
// reached only after reading it.
constexpr int GRID_PARTS = 444;  // parts of a sum, at most (sum_parts): three teams on each of 148 SMs
struct GridSlots {
  double2 part[2][GRID_MAX_CTAS];
  double parts[2][GRID_PARTS];
  unsigned arrived;
};
constexpr int GRID_STAND_IN = 4;  // CTAs that one stands in for, at most
struct GridShared {
  double warp[GRID_STAND_IN][32][2];
  double sum[2];
  double parts[GRID_PARTS / 32 + 1];
};
template <int THREADS>
struct GridTeam {
  GridSlots* slots;
  GridShared& sh;
  unsigned meeting = 0;
  __device__ __forceinline__ GridTeam(GridSlots* s, GridShared& shared) : slots(s), sh(shared) {}

  // What the team wrote to global memory before is visible to all of
  // it after.  False, for the whole CTA, when another did not arrive within GRID_POLLS.
  __device__ __forceinline__ bool arrive_and_wait() {  // thread 0; the CTA's writes ordered before by a barrier
    ++meeting;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&slots->arrived) : "memory");
    const unsigned target = meeting * gridDim.x;
    unsigned seen, polls = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&slots->arrived) : "memory");
    } while ((int)(seen - target) < 0 && ++polls < GRID_POLLS);
    return (int)(seen - target) >= 0;
  }
  // A meeting without a sum.
  __device__ __forceinline__ bool meet() {
    __syncthreads();
    bool late = false;
    if (threadIdx.x == 0) late = !arrive_and_wait();
    else ++meeting;
    return !__syncthreads_or(late);
  }
  // Sums a (and b, when TWO) over every thread of the grid: the same totals, added in the same order, for
  // every thread, in a[0] and b[0].  A meeting.  The sum is that of `slots_used` CTAs with one value per thread; a thread
  // that stands in for V of them (CTAs blockIdx.x + v gridDim.x) has the values of all: a[v] and b[v].
  template <bool TWO, int V>
  __device__ __forceinline__ bool sum(double (&a)[V], double (&b)[V], int slots_used) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int v = 0; v < V; ++v) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        a[v] += __shfl_xor_sync(0xffffffffu, a[v], o);
        if (TWO) b[v] += __shfl_xor_sync(0xffffffffu, b[v], o);
      }
      if (lane == 0) {
        sh.warp[v][wid][0] = a[v];
        if (TWO) sh.warp[v][wid][1] = b[v];
      }
    }
    __syncthreads();
    double2* half = slots->part[meeting & 1u];
    bool late = false;
    auto store = [&](int v, int slot) {
      double2 p = make_double2(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < THREADS / 32; ++q) {
        p.x += sh.warp[v][q][0];
        if (TWO) p.y += sh.warp[v][q][1];
      }
      __stcg(half + slot, p);
    };
    if constexpr (V > 1) {
      const int slot = (int)(blockIdx.x + threadIdx.x * gridDim.x);
      if ((int)threadIdx.x < V && slot < slots_used) store(threadIdx.x, slot);
      if (wid == 0) __syncwarp();  // the other threads' slots before the first arrives
    }
    if (threadIdx.x == 0) {
      if constexpr (V == 1) store(0, blockIdx.x);
      late = !arrive_and_wait();
    } else {
      ++meeting;
    }
    if (__syncthreads_or(late)) return false;
    if (wid == 0) {
      constexpr int PER = (GRID_MAX_CTAS + 31) / 32;
      double2 v[PER];
#pragma unroll
      for (int e = 0; e < PER; ++e) {
        const int q = lane + 32 * e;
        v[e] = q < (V == 1 ? (int)gridDim.x : slots_used) ? __ldcg(half + q) : make_double2(0.0, 0.0);
      }
      double x = 0.0, y = 0.0;
#pragma unroll
      for (int e = 0; e < PER; ++e) {
        x += v[e].x;
        if (TWO) y += v[e].y;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        x += __shfl_xor_sync(0xffffffffu, x, o);
        if (TWO) y += __shfl_xor_sync(0xffffffffu, y, o);
      }
      if (lane == 0) {
        sh.sum[0] = x;
        sh.sum[1] = y;
      }
    }
    __syncthreads();
    a[0] = sh.sum[0];
    b[0] = sh.sum[1];
    return true;
  }
  // Where the parts of the next sum_parts go: parts 0 .. n - 1, each written by one thread of the grid.
  __device__ __forceinline__ double* next_parts() { return slots->parts[meeting & 1u]; }
  // The sum of n <= min(THREADS, GRID_PARTS) parts, in an order that depends on n alone: the same total for every
  // thread of any grid.  A meeting.
  __device__ __forceinline__ double sum_parts(int n, bool& met) {
    const double* parts = next_parts();
    met = meet();
    if (!met) return 0.0;
    const int warps = (n + 31) >> 5;
    if ((int)threadIdx.x < 32 * warps) {
      double v = (int)threadIdx.x < n ? __ldcg(parts + threadIdx.x) : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if ((threadIdx.x & 31) == 0) sh.parts[threadIdx.x >> 5] = v;
    }
    __syncthreads();
    double a = sh.parts[0];
    for (int q = 1; q < warps; ++q) a += sh.parts[q];
    return a;
  }
};

// The meeting counter to 0, before a launch that meets; below 0 by `absent` CTAs that will not come (for tests: every
// meeting then runs out).
__global__ void k_grid_reset(GridSlots* slots, unsigned absent) {
  KSTART();
  slots->arrived = 0u - absent;
}

// A cell's row kept on chip, as Geo::rec keeps it: per face the aperture onto a fluid neighbour, or the ghost's
// 1/theta (the lid: twice the aperture).  A ghost face with an aperture other than 1 (RC_CUT_GHOST) reads that
// aperture again.
__device__ __forceinline__ void kept_row(const Geo& g, unsigned code, int i, int j, int k, float (&w)[6]) {
  const bool unit = code & RC_UNIT;
  const int axis[6] = {0, 0, 1, 1, 2, 2};
  const int fi[6] = {fu(g, i, j, k), fu(g, i + 1, j, k), fv(g, i, j, k), fv(g, i, j + 1, k), fw(g, i, j, k),
                     fw(g, i, j, k + 1)};
  const int xs[4] = {i - 1, i + 1, i, i}, ys[4] = {j, j, j - 1, j + 1};
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const unsigned st = face_state(code, f);
    w[f] = 0.f;
    if (!st) continue;
    if (st == 1 || g.linear) {
      const float a = unit ? 1.f : aper3(g, axis[f], fi[f]);
      w[f] = st == 1 ? a : 2.f * a;
    } else {
      w[f] = f == 5 ? ghost_it_up(g, i, j, k) : ghost_it_side(g, i, j, k, xs[f < 4 ? f : 0], ys[f < 4 ? f : 0]);
    }
  }
}
__device__ __noinline__ float face_aperture(const Geo& g, int c, int f) {
  int i, j, k;
  cell_ijk(g, c, i, j, k);
  if (f < 2) return aper3(g, 0, fu(g, i + f, j, k));
  if (f < 4) return aper3(g, 1, fv(g, i, j + f - 2, k));
  return aper3(g, 2, fw(g, i, j, k + f - 4));
}
// W(f): the kept coefficient of face f; v: the operand at the six neighbours (any value where the face has
// no fluid neighbour).
template <class W>
__device__ __forceinline__ float apply_kept(const Geo& g, unsigned code, int c, float pc, W w, const float (&v)[6]) {
  float acc = 0.f;
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const unsigned st = face_state(code, f);
    float ghost = pc * w(f);
    if ((code & RC_CUT_GHOST) && st == 2u) ghost = face_aperture(g, c, f) * pc * w(f);
    acc += st == 1u ? w(f) * (pc - v[f]) : (st == 2u ? ghost : 0.f);
  }
  return acc * g.inv;
}

// The Jacobi-PCG loop (delta3d_mobile.rs:515-545 with z = prec r): its prime, then iterations until
// S->active drops, with the scalar steps of apply_op (f64 reductions).  Thread t of the T threads of the
// grid owns the cells t, t + T, ...: CELLS of them, each with r, prec, its code and direction in registers
// and p and its row's coefficients in shared memory (14 KB per cell of a thread).
// Per iteration: d = z + beta d at the cell and, recomputed from z and the previous d, at its neighbours;
// q = A d; d.q | p += alpha d, r -= alpha q, z = prec r; r.r and r.z together.  z and the two
// alternating direction buffers live in global memory, read past L1 (other SMs write them).
//
// The sums are those of a grid of `ctas` CTAs, whatever the grid: with fewer, a CTA stands in for V of them and its threads
// own the cells of as many (a batch runs its volumes on a part of the SMs each, and a volume has the same bits there).
template <int CELLS, int V>
__global__ void __launch_bounds__(GRID_THREADS, 1)
    k_cg_loop(const __grid_constant__ Geo g, const unsigned short* __restrict__ codes, const float* __restrict__ prec, float* p,
              float* r, float* d0, float* d1, float* z, Scalars* S, GridSlots* slots, int ctas) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // no early start of the next kernel: its CTAs find no room
  if (!S->active) return;
  extern __shared__ float kept[];  // [CELLS][7][GRID_THREADS]: six coefficients and p
  __shared__ GridShared sh;
  GridTeam<GRID_THREADS> team(slots, sh);
  auto K = [&](int s, int f) -> float& { return kept[(s * 7 + f) * GRID_THREADS + threadIdx.x]; };
  constexpr int PAIR = CELLS < 2 ? 1 : 2;
  const int nxny = g.nx * g.ny;
  // cell s of this thread (n or more: none): cell s % EACH of the thread's place in CTA s / EACH of those it stands in for
  constexpr int EACH = CELLS / V;
  const int T = (V == 1 ? (int)gridDim.x : ctas) * GRID_THREADS, t0 = blockIdx.x * GRID_THREADS + threadIdx.x;
  auto cell = [&](int s) {
    if (V == 1) return t0 + s * T;
    const int v = s / EACH * (int)gridDim.x;
    return (int)blockIdx.x + v < ctas ? t0 + v * GRID_THREADS + s % EACH * T : g.n;
  };
  float rc[CELLS], mc[CELLS], dc[CELLS], qc[CELLS];
  unsigned code[CELLS];
  double acc[V] = {}, acc2[V] = {};
  auto clear = [&] {
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = acc2[v] = 0.0;
  };
#pragma unroll
  for (int s = 0; s < CELLS; ++s) {
    const int c = cell(s);
    rc[s] = mc[s] = dc[s] = qc[s] = 0.f;
    code[s] = 0u;
    if (c < g.n) {
      K(s, 6) = p[c];
      rc[s] = r[c];
      mc[s] = prec[c];
      const unsigned rc16 = codes[c];
      if (rc16 & RC_WET) {
        int i, j, k;
        cell_ijk(g, c, i, j, k);
        float w[6];
        code[s] = rc16;
        kept_row(g, rc16, i, j, k, w);
#pragma unroll
        for (int f = 0; f < 6; ++f) K(s, f) = w[f];
      }
      z[c] = mc[s] * rc[s];
      acc[s / EACH] += (double)rc[s] * (double)mc[s] * (double)rc[s];
    }
  }
  double rz, rr = S->rr;
  const double tolb2 = S->tolb2, phys = S->phys;
  unsigned it = S->it;
  const unsigned max_iters = S->max_iters;
  int status = 0, brk = 0;
  float beta = 0.f;
  float* din = d0;
  float* dout = d1;
  if (!team.template sum<false, V>(acc, acc2, ctas)) status = 100;
  rz = acc[0];
  if (!status && !isfinite(rz)) status = 2;
  while (!status) {
    clear();
    // PAIR cells' twelve loads each go out together; the stores of the direction come after them all
#pragma unroll
    for (int s0 = 0; s0 < CELLS; s0 += PAIR) {
      float v[PAIR][6];
#pragma unroll
      for (int e = 0; e < PAIR; ++e) {
        const int s = s0 + e, c = cell(s);
        if (s >= CELLS) continue;
        const int nb[6] = {c - 1, c + 1, c - g.nx, c + g.nx, c - nxny, c + nxny};
        float zn[6], dn[6];
#pragma unroll
        for (int f = 0; f < 6; ++f) {
          const bool on = face_state(code[s], f) == 1u;
          zn[f] = on ? __ldcg(z + nb[f]) : 0.f;
          dn[f] = on && beta != 0.f ? __ldcg(din + nb[f]) : 0.f;
        }
#pragma unroll
        for (int f = 0; f < 6; ++f) v[e][f] = beta == 0.f ? zn[f] : zn[f] + beta * dn[f];
      }
#pragma unroll
      for (int e = 0; e < PAIR; ++e) {
        const int s = s0 + e, c = cell(s);
        if (s >= CELLS) continue;
        const float zc = mc[s] * rc[s];
        const float d = beta == 0.f ? zc : zc + beta * dc[s];
        qc[s] = (code[s] & RC_WET) ? apply_kept(g, code[s], c, d, [&](int f) { return K(s, f); }, v[e]) : 0.f;
        dc[s] = d;
        acc[s / EACH] += (double)d * (double)qc[s];
      }
    }
#pragma unroll
    for (int s = 0; s < CELLS; ++s) {
      const int c = cell(s);
      if (c < g.n) dout[c] = dc[s];
    }
    if (!team.template sum<false, V>(acc, acc2, ctas)) { status = 100; break; }
    if (!(acc[0] > 0.0)) { brk = 1; break; }  // FIN_DQ
    const float alpha = (float)(rz / acc[0]);
    clear();
#pragma unroll
    for (int s = 0; s < CELLS; ++s) {
      const int c = cell(s);
      if (c < g.n) {
        K(s, 6) += alpha * dc[s];
        const float rn = rc[s] - alpha * qc[s];
        rc[s] = rn;
        z[c] = mc[s] * rn;
        acc[s / EACH] += (double)rn * (double)rn;
        acc2[s / EACH] += (double)rn * (double)mc[s] * (double)rn;
      }
    }
    if (!team.template sum<true, V>(acc, acc2, ctas)) { status = 100; break; }
    if (!isfinite(acc[0])) { status = 2; break; }  // FIN_RN
    ++it;
    rr = acc[0];
    if (!((rr > tolb2 || rr > phys) && it < max_iters)) break;
    if (!isfinite(acc2[0])) { status = 2; break; }  // FIN_RZ_ITER
    beta = (float)(acc2[0] / rz);
    rz = acc2[0];
    float* t = din;
    din = dout;
    dout = t;
  }
#pragma unroll
  for (int s = 0; s < CELLS; ++s) {
    const int c = cell(s);
    if (c < g.n) { p[c] = K(s, 6); r[c] = rc[s]; }
  }
  // every CTA has met for the last time here, but one that gave up says so whichever it is
  if (threadIdx.x == 0 && (blockIdx.x == 0 || status == 100)) {
    S->rr = rr;
    S->rz = rz;
    S->it = it;
    S->brk = brk;
    if (status) S->status = status;
    S->active = 0;
  }
}

}  // namespace fd3
