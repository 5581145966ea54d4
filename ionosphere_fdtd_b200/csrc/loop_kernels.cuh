// Many leapfrog steps in one cooperative launch, for meshes whose phases are a
// few microseconds of work (sm_100a).
//
// Every thread takes runs (an edge or a face, then a vertex or an edge, and one
// radial quad) of the flat run list, one per round of the whole grid, with the
// per-run arithmetic and the direct gathers of kh_kernel / ke_kernel, so the
// results are the same bits.  A grid barrier follows each phase.  Bound by
// latency: a phase is the barrier (one atomic add per CTA, then polling), one
// trip to L2 for a run's table entries and one for its rows.  What this saves
// against a launch per phase is the launch, the record, the layer rows and, for
// the ring kernels, the descriptors and the staging: 5.0 us per step at s2 / 24
// cells against 9.2 us of ring launches in a graph, 13.2 against 14.1 at s5 / 37.
// The next run's table entries are read before the current run's rows are used
// (and before the barrier for a phase's first run), and a block has only as many
// threads as its runs need: 5.6 without either at s2 / 24, 14.6 at s5 / 37.
//
// Receivers are sampled by a warp of their own in every CTA while the others
// work: Er / Et rows in the next H phase and Hr / Ht rows in the same step's E
// phase, the phases that only read them.
//
// Every wait is bounded by the global timer.  A CTA whose wait runs out sets
// bit 0 of the status word, counts itself out of the remaining barriers and
// returns, so the others' waits end and the barrier is whole for the next
// launch.
#pragma once

#include "pipe_kernels.cuh"
#include "step_kernels.cuh"

namespace ifdtd {

struct LoopArgs {
  int steps, done, total, every;  // this launch's steps, those before it in the run, the run's; steps per sample
  const double* currents;         // (steps) source current, or null
  unsigned long long* arrivals;   // CTA arrivals so far: a multiple of the grid size between launches
  SampleSlot slot[kMaxSlots];
};

// Most threads of a CTA (one warp of them only samples).
template <typename real, bool PLASMA>
constexpr int kLoopThreads = sizeof(real) == 8 || PLASMA ? 512 : 768;

// This CTA's rows of the slots with E kinds (e) or H kinds, if the state after
// the launch's step `step` is to be sampled; one warp.
template <typename real>
__device__ __forceinline__ void loop_sample(const Rec<real>& R, const LoopArgs& A, int step, bool e) {
  const int n = A.done + step + 1;
  if (n % A.every != 0 && n != A.total) return;
#pragma unroll
  for (int q = 0; q < kMaxSlots; ++q)
    if ((A.slot[q].kind < 2) == e)
      for (int r = blockIdx.x; r < A.slot[q].rows; r += gridDim.x)
        sample_row(R, A.slot[q], r, (size_t)((n - 1) / A.every));
}

// Wait (bounded) until `arrivals` reaches target.
__device__ __forceinline__ bool wait_arrivals(const unsigned long long* arrivals, unsigned long long target,
                                              int* status) {
  auto seen = [&] {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(arrivals) : "memory");
    return v;
  };
  if (seen() >= target) return true;
  const uint64_t t0 = pipe::global_ns();
  for (uint32_t i = 1; i < (1u << 30); ++i) {
    if (seen() >= target) return true;
    if ((i & 15u) == 0 && pipe::global_ns() - t0 > pipe::kWaitNs) break;
  }
  atomicOr(status, 1);
  return false;
}

// Table entries of one H run (edge: tail, head; face: edges, vertices) and of
// one E run (vertex: its slots' edges and faces; edge: left, right face).
struct HRunTables {
  int4 a, b;
};
template <int MAXDEG>
struct ERunTables {
  int v, edge[MAXDEG], face[MAXDEG];
};

template <typename real, bool PLASMA, int MAXDEG>
__global__ void __launch_bounds__(kLoopThreads<real, PLASMA>, 1)
    kd_loop(const Rec<real>* __restrict__ recs, const LoopArgs A) {
  constexpr int N = Lanes<real>::N;
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  __shared__ Rec<real> R;
  __shared__ int go_on;
  load_rec(R, recs);
  Layers<real> Ls;
  load_layers(R, reinterpret_cast<real*>(dyn_smem), Ls, threadIdx.x, blockDim.x);
  __syncthreads();
  const int T = blockDim.x - 32;
  const int Pn = R.Pn, Pm = R.Pm, SW = R.slot_width, cn = Pn / N, cm = Pm / N;
  const uint32_t mag_cn = div_magic(cn), mag_cm = div_magic(cm);
  const real* Jsum = PLASMA ? jsum(R) : nullptr;
  // whether Er / Et rows are sampled (after the E phase, by the next H phase) and Hr / Ht rows
  bool late = false, early = false;
#pragma unroll
  for (int q = 0; q < kMaxSlots; ++q)
    if (A.slot[q].rows > 0) (A.slot[q].kind < 2 ? late : early) = true;
  const bool sampler = threadIdx.x >= T;
  const int first = blockIdx.x * T + threadIdx.x, stride = gridDim.x * T;
  const int h_edges = R.nE * cn, h_runs = h_edges + R.nF * cm, e_verts = R.nV * cn, e_runs = e_verts + R.nE * cm;
  // after every phase but the last, and after that one when its E values are still to be sampled
  const int barriers = 2 * A.steps - (late ? 0 : 1);
  int arrived = 0;              // barriers this CTA has arrived at
  unsigned long long base = 0;  // arrivals when the launch began: this CTA's own is still missing, so
  if (threadIdx.x == 0) {       // no barrier of this launch can be complete yet
    const unsigned long long seen = *reinterpret_cast<volatile unsigned long long*>(A.arrivals);
    base = seen - seen % gridDim.x;
  }
  auto barrier = [&] {
    __syncthreads();
    ++arrived;
    if (threadIdx.x == 0) {
      asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(A.arrivals), "l"(1ull) : "memory");
      go_on = wait_arrivals(A.arrivals, base + (unsigned long long)arrived * gridDim.x, R.status);
    }
    __syncthreads();
    return go_on != 0;
  };
  auto h_tables = [&](int it) {
    HRunTables t{};
    if (it < h_edges) {
      const int2 th = __ldg(R.edge_th + fast_div(it, mag_cn));
      t.a.x = th.x;
      t.a.y = th.y;
    } else if (it < h_runs) {
      const int f = fast_div(it - h_edges, mag_cm);
      t.a = __ldg(R.face_e + f);
      if (PLASMA) t.b = __ldg(R.face_v + f);
    }
    return t;
  };
  auto e_tables = [&](int it) {
    ERunTables<MAXDEG> t{};
    if (it < e_verts) {
      const int slot = fast_div(it, mag_cn);
      t.v = __ldg(R.vlist + slot);
#pragma unroll
      for (int q = 0; q < MAXDEG; ++q) {
        t.edge[q] = __ldg(R.ps_edge + (size_t)slot * SW + q);
        if (PLASMA) t.face[q] = __ldg(R.ps_face + (size_t)slot * SW + q);
      }
    } else if (it < e_runs) {
      const int2 lr = __ldg(R.edge_lr + fast_div(it - e_verts, mag_cm));
      t.edge[0] = lr.x;
      t.edge[1] = lr.y;
    }
    return t;
  };
  HRunTables ht = h_tables(first);
  bool ok = true;
  for (int step = 0; step < A.steps; ++step) {
    if (sampler) {
      if (late && step > 0) loop_sample(R, A, step - 1, true);
    } else {
      for (int it = first; it < h_runs; it += stride) {
        const HRunTables t = ht;
        ht = h_tables(it + stride);
        if (it < h_edges) {
          const int e = fast_div(it, mag_cn), k0 = (it - e * cn) * N;
          h_edge_run(R, Ls, h_edge_layer(R, Ls, k0), e, k0, R.er + (size_t)t.a.y * Pn, R.er + (size_t)t.a.x * Pn,
                     R.et + (size_t)e * Pm, R.ht + (size_t)e * Pn, R.ht + (size_t)e * Pn, __ldg(R.inv_theta + e),
                     R.si_mem + (size_t)e * R.si_terms, R.si_mem + (size_t)e * R.si_terms, R.si_scale + e);
        } else {
          const int i = it - h_edges, f = fast_div(i, mag_cm), j0 = (i - f * cm) * N;
          h_face_run<real, PLASMA>(R, Ls, ld16(Ls.hC + j0), f, j0, R.et + (size_t)t.a.x * Pm, R.et + (size_t)t.a.y * Pm,
                                   R.et + (size_t)t.a.z * Pm, R.hr + (size_t)f * Pm, R.hr + (size_t)f * Pm,
                                   R.er + (size_t)t.b.x * Pn, R.er + (size_t)t.b.y * Pn, R.er + (size_t)t.b.z * Pn,
                                   nullptr, 0, R.n_species > 1 ? R.Jtot + (size_t)f * 3 * Pm : nullptr,
                                   R.face_w + 4 * (size_t)f, PLASMA ? R.face_pl + 12 * (size_t)f : nullptr);
        }
      }
    }
    ERunTables<MAXDEG> et = e_tables(first);
    if (!(ok = barrier())) break;
    if (sampler) {
      if (early) loop_sample(R, A, step, false);
    } else {
      const real current = A.currents && (R.n_src_er + R.n_src_et) > 0 ? (real)__ldg(A.currents + step) : real(0);
      for (int it = first; it < e_runs; it += stride) {
        const ERunTables<MAXDEG> t = et;
        et = e_tables(it + stride);
        if (it < e_verts) {
          const int slot = fast_div(it, mag_cn), k0 = (it - slot * cn) * N;
          const real* hrows[MAXDEG];
          const real* jrows[MAXDEG];
#pragma unroll
          for (int q = 0; q < MAXDEG; ++q) {
            hrows[q] = R.ht + (size_t)t.edge[q] * Pn;
            jrows[q] = PLASMA ? Jsum + (size_t)t.face[q] * 3 * Pm : nullptr;
          }
          e_vertex_run<real, PLASMA, MAXDEG>(R, vertex_layer(R, Ls, t.v, k0), R.n_src_er > 0, t.v, k0, hrows, jrows,
                                             R.ps_coef + (size_t)slot * SW,
                                             PLASMA ? R.ps_wc + (size_t)slot * SW * 4 : nullptr, R.er + (size_t)t.v * Pn,
                                             R.er + (size_t)t.v * Pn, current);
        } else {
          const int i = it - e_verts, e = fast_div(i, mag_cm), j0 = (i - e * cm) * N;
          const int l = t.edge[0], r = t.edge[1];
          e_edge_run<real, PLASMA>(R, edge_layer(R, Ls, e, j0), R.n_src_et > 0, e, j0, R.hr + (size_t)l * Pm,
                                   R.hr + (size_t)r * Pm, R.ht + (size_t)e * Pn,
                                   PLASMA ? Jsum + (size_t)l * 3 * Pm : nullptr, PLASMA ? Jsum + (size_t)r * 3 * Pm : nullptr,
                                   R.et + (size_t)e * Pm, R.et + (size_t)e * Pm, current, __ldg(R.inv_phi + e),
                                   PLASMA ? R.tan + 8 * (size_t)e : nullptr);
        }
      }
    }
    ht = h_tables(first);
    if ((step + 1 < A.steps || late) && !(ok = barrier())) break;
  }
  if (ok && late && sampler) loop_sample(R, A, A.steps - 1, true);
  if (threadIdx.x == 0 && arrived < barriers) atomicAdd(A.arrivals, (unsigned long long)(barriers - arrived));
}

}  // namespace ifdtd
