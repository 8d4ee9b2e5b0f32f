// Grid-wide reductions and halo exchange of cooperative launches, by tagged
// words: a value and the number of the exchange it belongs to are stored
// together as one 16-byte word, so the reader that finds the number it waits
// for has the value too.  A reduction is then one store and one poll of every
// block's word, without a counter, a fence and a second read (as a counter
// barrier it took about 3 us of an iteration on 148 blocks).  Every block is
// resident, so a wait ends; it is bounded all the same, and a wait that runs
// out ends the kernel with an error flag the host reads.
#pragma once
#include "common.cuh"

namespace phastb {

// A wait gives up after kGridLimitNs of the GPU's global timer (a normal wait is
// a few microseconds); kGridPolls polls bound it a second time.
constexpr unsigned long long kGridLimitNs = 2000000000ull;
constexpr unsigned kGridPolls = 1u << 28;

__device__ __forceinline__ unsigned long long grid_clock_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A value with its tag; both move in one 128-bit access (16-byte aligned).
struct __align__(16) Tagged {
  double v;
  unsigned long long tag;
};

__device__ __forceinline__ void st_tagged(Tagged* p, double v, unsigned long long tag) {
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ Tagged ld_tagged(const Tagged* p) {
  long long lo, hi;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  return Tagged{__longlong_as_double(lo), (unsigned long long)hi};
}

// Waits (bounded) until p carries `tag`; its value through *v.  False: gave up, or another wait of the grid has.
__device__ __forceinline__ bool wait_tagged(const Tagged* p, unsigned long long tag, double* v, unsigned* err,
                                            unsigned long long limit_ns = kGridLimitNs) {
  Tagged t = ld_tagged(p);
  if (t.tag != tag) {
    const unsigned long long t0 = grid_clock_ns();
    for (unsigned i = 1;; ++i) {
      t = ld_tagged(p);
      if (t.tag == tag) break;
      if ((i & 255u) == 0u && (*reinterpret_cast<volatile unsigned*>(err) != 0u || i >= kGridPolls ||
                               grid_clock_ns() - t0 > limit_ns)) {
        atomicExch(err, 1u);
        return false;
      }
    }
  }
  *v = t.v;
  return true;
}

// Three single-precision values and the step they belong to in one 16-byte word.
__device__ __forceinline__ void st_node(Tagged* p, float x, float y, float z, unsigned tag) {
  st_tagged(p, __hiloint2double(__float_as_int(y), __float_as_int(x)),
            ((unsigned long long)tag << 32) | (unsigned)__float_as_int(z));
}
// Waits (bounded) for the word of step `tag`; false: gave up, or another wait of the grid has.
__device__ __forceinline__ bool wait_node(const Tagged* p, unsigned tag, float (&v)[3], unsigned* err,
                                          unsigned long long limit_ns = kGridLimitNs) {
  Tagged t = ld_tagged(p);
  if ((unsigned)(t.tag >> 32) != tag) {
    const unsigned long long t0 = grid_clock_ns();
    for (unsigned i = 1;; ++i) {
      t = ld_tagged(p);
      if ((unsigned)(t.tag >> 32) == tag) break;
      if ((i & 255u) == 0u && (*reinterpret_cast<volatile unsigned*>(err) != 0u || i >= kGridPolls ||
                               grid_clock_ns() - t0 > limit_ns)) {
        atomicExch(err, 1u);
        return false;
      }
    }
  }
  v[0] = __int_as_float(__double2loint(t.v));
  v[1] = __int_as_float(__double2hiint(t.v));
  v[2] = __int_as_float((int)(unsigned)t.tag);
  return true;
}

// Barrier of the `threads` threads that share id (1..15) inside a block.
__device__ __forceinline__ void sub_barrier(int id, int threads) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

constexpr int kGridValues = 3;     // values of one reduction
constexpr int kGridBlocks = 148;   // at most one block per SM
constexpr int kGridDirect = 32;    // up to so many blocks read one another's words directly
inline size_t grid_slot_bytes() { return sizeof(Tagged) * 4 * kGridValues * kGridBlocks; }

// One launch's exchange: two slots of kGridValues words per block for the operands and two for the results, and
// the error flag, all zero at launch.
struct GridSync {
  Tagged* slots;
  unsigned* err;
  unsigned long long phase;  // reductions done, the same in every thread of the grid
  unsigned long long limit_ns = kGridLimitNs;  // of one wait
};

// Sums of v[0..K) and minima of v[K..K+M) over every thread of the grid, in every thread, in an order fixed by
// the grid and block size.  Blocks of kT threads.  False: a wait ran out somewhere (leave the kernel).  While the
// first K + M warps wait, the others run overlap(thread, threads): what does not need the result.
//
// Up to kGridDirect blocks every block reads all words.  More readers than that queue on the few lines the words
// lie in (measured per reduction, 148 blocks: 3.8 us; 32: 1.3; 16: 1.0), so there block 0 alone reads them and
// stores the result to one word per block: 1.6 us at 148 blocks (a counter barrier and a second read: 1.9).
// The words alternate between two slots: a word is written again two reductions later, which its reader has
// entered after reading it.
template <int K, int M, int kT, class Overlap>
__device__ __forceinline__ bool grid_reduce(double (&v)[K + M], GridSync& g, Overlap overlap) {
  constexpr int N = K + M, kW = kT / 32, kFold = (kGridBlocks + 31) / 32;
  static_assert(N <= kGridValues && N < kW && kW <= 32, "a warp per value and one to spare, a lane per warp's share");
  __shared__ double s_warp[N][kW];
  __shared__ double s_fold[N][kFold];
  __shared__ double s_out[N];
  __shared__ int s_bad;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, G = gridDim.x;
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = k < K ? warp_sum(v[k]) : warp_min(v[k]);
  if (l == 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) s_warp[k][w] = v[k];
  }
  if (threadIdx.x == 0) s_bad = 0;
  __syncthreads();
  const unsigned long long tag = g.phase + 1;
  Tagged* in = g.slots + (size_t)(g.phase & 1ull) * kGridValues * G;
  Tagged* res = g.slots + (size_t)(2 + (g.phase & 1ull)) * kGridValues * G;
  auto fold = [](bool sum, double t) { return sum ? warp_sum(t) : warp_min(t); };
  const bool direct = G <= kGridDirect, root = blockIdx.x == 0;
  // warp k: the block's value k
  if (w < N) {
    const bool sum = w < K;
    double t = fold(sum, l < kW ? s_warp[w][l] : (sum ? 0.0 : INFINITY));
    if (G == 1) {
      if (l == 0) s_out[w] = t;
    } else {
      if (l == 0) st_tagged(in + (size_t)w * G + blockIdx.x, t, tag);
      if (direct) {
        t = sum ? 0.0 : INFINITY;
        if (l < G && !wait_tagged(in + (size_t)w * G + l, tag, &t, g.err, g.limit_ns)) s_bad = 1;
        t = fold(sum, t);
        if (l == 0) s_out[w] = t;
      } else if (!root) {
        if (l == 0 && !wait_tagged(res + (size_t)w * G + blockIdx.x, tag, &s_out[w], g.err, g.limit_ns)) s_bad = 1;
      }
    }
  }
  if (G > 1 && !direct && root) {
    // kFold parts per value, one word per thread
    for (int j = w; j < N * kFold; j += kW) {
      const int k = j / kFold, part = j - k * kFold;
      const bool sum = k < K;
      const int b = 32 * part + l;
      double t = sum ? 0.0 : INFINITY;
      if (b < G && !wait_tagged(in + (size_t)k * G + b, tag, &t, g.err, g.limit_ns)) s_bad = 1;
      t = fold(sum, t);
      if (l == 0) s_fold[k][part] = t;
    }
    __syncthreads();
    if (threadIdx.x < G) {
      const int parts = (G + 31) / 32;
#pragma unroll
      for (int q = 0; q < N; ++q) {
        double t = s_fold[q][0];
        for (int i = 1; i < parts; ++i) t = q < K ? t + s_fold[q][i] : fmin(t, s_fold[q][i]);
        st_tagged(res + (size_t)q * G + threadIdx.x, t, tag);
        if (threadIdx.x == 0) s_out[q] = t;
      }
    }
  }
  if (w >= N) overlap((int)threadIdx.x - 32 * N, kT - 32 * N);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = s_out[k];
  const bool ok = s_bad == 0;
  ++g.phase;
  return ok;
}
template <int K, int M, int kT>
__device__ __forceinline__ bool grid_reduce(double (&v)[K + M], GridSync& g) {
  return grid_reduce<K, M, kT>(v, g, [](int, int) {});
}

}  // namespace phastb
