// Shared device machinery of the BTA dataflow kernels.
//
// Every kernel of this library is a persistent "task" kernel: one CTA per SM pulls
// task tickets from a global counter in a topological order of the tile DAG, waits
// (bounded) on per-tile ready flags, runs the task on TS x TS FP64 tiles and
// publishes its output tile with a release store of the flag.  Because a CTA only
// waits for tasks with smaller tickets, and a ticket is only handed to a CTA that
// is already running, the kernels make progress without co-residency guarantees.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "bta_internal.h"

namespace gbta {

constexpr int NT = 128;          // threads per CTA
constexpr int LDS = TS + 1;      // shared-memory row stride (odd: column reads hit distinct banks)
constexpr int TILE_SMEM = TS * LDS;
constexpr int PER_THREAD = TS * TS / NT;   // tile elements staged per thread (8)

// Control block (ints) shared by all kernels of a solver.
enum {
  CTRL_TICKET = 0,   // next task ticket
  CTRL_ABORT = 1,    // set when any task fails; every wait returns early
  CTRL_INFO = 2,     // sticky: 1-based global row of the first non-positive pivot
  CTRL_ERR = 3,      // sticky: ERR_* code
  CTRL_MMA = 4,      // words 4-5: tile-pair products issued by the launch (one 64-bit count)
  CTRL_N = 8
};
enum { ERR_NONE = 0, ERR_TIMEOUT = 1 };

struct Ctl {
  int* ctrl;
  int* flags;
  int epoch;
  unsigned long long wait_ns;
  long long* trace;   // optional: TRACE_WORDS int64 per task (see trace_task), or null
};

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Release-add at GPU scope without a return value (no round trip for the issuer).
__device__ __forceinline__ void red_add_release(int* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Atomic add with acquire-release semantics at GPU scope; returns the old value.
__device__ __forceinline__ int atom_add_acq_rel(int* p, int v) {
  int old;
  asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
// Words that carry their own readiness: a buffer is filled with WORD_EMPTY (one particular
// NaN, replaced by another when a value has its bits), its producer writes each word once
// and a consumer polls the words it needs.  A hop is then one store and one load, without
// the release, the flag and the reload of a published tile.
constexpr long long WORD_EMPTY = -1ll;
__device__ __forceinline__ void st_word(double* p, double v) {
  const int hi = __double2hiint(v);   // (all ones: a NaN)
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p),
               "d"(__hiloint2double(hi == -1 ? 0x7ff80000 : hi, __double2loint(v)))
               : "memory");
}
__device__ __forceinline__ long long ld_word(const double* p) {
  long long v;
  asm volatile("ld.relaxed.gpu.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int ld_relaxed(const int* p) {
  return *(volatile const int*)p;
}
__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned smid() {
  unsigned r;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(r));
  return r;
}
// Task trace record (thread 0): [ticket, (type << 16) | sm, t_start, t_end, m0..m3] in
// globaltimer nanoseconds, m0..m3 optional intermediate marks (0 when unused);
// written only when tracing is enabled.
constexpr int TRACE_WORDS = 8;
__device__ __forceinline__ void trace_task(const Ctl& c, int ticket, int type, unsigned long long t0) {
  if (c.trace && threadIdx.x == 0) {
    long long* r = c.trace + (long long)TRACE_WORDS * ticket;
    r[0] = ticket;
    r[1] = ((long long)blockIdx.x << 32) | ((long long)type << 16) | smid();
    r[2] = (long long)t0;
    r[3] = (long long)gtimer();
  }
}
__device__ __forceinline__ void trace_clear_marks(const Ctl& c, int ticket) {
  if (c.trace && threadIdx.x == 0)
    for (int k = 4; k < TRACE_WORDS; ++k) c.trace[(long long)TRACE_WORDS * ticket + k] = 0;
}
__device__ __forceinline__ void trace_mark(const Ctl& c, int ticket, int k) {
  if (c.trace && threadIdx.x == 0) c.trace[(long long)TRACE_WORDS * ticket + 4 + k] = (long long)gtimer();
}
__device__ __forceinline__ void trace_put(const Ctl& c, int ticket, int k, long long v) {
  if (c.trace && threadIdx.x == 0) c.trace[(long long)TRACE_WORDS * ticket + 4 + k] = v;
}

__device__ __forceinline__ void raise_abort(const Ctl& c) { atomicExch(c.ctrl + CTRL_ABORT, 1); }

// Thread-0 helper: spin (bounded in time) until flag >= epoch.  Returns false on
// abort or timeout (timeout also records ERR_TIMEOUT and aborts the launch).
// Only thread 0 of a CTA polls, and a persistent kernel runs one to three CTAs per SM, so
// the first SPIN_NS of a wait are a tight acquire-load loop (the hop latency of the
// dependency chains is what bounds these kernels; 20 to 150 ns of sleep between the polls
// measured equal to 0.7 % slower); longer waits back off with a short sleep.
constexpr unsigned long long SPIN_NS = 200000;

static __device__ bool spin_ready(const Ctl& c, const int* flag, int* seen = nullptr, int plus = 0) {
  const int want = c.epoch + plus;
  int v = ld_acquire(flag);
  if (v >= want) {
    if (seen) *seen = v;
    return true;
  }
  const unsigned long long t0 = gtimer();
  for (unsigned it = 1;; ++it) {
    v = ld_acquire(flag);
    if (v >= want) {
      if (seen) *seen = v;
      return true;
    }
    if ((it & 63) == 0) {
      if (ld_relaxed(c.ctrl + CTRL_ABORT)) return false;
      const unsigned long long dt = gtimer() - t0;
      if (dt > c.wait_ns) {
        atomicCAS(c.ctrl + CTRL_ERR, ERR_NONE, ERR_TIMEOUT);
        raise_abort(c);
        return false;
      }
      if (dt > SPIN_NS) __nanosleep(256);
    }
  }
}

// This thread: wait (bounded as spin_ready) for a word of a WORD_EMPTY-filled buffer.
// (the polling loop is out of line: its callers sit in unrolled code)
static __device__ __noinline__ long long poll_word(int* ctrl, unsigned long long wait_ns, const double* p) {
  const Ctl c{ctrl, nullptr, 0, wait_ns, nullptr};
  long long x = ld_word(p);
  if (x == WORD_EMPTY) {
    const unsigned long long t0 = gtimer();
    for (unsigned it = 1; (x = ld_word(p)) == WORD_EMPTY; ++it) {
      if ((it & 63) == 0) {
        if (ld_relaxed(c.ctrl + CTRL_ABORT)) return WORD_EMPTY;
        const unsigned long long dt = gtimer() - t0;
        if (dt > c.wait_ns) {
          atomicCAS(c.ctrl + CTRL_ERR, ERR_NONE, ERR_TIMEOUT);
          raise_abort(c);
          return WORD_EMPTY;
        }
        if (dt > SPIN_NS) __nanosleep(256);
      }
    }
  }
  return x;
}
static __device__ __forceinline__ bool wait_word(const Ctl& c, const double* p, double& v) {
  const long long x = poll_word(c.ctrl, c.wait_ns, p);
  v = __longlong_as_double(x);
  return x != WORD_EMPTY;
}

// CTA-wide wait on up to two flags (nullptr = no flag).  All threads return the
// same value.  Contains __syncthreads().
static __device__ bool cta_wait(const Ctl& c, const int* f0, const int* f1, int* s_ok) {
  if (threadIdx.x == 0) {
    bool ok = true;
    if (f0) ok = spin_ready(c, f0);
    if (ok && f1) ok = spin_ready(c, f1);
    *s_ok = ok ? 1 : 0;
  }
  __syncthreads();
  const bool ok = *s_ok != 0;
  __syncthreads();
  return ok;
}

// CTA-wide wait on one flag that also returns the flag word seen (epoch + payload) to
// every thread through *s_val.  Contains __syncthreads().
static __device__ bool cta_wait_val(const Ctl& c, const int* f, int* s_ok, int* s_val) {
  if (threadIdx.x == 0) *s_ok = spin_ready(c, f, s_val) ? 1 : 0;
  __syncthreads();
  const bool ok = *s_ok != 0;
  __syncthreads();
  return ok;
}

// Wait until *f >= epoch + plus: a flag that was published (epoch) and then raised by
// `plus` with cta_raise for a second product of the same task.
static __device__ bool cta_wait_plus(const Ctl& c, const int* f, int plus, int* s_ok) {
  if (threadIdx.x == 0) *s_ok = spin_ready(c, f, nullptr, plus) ? 1 : 0;
  __syncthreads();
  const bool ok = *s_ok != 0;
  __syncthreads();
  return ok;
}

// Publish a tile with a payload in its flag word (see EPOCH_SHIFT).  The barrier
// orders every thread's writes before thread 0's release store, which is cumulative,
// so no separate fence is needed.
__device__ __forceinline__ void cta_publish_val(const Ctl& c, int* flag, int payload) {
  __syncthreads();
  if (threadIdx.x == 0) st_release(flag, c.epoch + payload);
}

// Readiness scan for pipelined product loops.  Warp 0 advances *s_ready (the number of
// leading steps whose operand flags are all set) by checking up to SCAN_AHEAD further
// steps at once: lane 2k loads the first flag of step *s_ready + k and lane 2k+1 its
// second, each with an acquire load, so one memory round trip covers all of them and
// no GPU-scope fence is needed (a fence waits for the CTA's own outstanding writes,
// which costs thousands of cycles in a busy kernel).  `flags_of(s, f0, f1)` returns the
// step's flags (nullptr = none).  The caller synchronises the CTA before the call (the
// other warps decide from *s_ready whether to call it, so they must have read it before
// warp 0 rewrites it; a warp that read the new value would skip the call and its
// barriers) and afterwards, which extends the acquires to all its threads.
constexpr int SCAN_AHEAD = 16;
static_assert(2 * SCAN_AHEAD <= 32, "one lane per flag");

__device__ __forceinline__ int ld_relaxed_gpu(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// With `ring` (SCAN_RING ints), the first flag word of every step found ready is kept
// at ring[step % SCAN_RING] (read while step - *s_ready < SCAN_RING - SCAN_AHEAD).
constexpr int SCAN_RING = 2 * SCAN_AHEAD;
template <class FlagsOf>
__device__ __forceinline__ void scan_ready(const Ctl& c, int nsteps, FlagsOf flags_of, int* s_ready,
                                           int* ring = nullptr) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const int r0 = *s_ready;
    const int k = lane >> 1;
    int word = c.epoch;
    bool ready = true;
    if (k < SCAN_AHEAD) {
      if (r0 + k < nsteps) {
        const int* f0;
        const int* f1;
        flags_of(r0 + k, f0, f1);
        const int* f = (lane & 1) ? f1 : f0;
        if (f) {
          word = ld_acquire(f);
          ready = word >= c.epoch;
        }
      } else {
        ready = false;
      }
    }
    const unsigned ok = __ballot_sync(0xffffffffu, ready);
    int r = r0;
#pragma unroll
    for (int kk = 0; kk < SCAN_AHEAD; ++kk) {
      const int w0 = __shfl_sync(0xffffffffu, word, 2 * kk);
      if (r == r0 + kk && ((ok >> (2 * kk)) & 3u) == 3u) {
        if (ring && lane == 0) ring[r % SCAN_RING] = w0;
        ++r;
      }
    }
    if (lane == 0) *s_ready = r;
  }
}

// CTA-wide non-blocking poll of up to two flags.  Contains __syncthreads().
static __device__ bool cta_poll(const Ctl& c, const int* f0, const int* f1, int* s_ok) {
  if (threadIdx.x == 0) {
    bool ok = true;
    if (f0) ok = ld_acquire(f0) >= c.epoch;
    if (ok && f1) ok = ld_acquire(f1) >= c.epoch;
    *s_ok = ok ? 1 : 0;
  }
  __syncthreads();
  const bool ok = *s_ok != 0;
  __syncthreads();
  return ok;
}

// Publish a tile: every thread's stores are ordered before the flag release.
__device__ __forceinline__ void cta_publish(const Ctl& c, int* flag) {
  __syncthreads();   // every thread's writes before thread 0's (cumulative) release store
  if (threadIdx.x == 0) st_release(flag, c.epoch);
}

// Raise a published flag by v (< 512, so it stays below the next launch's epoch) once
// every thread's writes since the publication are done; the barrier and the cumulative
// release order them as in cta_publish.
__device__ __forceinline__ void cta_raise(int* flag, int v) {
  __syncthreads();
  if (threadIdx.x == 0) red_add_release(flag, v);
}

// Thread 0: add a task's tile-pair products (32 x 32 x 32 fp16 MMAs of two digit planes)
// to the launch's count.
__device__ __forceinline__ void count_pairs(const Ctl& c, unsigned long long n) {
  if (threadIdx.x == 0 && n) atomicAdd(reinterpret_cast<unsigned long long*>(c.ctrl + CTRL_MMA), n);
}

// Pull the next ticket (CTA-uniform).
// Between tasks every thread also orders its generic shared-memory writes (a task's
// FP64 scratch) before the bulk copies (async proxy) that a later task issues into the
// same bytes.
__device__ __forceinline__ int cta_ticket(const Ctl& c, int* s_t) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0) *s_t = ld_relaxed(c.ctrl + CTRL_ABORT) ? -1 : atomicAdd(c.ctrl + CTRL_TICKET, 1);
  __syncthreads();
  return *s_t;
}

// Whether this CTA leaves at once (see SpareRule; uniform).  The first nsm CTAs of a grid,
// and the second, are placed one per SM, so those that stay are spread evenly; the tickets go
// to whoever is there.  s: a shared word.
__device__ __forceinline__ bool cta_spare(const SpareRule& r, int* s) {
  if (!r.kf || (int)blockIdx.x < r.nsm) return false;
  if (threadIdx.x == 0) *s = 0;
  __syncthreads();
  int live = 0;
  for (int k = threadIdx.x; k < r.rows; k += NT) live += r.B - r.kf[k];
  atomicAdd(s, live);
  __syncthreads();
  const long long n = *s;
  __syncthreads();
  return (int)blockIdx.x >= (n <= r.lim1 ? 1 : n <= r.lim2 ? 2 : 8) * r.nsm;
}

// A tile view into a row-major matrix: rows x cols valid elements (<= TS each).
struct Tile {
  const double* p;
  int ld;
  int rows;
  int cols;
};

__device__ __forceinline__ Tile make_tile(const double* base, int ld, int row0, int col0, int nrows_total,
                                          int ncols_total) {
  Tile t;
  t.p = base + (size_t)row0 * ld + col0;
  t.ld = ld;
  t.rows = min(TS, nrows_total - row0);
  t.cols = min(TS, ncols_total - col0);
  return t;
}

// Register staging of one tile: element k of this thread is (r, c) with
// idx = threadIdx.x + k*NT, r = idx / TS, c = idx % TS (a warp reads one 256-B row).
// Loads bypass L1 (ld.global.cg): tiles are produced by other SMs inside the launch.
__device__ __forceinline__ void tile_ldg(double (&v)[PER_THREAD], const Tile& t) {
#pragma unroll
  for (int k = 0; k < PER_THREAD; ++k) {
    const int idx = threadIdx.x + k * NT;
    const int r = idx / TS, c = idx % TS;
    v[k] = (r < t.rows && c < t.cols) ? __ldcg(t.p + (size_t)r * t.ld + c) : 0.0;
  }
}
__device__ __forceinline__ void tile_sts(double* S, const double (&v)[PER_THREAD]) {
#pragma unroll
  for (int k = 0; k < PER_THREAD; ++k) {
    const int idx = threadIdx.x + k * NT;
    S[(idx / TS) * LDS + (idx % TS)] = v[k];
  }
}
// Transposed store: S[c][r] = element (r, c).
__device__ __forceinline__ void tile_sts_t(double* S, const double (&v)[PER_THREAD]) {
#pragma unroll
  for (int k = 0; k < PER_THREAD; ++k) {
    const int idx = threadIdx.x + k * NT;
    S[(idx % TS) * LDS + (idx / TS)] = v[k];
  }
}
__device__ __forceinline__ void tile_sts_op(double* S, const double (&v)[PER_THREAD], bool trans) {
  if (trans)
    tile_sts_t(S, v);
  else
    tile_sts(S, v);
}
// Direct global -> shared tile load (used outside the pipelined loops).
__device__ __forceinline__ void tile_load(double* S, const Tile& t) {
  double v[PER_THREAD];
  tile_ldg(v, t);
  tile_sts(S, v);
}
// Set the padded part of a diagonal tile's diagonal to one (rows/cols >= n).
__device__ __forceinline__ void tile_pad_identity(double* S, int n) {
  for (int j = n + threadIdx.x; j < TS; j += NT) S[j * LDS + j] = 1.0;
}
// Store the valid part of a shared tile.
__device__ __forceinline__ void tile_store(double* dst, int ld, int rows, int cols, const double* S) {
#pragma unroll
  for (int k = 0; k < PER_THREAD; ++k) {
    const int idx = threadIdx.x + k * NT;
    const int r = idx / TS, c = idx % TS;
    if (r < rows && c < cols) dst[(size_t)r * ld + c] = S[r * LDS + c];
  }
}
__device__ __forceinline__ void tile_store_zero(double* dst, int ld, int rows, int cols) {
#pragma unroll
  for (int k = 0; k < PER_THREAD; ++k) {
    const int idx = threadIdx.x + k * NT;
    const int r = idx / TS, c = idx % TS;
    if (r < rows && c < cols) dst[(size_t)r * ld + c] = 0.0;
  }
}

// ---------------------------------------------------------------------------
// Tile GEMM micro-kernel: acc (+|-)= op(A) * op(B) on TS x TS shared tiles.
// Thread (ty, tx) = (tid / 8, tid % 8) owns rows {2ty, 2ty+1} and columns
// {tx, tx+8, tx+16, tx+24}.
// ---------------------------------------------------------------------------
struct Acc {
  double v[2][4];
};

__device__ __forceinline__ void acc_zero(Acc& a) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) a.v[i][q] = 0.0;
}
__device__ __forceinline__ int acc_row(int i) { return (threadIdx.x / 8) * 2 + i; }
__device__ __forceinline__ int acc_col(int q) { return (threadIdx.x % 8) + 8 * q; }

__device__ __forceinline__ void acc_from_smem(Acc& a, const double* S) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) a.v[i][q] = S[acc_row(i) * LDS + acc_col(q)];
}
__device__ __forceinline__ void acc_to_smem(const Acc& a, double* S) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) S[acc_row(i) * LDS + acc_col(q)] = a.v[i][q];
}

// acc (+|-)= A * B with A(i,m) = As[i][m], B(m,j) = Bs[m][j] (transposes are applied
// when the tiles are staged into shared memory).
template <bool SUB>
__device__ __forceinline__ void tile_mma(Acc& acc, const double* As, const double* Bs) {
  const int i0 = (threadIdx.x / 8) * 2;
  const int j0 = threadIdx.x % 8;
#pragma unroll 8
  for (int m = 0; m < TS; ++m) {
    const double a0 = As[i0 * LDS + m];
    const double a1 = As[(i0 + 1) * LDS + m];
    double bq[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) bq[q] = Bs[m * LDS + j0 + 8 * q];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (SUB) {
        acc.v[0][q] = fma(-a0, bq[q], acc.v[0][q]);
        acc.v[1][q] = fma(-a1, bq[q], acc.v[1][q]);
      } else {
        acc.v[0][q] = fma(a0, bq[q], acc.v[0][q]);
        acc.v[1][q] = fma(a1, bq[q], acc.v[1][q]);
      }
    }
  }
}

// One step of a tile K-loop: operand tiles, whether each is staged transposed, and
// the ready flags to wait on (nullptr: no wait).
struct Step {
  Tile a, b;
  bool ta, tb;
  const int* fa;
  const int* fb;
};

// Pipelined K-loop: acc (+|-)= sum_s op(A_s) op(B_s).  The next step's tiles are
// fetched into registers while the current step computes, when their flags are
// already set (otherwise after the compute, with a bounded wait).  `bufs` holds
// four shared tiles.  Returns false (uniformly) on abort/timeout.
template <bool SUB, class StepFn>
static __device__ bool kloop(Acc& acc, int nsteps, StepFn step_of, const Ctl& c, double* bufs, int* s_ok) {
  if (nsteps <= 0) return true;
  double ra[PER_THREAD], rb[PER_THREAD];
  Step st = step_of(0);
  if (!cta_wait(c, st.fa, st.fb, s_ok)) return false;
  tile_ldg(ra, st.a);
  tile_ldg(rb, st.b);
  tile_sts_op(bufs, ra, st.ta);
  tile_sts_op(bufs + TILE_SMEM, rb, st.tb);
  __syncthreads();
  for (int s = 0; s < nsteps; ++s) {
    double* cur = bufs + (s & 1) * 2 * TILE_SMEM;
    double* nxt = bufs + ((s + 1) & 1) * 2 * TILE_SMEM;
    const bool more = s + 1 < nsteps;
    bool pre = false;
    if (more) {
      st = step_of(s + 1);
      pre = cta_poll(c, st.fa, st.fb, s_ok);
      if (pre) {
        tile_ldg(ra, st.a);
        tile_ldg(rb, st.b);
      }
    }
    tile_mma<SUB>(acc, cur, cur + TILE_SMEM);
    if (more) {
      if (!pre) {
        if (!cta_wait(c, st.fa, st.fb, s_ok)) return false;
        tile_ldg(ra, st.a);
        tile_ldg(rb, st.b);
      }
      tile_sts_op(nxt, ra, st.ta);
      tile_sts_op(nxt + TILE_SMEM, rb, st.tb);
    }
    __syncthreads();
  }
  return true;
}

// ---------------------------------------------------------------------------
// Small dense kernels on shared tiles (whole CTA).
// ---------------------------------------------------------------------------

// Scalar FP64 helpers.  On GB300 a warp-wide FP64 instruction occupies its SM
// sub-partition's FP64 unit for ~64-76 cycles, whether it is dependent, independent or
// even predicated off, so the sequential work of the tile routines below is counted in
// FP64 instructions.  Reciprocals and inverse square roots start from the hardware
// approximations rcp.approx / rsqrt.approx (~20 correct bits) and take ONE third-order
// correction (a truncated binomial series, i.e. a third-order Householder step), which
// leaves a truncation error of order e^3 ~ 2^-57:
//   1/d:       e = 1 - d y,    y <- y (1 + e + e^2)
//   1/sqrt(d): e = 1 - d y^2,  y <- y (1 + e/2 + 3 e^2 / 8)
__device__ __forceinline__ double rcp3(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-d, y, 1.0);
  const double p = 1.0 + e;
  const double ye = y * e;
  return fma(ye, p, y);
}
__device__ __forceinline__ double rsqrt3(double d) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double dy = d * y;
  const double e = fma(-dy, y, 1.0);
  const double p = fma(e, 0.375, 0.5);
  const double ye = y * e;
  return fma(ye, p, y);
}

// rd[j] = 1 / F[j][j] for the TS diagonal entries (one lane each).  Caller syncs.
__device__ __forceinline__ void tile_diag_recip(const double* F, double* rd) {
  if (threadIdx.x < TS) rd[threadIdx.x] = rcp3(F[threadIdx.x * LDS + threadIdx.x]);
}

// ---- register-resident tile factorization and triangular solves ------------------
// In the solve of a whole tile (smem_trsm_rlt), thread (lane r, warp g) holds row r of the
// tile at the eight columns c = g + 4q (q = 0..7) in registers, so every FP64 instruction
// has 32 useful lanes.  Columns are processed in order; the warp owning the current column
// finalises it and publishes it through shared memory with one CTA barrier per column,
// and every warp then updates its later columns with one FMA per element.  (The Cholesky,
// smem_potrf, and the other solves, which give a row's columns to lanes of one warp and
// need no barrier, split the work differently; see there.)  The loops over
// columns and register slots are fully unrolled: the conditions "column c = g + 4q
// is after column j" are written as a compile-time part plus a runtime part that
// only the one boundary slot needs, because an FP64 instruction issued under a false
// predicate still costs a full pipe slot.
__device__ __forceinline__ bool col_after(int q, int j, int g) {   // g + 4q > j
  return 4 * q > j || (4 * q + 3 > j && g > j - 4 * q);
}

// Named CTA barriers (ids 1 .. 15; id 0 is __syncthreads) for a producer warp that
// hands shared-memory data to the other warps: the producer arrives (release), the
// consumers sync (acquire); NT threads take part.
__device__ __forceinline__ void nbar_arrive(int id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(NT) : "memory");
}
__device__ __forceinline__ void nbar_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(NT) : "memory");
}

// Named barriers with a thread count other than NT (both sides must agree on N).
template <int N> __device__ __forceinline__ void nbar_arrive_n(int id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(N) : "memory");
}
template <int N> __device__ __forceinline__ void nbar_sync_n(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(N) : "memory");
}

// Barrier ids of smem_potrf: POTRF_BAR_L + (j & 7) hands pivot j from the pivot warp
// to the three update warps (NT threads); POTRF_BAR_C + (j & 3) hands column j+2,
// updated through pivot j, from its owner to the pivot warp (64 threads).
constexpr int POTRF_BAR_L = 1, POTRF_BAR_C = 9;

// x > 0 (false for zeros and NaN, true for +inf) by integer compares on the bits: a
// double compare is an FP64-unit instruction, and on the pivot chain it would occupy
// that unit for a full slot per pivot.
__device__ __forceinline__ bool positive_bits(double x) {
  const long long b = __double_as_longlong(x);
  return b > 0 && b <= 0x7ff0000000000000ll;
}

// 1/d on the integer pipe, for a chain that waits on every reciprocal: an FP64 instruction
// takes 64 cycles, so the hardware's seed with a third-order refinement in three dependent
// FMAs costs 227 cycles (measured), this 120 with the same error (at most 1.11e-16 relative over 2^20 values).  rcp_seed starts the hardware's
// fp32 reciprocal of the leading 24 significand bits; rcp_finish takes d's significand m
// (2^52 <= m < 2^53) and the seed Y0 (24 bits, Y0 2^-24 ~ 2^52 / m), forms delta = m Y0 -
// 2^76 modulo 2^64 (|delta| < 2^54) and Y = Y0 2^29 (1 - delta 2^-76 + (delta 2^-76)^2),
// the reciprocal's significand.  Where 1/d is subnormal (d from 2^1022 on) it is Y shifted by
// one or two places, truncated (50 bits at least).
// A zero, subnormal or infinite d gives NaN; so does a negative d or a NaN (a failed pivot
// anyway).
__device__ __forceinline__ float rcp_seed(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const float f = __uint_as_float(0x3f800000u | (__funnelshift_l(lo, hi, 3) & 0x7fffffu));
  float y;
  asm volatile("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
  return y;
}
__device__ __forceinline__ double rcp_finish(double d, float seed) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const unsigned mh = (hi & 0xfffffu) | 0x100000u;
  const unsigned Y0 = (min(__float_as_uint(seed), 0x3f7fffffu) & 0x7fffffu) | 0x800000u;
  const unsigned long long t0 = (unsigned long long)lo * Y0;
  const int dh = (int)((unsigned)(t0 >> 32) + mh * Y0);   // delta >> 32
  const long long c = (long long)dh * (int)Y0 + (long long)__umulhi((unsigned)t0, Y0);   // (Y0 delta) >> 32
  const unsigned sq = (unsigned)(((long long)dh * dh) >> 20);
  const long long q2 = (long long)(((unsigned long long)sq * Y0) >> 24);
  const long long Y = ((long long)Y0 << 29) - ((c - q2 + (1ll << 14)) >> 15);
  // (the exponent word and the shift depend on d alone: one shift and one addition behind Y)
  const unsigned ex = hi >> 20, sub = ex - 2044u;   // sub: 1 or 2 where 1/d is subnormal
  const unsigned eb = ex - 1u < 2044u ? (2044u << 20) - (hi & 0x7ff00000u) : sub - 1u < 2u ? 0u : 0x7ffu << 20;
  const unsigned n = ex - 1u < 2044u ? 0u : sub - 1u < 2u ? sub : 2u;   // (2: a NaN's quarter stays one)
  return __longlong_as_double((long long)((unsigned long long)eb << 32) + (Y >> n));
}

// Register slots of the update warps of smem_potrf.  Slot s < 14 holds column s + 2
// (lane = row); slot s >= 14 holds the pair of columns c0 = 16 + 2 (s - 14) and c0 + 1,
// rows 16..31 only (lane l: row 16 + (l & 15), column c0 + (l >> 4)): a column c needs
// rows c..31, so for c >= 16 half a warp covers it.  Owners rotate over the three warps
// (any seven consecutive columns have all three owners).
constexpr int POTRF_SLOTS = 22, POTRF_FULL = 14;
__host__ __device__ constexpr int potrf_slot_col(int s) { return s < POTRF_FULL ? s + 2 : 16 + 2 * (s - POTRF_FULL); }
__host__ __device__ constexpr int potrf_slot_last(int s) { return s < POTRF_FULL ? s + 2 : 17 + 2 * (s - POTRF_FULL); }
__host__ __device__ constexpr int potrf_slot_owner(int s) { return s < POTRF_FULL ? s % 3 : (s - 12) % 3; }

// When the update warps apply which pivot to which slot: done[j][s] pivots have been
// applied to slot s after step j (the step that starts when pivot j is published).  A step
// applies every pivot so far to the look-ahead slot (column j + 2), and then up to
// POTRF_BUDGET more per warp, to the slots whose columns are needed first; the pivots that
// wait are kept (smem_potrf's Wt holds all).  Applying each pivot to every slot at once
// made the first dozen steps wait for the update warps (eight FP64 instructions a step, 460
// to 680 cycles against the chain's 352) that idled in the last dozen.
constexpr int POTRF_BUDGET = 4;
struct PotrfSchedule {
  int done[TS][POTRF_SLOTS];
};
__host__ __device__ constexpr PotrfSchedule potrf_schedule() {
  PotrfSchedule t{};
  for (int j = 0; j < TS - 2; ++j) {
    for (int s = 0; s < POTRF_SLOTS; ++s) t.done[j][s] = j ? t.done[j - 1][s] : 0;
    for (int w = 0; w < 3; ++w) {
      int left = POTRF_BUDGET;
      for (int s = 0; s < POTRF_SLOTS; ++s) {
        if (potrf_slot_owner(s) != w || potrf_slot_last(s) < j + 2) continue;
        while (t.done[j][s] <= j && (potrf_slot_col(s) <= j + 2 || left > 0)) {
          ++t.done[j][s];
          --left;
        }
      }
    }
  }
  return t;
}

constexpr PotrfSchedule POTRF_SCHEDULE = potrf_schedule();

// The slots from s on of step J of update warp W (see potrf_update_step).
template <int W, int J, int s>
__device__ __forceinline__ void potrf_update_slot(double* S, const double* Wt, int lane, double (&acc)[POTRF_SLOTS]) {
  if constexpr (potrf_slot_owner(s) == W && potrf_slot_last(s) >= J + 2) {
    const int prow = 16 + (lane & 15), half = lane >> 4;
    constexpr int c = potrf_slot_col(s), from = J ? POTRF_SCHEDULE.done[J ? J - 1 : 0][s] : 0,
                  to = POTRF_SCHEDULE.done[J][s];
    if constexpr (to > from) {
#pragma unroll
      for (int p = from; p < to; ++p)
        acc[s] = s < POTRF_FULL ? fma(-Wt[p * TS + lane], S[c * LDS + p], acc[s])
                                : fma(-Wt[p * TS + prow], S[(c + half) * LDS + p], acc[s]);
    }
    if constexpr (c == J + 2 || potrf_slot_last(s) == J + 2) {
      if (s < POTRF_FULL) S[lane * LDS + c] = acc[s];
      else if (c + half == J + 2) S[prow * LDS + c + half] = acc[s];
      nbar_arrive_n<64>(POTRF_BAR_C + (J & 3));
    }
  }
  if constexpr (s + 1 < POTRF_SLOTS) potrf_update_slot<W, J, s + 1>(S, Wt, lane, acc);
}
// Step J (pivot J published) of update warp W (0..2; warp W + 1) of smem_potrf: the
// look-ahead column J + 2 first, handed to the pivot warp, then the other slots that
// potrf_schedule gives this step: a_rc -= w_rp u_cp for the slot's next pivots p in order
// (w_rp = u_rp / d_p from the pivot warp, u_cp from S).  Slots and pivots are compile-time,
// so no predicated-off FMA is issued.
template <int W, int J>
__device__ __forceinline__ void potrf_update_step(double* S, const double* Wt, int lane,
                                                  double (&acc)[POTRF_SLOTS]) {
  nbar_sync(POTRF_BAR_L + (J & 7));
  potrf_update_slot<W, J, 0>(S, Wt, lane, acc);
  if constexpr (J + 1 < TS - 2) potrf_update_step<W, J + 1>(S, Wt, lane, acc);
}
template <int W>
__device__ __forceinline__ void potrf_update_warp(double* S, const double* Wt, int lane) {
  const int prow = 16 + (lane & 15), half = lane >> 4;
  double acc[POTRF_SLOTS];
#pragma unroll
  for (int s = 0; s < POTRF_SLOTS; ++s)
    if (potrf_slot_owner(s) == W)
      acc[s] = s < POTRF_FULL ? S[lane * LDS + potrf_slot_col(s)] : S[prow * LDS + potrf_slot_col(s) + half];
  potrf_update_step<W, 0>(S, Wt, lane, acc);
}

// In-place lower Cholesky of S (TS x TS; entries past n must already be identity).
// Returns 0, or the 1-based column of the first non-positive (or NaN) pivot (the
// tile then holds NaNs).  The strict upper triangle is zeroed.
// The elimination runs in the square-root-free form S = U D^-1 U^T (u_rk: column k
// after pivots 0..k-1, d_k = u_kk), and L = U D^{-1/2} is formed at the end.  Warp 0 does nothing but the pivot chain: for pivot k it takes
// column k, already updated through pivot k-2 by its owner (awaited and loaded while
// pivot k-1's reciprocal was formed), applies pivot k-1 itself
// (it holds w_{:,k-1} = u_{:,k-1} / d_{k-1} in registers, the multiplier u_{k,k-1} is
// one shuffle), stores u_{:,k} to S, forms 1/d_k and w_{:,k}, and hands w_{:,k} to the
// update warps through Wt (TS x TS scratch, row k: w_{:,k}).  The chain is bound by
// latency: two FP64 instructions a pivot at 64 cycles, the reciprocal on the integer pipe
// (rcp_finish: 120 cycles against 227 in FP64), the shuffles.  Its loop is rolled
// (unrolled, the ~60 instructions a pivot run once each, at the rate of instruction fetch:
// ~5.5 cycles an instruction), and the next column's barrier and load sit behind the seed
// of the reciprocal, under its latency.  In the factorization kernel a tile takes 14.2k
// cycles, ~405 a pivot (18k before the integer reciprocal, the update schedule and the
// scaling of the first 30 columns beside the last two pivots): a column link at b = 128 or
// 333 took 19.2 us instead of 20.3 for it, and takes 15.4 with the solves that follow the
// pivots (smem_trsm_follow).
// Warps 1-3 apply every pivot to the later columns (potrf_update_warp), the column that
// the pivot warp needs next first; each entry receives its updates in pivot order.
// Barrier ids rotate over 8 (pivots) and 4 (look-ahead columns): before the pivot warp
// publishes pivot p+8 (the barrier id of pivot p again), each update warp has handed it
// one of columns p+2 .. p+8 (seven consecutive columns have all three owners) and so
// consumed pivot p; the pivot warp consumes look-ahead column p before it can publish
// the pivot that look-ahead column p+4 needs.
// With Wg (TS x TS words of global memory holding WORD_EMPTY) every pivot k is also written
// there as it forms, row k: w_{:,k} with d_k in w_kk's place, for tasks on other SMs that
// follow the elimination (wait_word).  A non-positive pivot and those after it are not: the
// followers wait until the launch is given up, so no later tile starts from this one, and no
// row behind it can be reported in its place.
// Out of line: its code is ~25 KB, once per kernel is enough.
static __device__ __noinline__ int smem_potrf_at(unsigned s_addr, unsigned w_addr, double* Wg) {
  double* S = reinterpret_cast<double*>(__cvta_shared_to_generic(s_addr));
  double* Wt = reinterpret_cast<double*>(__cvta_shared_to_generic(w_addr));
  __shared__ int s_info;
  const int r = threadIdx.x & 31, g = threadIdx.x >> 5;
  __syncthreads();
  if (g == 0) {
    double a = S[r * LDS];         // column k through pivot k-1 (column 0 of U is column 0 of S)
    double an = S[r * LDS + 1];    // column k+1 through pivot k-1 (column 1: no update yet)
    double dk = 1.0;               // lane k keeps d_k
    int bad = 0;                   // the first non-positive pivot
#pragma unroll 1
    for (int k = 0; k < TS; ++k) {
      const double d = __shfl_sync(0xffffffffu, a, k);
      const double ub = __shfl_sync(0xffffffffu, a, (k + 1) & 31);   // u_{k+1,k}
      const float seed = rcp_seed(d);
      // Column k+1, updated through pivot k-1 by its owner, is awaited and loaded while
      // this pivot's reciprocal is formed, off the chain.
      if (k >= 1 && k < TS - 1) {
        nbar_sync_n<64>(POTRF_BAR_C + ((k - 1) & 3));
        an = S[r * LDS + k + 1];
      }
      S[r * LDS + k] = a;   // (rows below k only; the others are left out when L is formed)
      if (r == k) dk = d;
      const double w = a * rcp_finish(d, seed);
      a = fma(-w, ub, an);
      if (k < TS - 2) {
        Wt[k * TS + r] = w;
        nbar_arrive(POTRF_BAR_L + (k & 7));
      }
      if (!bad && !positive_bits(d)) bad = k + 1;   // (uniform)
      if (Wg && !bad) st_word(Wg + k * TS + r, r == k ? d : w);
    }
    if (r == 0) s_info = bad;
    // L = U D^{-1/2}: the last two columns here, the others by warps 1-3, which have them
    // complete two pivots earlier
    const double y = rsqrt3(dk);
#pragma unroll
    for (int c = TS - 2; c < TS; ++c) {
      const double l = S[r * LDS + c] * __shfl_sync(0xffffffffu, y, c);
      S[r * LDS + c] = r >= c ? l : 0.0;
    }
  } else {
    if (g == 1)
      potrf_update_warp<0>(S, Wt, r);
    else if (g == 2)
      potrf_update_warp<1>(S, Wt, r);
    else
      potrf_update_warp<2>(S, Wt, r);
    // (each warp scales its columns from the diagonal it finds there before any is scaled)
    const double y = rsqrt3(S[r * LDS + r]);
    nbar_sync_n<NT - 32>(POTRF_BAR_L + 2);
#pragma unroll
    for (int q = 0; q < (TS - 2) / 3; ++q) {
      const int c = 3 * q + g - 1;
      const double l = S[r * LDS + c] * __shfl_sync(0xffffffffu, y, c);
      S[r * LDS + c] = r >= c ? l : 0.0;
    }
  }
  __syncthreads();
  const int info = s_info;
  __syncthreads();
  return info;
}

// (the call passes shared-window addresses, so that the body's accesses are shared ones)
static __device__ __forceinline__ int smem_potrf(double* S, double* Wt, double* Wg = nullptr) {
  return smem_potrf_at((unsigned)__cvta_generic_to_shared(S), (unsigned)__cvta_generic_to_shared(Wt), Wg);
}

// X <- X * F^{-T} with F lower triangular; rd = 1/diag(F) (tile_diag_recip).  Row r
// solves x_r F^T = X_r by forward substitution over the columns.
static __device__ void smem_trsm_rlt(double* X, const double* F, const double* rd) {
  __shared__ double xs[2 * TS];
  const int r = threadIdx.x & 31, g = threadIdx.x >> 5;
  __syncthreads();
  double acc[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) acc[q] = X[r * LDS + g + 4 * q];
#pragma unroll
  for (int j = 0; j < TS; ++j) {
    double* xb = xs + (j & 1) * TS;
    if (g == (j & 3)) {
      const double x = acc[j >> 2] * rd[j];
      acc[j >> 2] = x;
      xb[r] = x;
    }
    __syncthreads();
    const double xr = xb[r];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (col_after(q, j, g)) acc[q] = fma(-xr, F[(g + 4 * q) * LDS + j], acc[q]);
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) X[r * LDS + g + 4 * q] = acc[q];
  __syncthreads();
}

// Rows row0 .. row0 + 7 of X <- X * F^{-T} (F lower triangular, identity padded).
// Warp w solves rows row0 + 2w and row0 + 2w + 1: lane l holds columns (l & 15) and
// (l & 15) + 16 of row row0 + 2w + (l >> 4).  Column j is finished on the lane that
// holds it and broadcast to its row's 16 lanes with one shuffle, so the sweep needs no
// barrier; the later columns are updated with one FMA each.  With FS (a copy of F
// whose row j is scaled by 1/F_jj, see tile_scale_rows_by_recip) and X's columns
// pre-scaled the same way, no multiplication is left on the column chain.
static __device__ void smem_trsm_rlt_rows8(double* X, const double* FS, const double* rd, int row0) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int row = row0 + 2 * w + (lane >> 4), cg = lane & 15, base = lane & 16;
  __syncthreads();
  double a0 = X[row * LDS + cg] * rd[cg], a1 = X[row * LDS + cg + 16] * rd[cg + 16];
#pragma unroll
  for (int j = 0; j < TS; ++j) {
    const double xj = __shfl_sync(0xffffffffu, j < 16 ? a0 : a1, base | (j & 15));
    if (j < 15) {
      const double f0 = FS[cg * LDS + j];
      if (cg > j) a0 = fma(-xj, f0, a0);
    }
    const double f1 = FS[(cg + 16) * LDS + j];
    if (j < 16 || cg + 16 > j) a1 = fma(-xj, f1, a1);
  }
  __syncthreads();
  X[row * LDS + cg] = a0;
  X[row * LDS + cg + 16] = a1;
  __syncthreads();
}

// ---- solves that follow the factorization of their diagonal tile ------------------
// X <- X F^{-T} computed while the diagonal tile is still being factored on another SM: W
// (global words, see smem_potrf's Wg) gives w_kj = u_kj / d_j and d_j of pivot after pivot,
// and y_j = s_j - sum_{i<j} y_i w_ji, x_j = y_j / sqrt(d_j) is the solve in the
// square-root-free form.  Waiting for the finished tile instead puts its scaling, store,
// flag and reload and the whole solve (9.4 us for 32 rows) behind the last pivot, for every
// tile of the column.  Four pivots, one word a thread, are staged at a time into Ws (TS x TS,
// row j: w_:j) by follow_stage; the next four are requested before the four are used.
struct FollowWords {
  const double* W;
  long long ahead;   // this thread's word of the next four pivots, as last read
};
__device__ __forceinline__ bool follow_begin(FollowWords& f, const Ctl& c, const double* W) {
  double v;
  bool ok = true;
  if (threadIdx.x == 0) ok = wait_word(c, W, v);   // (one thread polls until the first pivot)
  ok = __syncthreads_and(ok);
  f.W = W;
  f.ahead = ld_word(W + threadIdx.x);
  return ok;
}
__device__ __forceinline__ bool follow_stage(FollowWords& f, const Ctl& c, double* Ws, int j0) {
  double v = __longlong_as_double(f.ahead);
  bool ok = true;
  if (f.ahead == WORD_EMPTY) ok = wait_word(c, f.W + j0 * TS + threadIdx.x, v);
  Ws[j0 * TS + threadIdx.x] = v;
  ok = __syncthreads_and(ok);
  if (j0 + 4 < TS) f.ahead = ld_word(f.W + (j0 + 4) * TS + threadIdx.x);
  return ok;
}

// Rows row0 .. row0 + 7 of X (the split of smem_trsm_rlt_rows8).  Returns false, uniformly,
// when a wait was given up.
static __device__ __forceinline__ bool smem_trsm_follow_rows8_at(unsigned x_addr, int* ctrl, unsigned long long wait_ns,
                                                              const double* W, unsigned ws_addr, int row0) {
  double* X = reinterpret_cast<double*>(__cvta_shared_to_generic(x_addr));
  double* Ws = reinterpret_cast<double*>(__cvta_shared_to_generic(ws_addr));
  const Ctl c{ctrl, nullptr, 0, wait_ns, nullptr};
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int row = row0 + 2 * w + (lane >> 4), cg = lane & 15, base = lane & 16;
  __syncthreads();
  double a0 = X[row * LDS + cg], a1 = X[row * LDS + cg + 16];
  double s0 = 0.0;
  FollowWords f;
  if (!follow_begin(f, c, W)) return false;
#pragma unroll 1
  for (int j0 = 0; j0 < TS; j0 += 4) {
    if (!follow_stage(f, c, Ws, j0)) return false;
    if (j0 < 16) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int j = j0 + q;
        const double yj = __shfl_sync(0xffffffffu, a0, base | j);
        const double f0 = Ws[j * TS + cg], f1 = Ws[j * TS + cg + 16];
        if (cg > j) a0 = fma(-yj, f0, a0);
        a1 = fma(-yj, f1, a1);
      }
    } else {
      if (j0 == 16) s0 = rsqrt3(Ws[cg * TS + cg]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int j = j0 + q;
        const double yj = __shfl_sync(0xffffffffu, a1, base | (j & 15));
        const double f1 = Ws[j * TS + cg + 16];
        if (cg + 16 > j) a1 = fma(-yj, f1, a1);
      }
    }
  }
  X[row * LDS + cg] = a0 * s0;
  X[row * LDS + cg + 16] = a1 * rsqrt3(Ws[(cg + 16) * TS + cg + 16]);
  __syncthreads();
  return true;
}

// All 32 rows of X: warp w owns rows 8 w .. 8 w + 7, four lanes a row with columns (lane &
// 3) + 4 q, so that a column goes to its row's lanes by one shuffle and only the staging has
// barriers.  144 FP64 instructions a warp (9.2k cycles), under the factorization's 14k.
// rs: TS doubles.
static __device__ __noinline__ bool smem_trsm_follow_at(unsigned x_addr, int* ctrl, unsigned long long wait_ns,
                                                        const double* W, unsigned ws_addr, unsigned rs_addr) {
  double* X = reinterpret_cast<double*>(__cvta_shared_to_generic(x_addr));
  double* Ws = reinterpret_cast<double*>(__cvta_shared_to_generic(ws_addr));
  double* rs = reinterpret_cast<double*>(__cvta_shared_to_generic(rs_addr));
  const Ctl c{ctrl, nullptr, 0, wait_ns, nullptr};
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int row = 8 * w + (lane >> 2), cg = lane & 3;
  FollowWords f;
  if (!follow_begin(f, c, W)) return false;   // (its barrier covers the caller's writes of X)
  double y[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) y[q] = X[row * LDS + cg + 4 * q];
#pragma unroll
  for (int J = 0; J < 8; ++J) {
    if (!follow_stage(f, c, Ws, 4 * J)) return false;
#pragma unroll
    for (int ph = 0; ph < 4; ++ph) {
      const double* wj = Ws + (4 * J + ph) * TS + cg;
      const double yj = __shfl_sync(0xffffffffu, y[J], (lane & 28) | ph);
      if (ph < 3 && cg > ph) y[J] = fma(-yj, wj[4 * J], y[J]);
#pragma unroll
      for (int q = J + 1; q < 8; ++q) y[q] = fma(-yj, wj[4 * q], y[q]);
    }
  }
  if (threadIdx.x < TS) rs[threadIdx.x] = rsqrt3(Ws[threadIdx.x * TS + threadIdx.x]);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 8; ++q) X[row * LDS + cg + 4 * q] = y[q] * rs[cg + 4 * q];
  __syncthreads();
  return true;
}

// The 32-row solve is out of line, as smem_potrf_at (inlined, the factorization at b = 3072
// takes 78.4 ms instead of 74.7); the row groups', on the column chain, is inlined (b = 333,
// nt = 60: 5.66 ms against 5.80).
static __device__ __forceinline__ bool smem_trsm_follow_rows8(double* X, const Ctl& c, const double* W, double* Ws,
                                                              int row0) {
  return smem_trsm_follow_rows8_at((unsigned)__cvta_generic_to_shared(X), c.ctrl, c.wait_ns, W,
                                   (unsigned)__cvta_generic_to_shared(Ws), row0);
}
static __device__ __forceinline__ bool smem_trsm_follow(double* X, const Ctl& c, const double* W, double* Ws,
                                                        double* rs) {
  return smem_trsm_follow_at((unsigned)__cvta_generic_to_shared(X), c.ctrl, c.wait_ns, W,
                             (unsigned)__cvta_generic_to_shared(Ws), (unsigned)__cvta_generic_to_shared(rs));
}

// FS <- F with row j scaled by rd[j] = 1/F_jj (the strict lower part is what the
// row solves read).  Caller syncs before and after.
__device__ __forceinline__ void tile_scale_rows_by_recip(double* FS, const double* F, const double* rd) {
#pragma unroll
  for (int k = 0; k < PER_THREAD; ++k) {
    const int idx = threadIdx.x + k * NT;
    const int r = idx / TS, c = idx % TS;
    FS[r * LDS + c] = F[r * LDS + c] * rd[r];
  }
}

// X <- X * F^{-1} with F lower triangular; rd = 1/diag(F).  Row r solves x_r F = X_r
// by backward substitution over the columns.  Warp w owns rows 8 w .. 8 w + 7, four lanes a
// row with columns (lane & 3) + 4 q: a column goes to its row's lanes by one shuffle, so the
// substitution has no barrier: 176 FP64 instructions a warp, 14.9k cycles a tile against 17k
// with lane = row, a column's owner warp and a barrier per column.
static __device__ void smem_trsm_rln(double* X, const double* F, const double* rd) {
  const int lane = threadIdx.x & 31, row = 8 * (threadIdx.x >> 5) + (lane >> 2), cg = lane & 3;
  __syncthreads();
  double y[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) y[q] = X[row * LDS + cg + 4 * q];
#pragma unroll
  for (int J = 7; J >= 0; --J) {
#pragma unroll
    for (int ph = 3; ph >= 0; --ph) {
      const int j = 4 * J + ph;
      const double* fj = F + j * LDS + cg;
      const double x = y[J] * rd[j];
      if (cg == ph) y[J] = x;
      const double xj = __shfl_sync(0xffffffffu, x, (lane & 28) | ph);
      if (ph > 0 && cg < ph) y[J] = fma(-xj, fj[4 * J], y[J]);
#pragma unroll
      for (int q = 0; q < J; ++q) y[q] = fma(-xj, fj[4 * q], y[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) X[row * LDS + cg + 4 * q] = y[q];
  __syncthreads();
}

}  // namespace gbta
