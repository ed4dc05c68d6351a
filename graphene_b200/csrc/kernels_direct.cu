// Block-ILU(0) / DILU substitution and Gauss-Seidel sweeps over row records
// read straight into registers (ilu/Solver.cpp:367-550,
// gauss-seidel/Solver.cpp:45-86; the operations and their order are those of
// the level-ring kernels, so results are the same bits).
//
// One thread block of WARPS warps per tile, every warp computing. A level's
// rows are spread over the block's threads (32 * WARPS rows a step). A
// record's address depends only on the step table, never on x, so every
// thread copies its own records DEPTH steps ahead (cp.async into places of
// shared memory that only it reads): no producer, no mbarrier and no
// hand-over between threads. Between two barriers lie the x reads, the row's
// arithmetic and one store.
#include <algorithm>
#include <type_traits>

#include "bulk.cuh"
#include "device.hpp"
#include "devmath.cuh"
#include "krylov.hpp"
#include "sell.cuh"

namespace gr {
namespace dev {

struct DirectView {
  const int* __restrict__ tileStart;
  const int* __restrict__ stepStart;
  const uint32_t* __restrict__ steps;
  const uint32_t* __restrict__ stepUnit;
  const uint4* __restrict__ data;  // the steps' blocks
  int xSlots;   // slots of x in shared memory (a multiple of 4)
  int maxRows;  // rows of the largest tile
  bool fetch;        // whether a block keeps its stream on its way to L2 ahead of its copies
  bool longForward;  // ILU: whether the forward sweep has rows of more than three entries
};

// Per-thread asynchronous copies of BYTES into shared memory (32-bit shared
// address), in groups that complete in order: copyOr0 fills with zeros when
// !on, copyIf leaves the old bytes.
template <int BYTES>
__device__ __forceinline__ void copyOr0(uint32_t dst, const void* src, bool on) {
  const uint32_t bytes = on ? BYTES : 0;
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(bytes)
                 : "memory");
}
template <int BYTES>
__device__ __forceinline__ void copyIf(uint32_t dst, const void* src, bool on) {
  if (BYTES == 16)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p cp.async.cg.shared.global [%0], [%1], 16;\n\t}" ::"r"(dst),
        "l"(src), "r"(static_cast<uint32_t>(on))
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p cp.async.ca.shared.global [%0], [%1], %2;\n\t}" ::"r"(dst),
        "l"(src), "n"(BYTES), "r"(static_cast<uint32_t>(on))
        : "memory");
}
template <bool FILL, int BYTES>
__device__ __forceinline__ void copyRec(uint32_t dst, const void* src, bool on) {
  if (FILL) copyOr0<BYTES>(dst, src, on);
  else copyIf<BYTES>(dst, src, on);
}
__device__ __forceinline__ void copyCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copyWait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Reads of shared memory at a 32-bit shared address.
__device__ __forceinline__ uint4 shared16(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(at)
               : "memory");
  return v;
}
__device__ __forceinline__ uint2 shared8(uint32_t at) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t shared4(uint32_t at) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
  return v;
}

// A thread's places for records in shared memory: planes of THREADS * DEPTH
// 16-byte words (one a triple for float, two for double), then 8 bytes of
// {tail word, diagonal} (float) or the diagonal (double), then the second
// triple's third slot (float). x follows.
template <class MV, int NT, int THREADS, int DEPTH>
struct DirectShape {
  static constexpr bool F32 = sizeof(MV) == 4;
  static constexpr int words = F32 ? 1 : 2;  // 16-byte words a triple
  static constexpr int plane = 16 * DEPTH * THREADS;
  static constexpr int tail = NT * words * plane;
  static constexpr int third = tail + 8 * DEPTH * THREADS;
  static constexpr int x = third + (F32 && NT == 2 ? 4 * DEPTH * THREADS : 0);
};

// A record in registers. A thread without a row in a step finds in its place
// zeros or an earlier record: its slots are some tile's, so reading x there
// is harmless, and it stores nothing.
template <class MV, int NT>
struct DirectRec {
  static constexpr bool F32 = sizeof(MV) == 4;
  static constexpr int words = F32 ? 1 : 2;
  uint4 a[NT * words];
  uint32_t t[NT];
  uint2 inv;  // the diagonal's bits (float: .x)

  // Starts the copies of this thread's record of the step with word w, whose
  // block starts at `block`, into the place at shared addresses pa (its first
  // word), pt and pc (tail and third slot). DIAG, LONG: whether the step has
  // diagonals and may have second triples.
  template <class S, bool FILL, bool DIAG, bool LONG>
  static __device__ __forceinline__ void copy(uint32_t pa, uint32_t pt, uint32_t pc, const uint4* block, uint32_t tid,
                                              uint32_t w) {
    const DirectBlock<sizeof(MV)> at(w, DIAG);
    const bool on = tid < (w & 0xFFu);
    const char* p = reinterpret_cast<const char*>(block + tid);
    copyRec<FILL, 16>(pa, p, on);
    if (!F32) copyRec<FILL, 16>(pa + S::plane, p + at.plane, on);
    const char* b = reinterpret_cast<const char*>(block);
    if (DIAG) copyRec<FILL, 8>(pt, b + at.tail + 8 * tid, on);
    else if (F32) copyRec<FILL, 4>(pt, b + at.tail + 4 * tid, on);
    if constexpr (LONG) {
      const bool two = tid < ((w >> kDirectLongShift) & 0xFFu);
      copyIf<16>(pa + words * S::plane, p + at.second, two);
      if (F32) copyIf<4>(pc, b + at.third + 4 * tid, two);
      else copyIf<16>(pa + 3 * S::plane, p + at.second + at.plane2, two);
    }
  }
  template <class S>
  __device__ __forceinline__ void read(uint32_t pa, uint32_t pt, uint32_t pc) {
#pragma unroll
    for (int w = 0; w < NT * words; ++w) a[w] = shared16(pa + w * S::plane);
    const uint2 u = shared8(pt);
    if (F32) {
      t[0] = u.x;
      inv.x = u.y;
      if (NT == 2) t[NT - 1] = shared4(pc);
    } else {
      inv = u;
#pragma unroll
      for (int k = 0; k < NT; ++k) t[k] = a[(2 * k + 1) % (NT * words)].w;
    }
  }
  // Slots as stored (4 x slot).
  __device__ __forceinline__ uint32_t row() const { return t[0] >> 16; }
  __device__ __forceinline__ uint32_t slots(int k) const { return F32 ? a[k].w : a[(2 * k + 1) % (NT * words)].z; }
  __device__ __forceinline__ uint32_t third(int k) const { return t[k] & 0xFFFFu; }
  static __device__ __forceinline__ MV of(uint32_t lo, uint32_t hi) {
    if constexpr (F32) return __uint_as_float(lo);
    else return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
  }
  __device__ __forceinline__ MV v(int k, int e) const {
    if constexpr (F32) return __uint_as_float(e == 0 ? a[k].x : e == 1 ? a[k].y : a[k].z);
    else return e == 0 ? of(a[2 * k].x, a[2 * k].y) : e == 1 ? of(a[2 * k].z, a[2 * k].w) : of(a[2 * k + 1].x, a[2 * k + 1].y);
  }
  __device__ __forceinline__ MV diag() const { return of(inv.x, inv.y); }
};

template <class W>
__device__ __forceinline__ W& slotOf(unsigned char* x, uint32_t stored) {
  return *reinterpret_cast<W*>(x + (sizeof(W) / 4) * stored);
}

// The x values that triple k of a record reads (padding: the zero slot), and
// temp - v0 x0 - v1 x1 - v2 x2 in order (padding: value 0, temp unchanged).
template <class W>
struct DirectX {
  W v[3];
  template <class MV, int NT>
  __device__ __forceinline__ void read(const DirectRec<MV, NT>& r, int k, unsigned char* x) {
    const uint32_t s = r.slots(k);
    v[0] = slotOf<W>(x, s & 0xFFFFu);
    v[1] = slotOf<W>(x, s >> 16);
    v[2] = slotOf<W>(x, r.third(k));
  }
  template <class MV, int NT>
  __device__ __forceinline__ W dot(W temp, const DirectRec<MV, NT>& r, int k) const {
#pragma unroll
    for (int e = 0; e < 3; ++e) temp = sub(temp, mul(cvt<W>(r.v(k, e)), v[e]));
    return temp;
  }
};

// 16 bytes of consecutive vector elements.
template <class X>
struct Vec16;
template <>
struct Vec16<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void load(const float* p, float (&o)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&o)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
  }
};
template <>
struct Vec16<double> {
  static constexpr int N = 2;
  static __device__ __forceinline__ void load(const double* p, double (&o)[2]) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    o[0] = v.x; o[1] = v.y;
  }
  static __device__ __forceinline__ void store(double* p, const double (&o)[2]) {
    *reinterpret_cast<double2*>(p) = make_double2(o[0], o[1]);
  }
};

// A tile's rows as 16-byte groups of vectors whose first element (row 0 of
// the matrix) is 16-byte aligned, from the tile's first 128-byte line on:
// rows [lead, lead + N * groups) of the tile. (Warps that start in the middle
// of a line make L2 fetch it twice.)
struct RowGroups {
  int lead, groups;
};
template <class X>
__device__ __forceinline__ RowGroups rowGroups(int base, int nRows, bool vec) {
  constexpr int N = Vec16<X>::N, L = 8 * N;
  if (!vec) return {0, 0};
  const int lead = min(nRows, (L - base % L) % L);
  return {lead, (nRows - lead) / N};
}

// The prologue's vector (SPro: b, or the fused p / s update, which is also
// written back) of the tile's rows into dst, 16 bytes a load and U groups a
// thread at once so that a block keeps up to 96 bytes a thread in flight;
// rows outside the groups one at a time.
template <int THREADS, class X, class W>
__device__ __forceinline__ void tilePrologue(const SPro<X>& pro, int base, int nRows, bool vec, W* dst) {
  constexpr int N = Vec16<X>::N, U = 2;
  X beta = X(0), omega = X(0), alpha = X(0);
  bool first = true;
  if (const KState* st = pro.state()) {
    beta = cvt<X>(st->beta);
    omega = cvt<X>(st->omega);
    alpha = cvt<X>(st->alpha);
    first = st->iter == 0;
  }
  const int tid = static_cast<int>(threadIdx.x);
  const RowGroups g = rowGroups<X>(base, nRows, vec);
  const bool plain = pro.kind == static_cast<int>(Prologue::Plain);
  const bool pu = pro.kind == static_cast<int>(Prologue::PUpdate);
  for (int i0 = tid; i0 < g.groups; i0 += U * THREADS) {
    X r[U][N], p[U][N], v[U][N];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (i0 + u * THREADS >= g.groups) continue;
      const int at = base + g.lead + N * (i0 + u * THREADS);
      if (plain) {
        Vec16<X>::load(pro.b + at, r[u]);
      } else {
        Vec16<X>::load(pro.r + at, r[u]);
        if (!(pu && first)) Vec16<X>::load(pro.v + at, v[u]);
        if (pu && !first) Vec16<X>::load(pro.pOrS + at, p[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (i0 + u * THREADS >= g.groups) continue;
      const int row = g.lead + N * (i0 + u * THREADS);
      if (!plain) {
#pragma unroll
        for (int j = 0; j < N; ++j) {
          if (!pu) r[u][j] = sub(r[u][j], mul(alpha, v[u][j]));
          else if (!first) r[u][j] = add(r[u][j], mul(beta, sub(p[u][j], mul(omega, v[u][j]))));
        }
        Vec16<X>::store(pro.pOrS + base + row, r[u]);
      }
#pragma unroll
      for (int j = 0; j < N; ++j) dst[row + j] = cvt<W>(r[u][j]);
    }
  }
  const int rest = nRows - N * g.groups;
  for (int i0 = tid; i0 < rest; i0 += 4 * THREADS) {
    int row[4];
    X v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = i0 + j * THREADS;
      row[j] = k >= rest ? -1 : k < g.lead ? k : k + N * g.groups;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (row[j] >= 0) v[j] = pro(base + row[j], beta, omega, alpha, first);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (row[j] >= 0) dst[row[j]] = cvt<W>(v[j]);
  }
}

// y rows of the tile from shared memory, 16 bytes a store where aligned.
template <int THREADS, class X, class W>
__device__ __forceinline__ void tileStore(X* __restrict__ y, int base, int nRows, bool vec, const W* xs) {
  constexpr int N = Vec16<X>::N;
  const RowGroups g = rowGroups<X>(base, nRows, vec);
  for (int i = threadIdx.x; i < g.groups; i += THREADS) {
    const int row = g.lead + N * i;
    X o[N];
#pragma unroll
    for (int j = 0; j < N; ++j) o[j] = cvt<X>(xs[row + j]);
    Vec16<X>::store(y + base + row, o);
  }
  const int rest = nRows - N * g.groups;
  for (int k = threadIdx.x; k < rest; k += THREADS) {
    const int row = k < g.lead ? k : k + N * g.groups;
    y[base + row] = cvt<X>(xs[row]);
  }
}

// 16-byte units of a tile's stream that its block keeps on their way to L2
// beyond its copies. With the stream in DRAM the copies alone, DEPTH steps
// ahead, leave too few bytes in flight: on B200, L2 flushed, 8 KB ahead ran
// the 128^3 / 1024 ILU(0) in 41.3 us against 45.9 without (float64 63.6
// against 68.3), 96^3 / 432 in 30.8 against 31.6, the 100^3 mesh's two sweeps
// in 51.6 against 56.1. Back to back, the 128^3 stream stays in L2 and nothing
// changes (35.1, 34.9 without); the float64 one does not (49.3, 53.4 without).
// 4 and 16 KB ran within 3 us of it, a whole tile ahead slower.
// Streams of less than 32 MB (kDirectFetchUnits) stay in L2 between a solve's
// applications, and the 32^3 / 64 one takes 8.2 us without and up to 10 with
// the prefetch, so they go without.
constexpr uint32_t kDirectL2 = 512;

// The copies, reads and barriers of a block's steps.
template <class MV, class W, int NT, int WARPS, int DEPTH>
struct DirectSteps {
  static constexpr int THREADS = 32 * WARPS, U = kDirectUnroll;
  static_assert(U == 4 && (DEPTH == U || DEPTH == 2 * U), "one or two groups of places");
  using S = DirectShape<MV, NT, THREADS, DEPTH>;
  using Rec = DirectRec<MV, NT>;
  const uint4* block;    // the next step's block to copy
  const uint4* last;     // the end of the tile's blocks
  uint32_t toFetch = 0;  // thread 0: units at its end that are not yet on their way to L2
  uint32_t steps;        // shared address of the next step's word
  uint32_t tid;
  uint32_t pa, pt, pc;   // shared addresses of the places of the current group of U steps
  int other = U * THREADS;  // elements from there to the other group's places
  uint32_t word, ahead;  // the words of the next step and of the step DEPTH after it
  Rec rec[2];            // the records of the next step and the one after, in turn

  // Starts the copies of the step DEPTH later (word w) into place d of the
  // current group. Threads without a row keep what their place held.
  template <int d, bool DIAG, bool LONG>
  __device__ __forceinline__ void copy(uint32_t w) {
    Rec::template copy<S, false, DIAG, LONG>(pa + 16 * THREADS * d, pt + 8 * THREADS * d, pc + 4 * THREADS * d, block,
                                             tid, w);
    block += w >> kDirectUnitShift;
    copyCommit();
  }
  // Keeps kDirectL2 units beyond the next copy on their way to L2.
  __device__ __forceinline__ void fetch() {
    const uint32_t left = static_cast<uint32_t>(last - block), keep = left > kDirectL2 ? left - kDirectL2 : 0;
    if (keep < toFetch) prefetchL2(last - toFetch, 16 * (toFetch - keep));
    toFetch = keep;
  }
  template <int d>
  __device__ __forceinline__ void copyFirst(uint32_t w) {
    const uint32_t qa = pa + 16 * THREADS * d, qt = pt + 8 * THREADS * d, qc = pc + 4 * THREADS * d;
    if (w & kDirectDiag) Rec::template copy<S, true, true, NT == 2>(qa, qt, qc, block, tid, w);
    else Rec::template copy<S, true, false, NT == 2>(qa, qt, qc, block, tid, w);
    block += w >> kDirectUnitShift;
    copyCommit();
  }
  // The first DEPTH steps' copies, by the table in global memory.
  __device__ __forceinline__ DirectSteps(const DirectView& V, const unsigned char* smem, int T,
                                         const uint32_t* stepsShared)
      : steps(smemAddr(stepsShared)), tid(threadIdx.x) {
    const int t0 = V.stepStart[T];
    const uint32_t* table = V.steps + t0;
    const uint32_t s = smemAddr(smem);
    pa = s + 16 * tid;
    pt = s + S::tail + 8 * tid;
    pc = s + S::third + 4 * tid;
    block = V.data + __ldg(V.stepUnit + t0);
    last = V.data + __ldg(V.stepUnit + V.stepStart[T + 1] - 1);
    if (V.fetch && tid == 0) {
      toFetch = static_cast<uint32_t>(last - block);
      fetch();
    }
    word = __ldg(table + kDirectHead);
    ahead = __ldg(table + kDirectHead + DEPTH);
    uint32_t w[DEPTH];
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) w[d] = __ldg(table + kDirectHead + d);
    copyFirst<0>(w[0]);
    copyFirst<1>(w[1]);
    copyFirst<2>(w[2]);
    copyFirst<3>(w[3]);
    if constexpr (DEPTH > U) {
      copyFirst<4>(w[DEPTH - 4]);
      copyFirst<5>(w[DEPTH - 3]);
      copyFirst<6>(w[DEPTH - 2]);
      copyFirst<7>(w[DEPTH - 1]);
    }
  }
  // Waits for the first step's record.
  __device__ __forceinline__ void start() {
    copyWait<DEPTH - 1>();
    rec[0].template read<S>(pa, pt, pc);
  }
  // One step, its record in place d of the current group. It reads its x
  // values, then, while they are on their way, starts the copy of the step
  // DEPTH later into its own place and reads the next step's record and
  // word; what follows the x values is the arithmetic, one store and the
  // barrier. begin(record, x's own value) and end(record, that value, the
  // sum) give the row's first and last operation. LONG: rows may have a
  // second triple; DIAG2, LONG2: the step DEPTH later has diagonals, may have
  // second triples.
  template <int d, bool LONG, bool DIAG2, bool LONG2, class F, class G>
  __device__ __forceinline__ void step(unsigned char* x, F&& begin, G&& end) {
    const Rec& r = rec[d & 1];
    const uint32_t w = word;
    const bool two = LONG && tid < ((w >> kDirectLongShift) & 0xFFu);
    W& xr = slotOf<W>(x, r.row());
    const W was = xr;
    DirectX<W> x1, x2;
    x1.read(r, 0, x);
    if (LONG && two) x2.read(r, NT - 1, x);
    copy<d, DIAG2, LONG2>(ahead);
    if (d == U - 1 && DEPTH > U) {
      pa += 16 * other;
      pt += 8 * other;
      pc += 4 * other;
      other = -other;
    }
    copyWait<DEPTH - 1>();
    constexpr int n = (d + 1) % U;
    rec[(d + 1) & 1].template read<S>(pa + 16 * THREADS * n, pt + 8 * THREADS * n, pc + 4 * THREADS * n);
    word = shared4(steps + 4 * (d + 1));
    ahead = shared4(steps + 4 * (d + 1 + DEPTH));
    W sum = x1.dot(begin(r, was), r, 0);
    if (LONG && two) sum = x2.dot(sum, r, NT - 1);
    const W v = end(r, was, sum);
    if (tid < (w & 0xFFu)) xr = v;
    if (WARPS == 1) __syncwarp();
    else if (w & kDirectEnd) __syncthreads();
  }
  // `count` steps, a multiple of U.
  template <bool LONG, bool DIAG2, bool LONG2, class F, class G>
  __device__ __forceinline__ void run(uint32_t count, unsigned char* x, F&& begin, G&& end) {
    const uint32_t stop = steps + 4 * count;
    while (steps != stop) {
      if (toFetch != 0) fetch();
      step<0, LONG, DIAG2, LONG2>(x, begin, end);
      step<1, LONG, DIAG2, LONG2>(x, begin, end);
      step<2, LONG, DIAG2, LONG2>(x, begin, end);
      step<3, LONG, DIAG2, LONG2>(x, begin, end);
      steps += 4 * U;
    }
  }
};

template <int WARPS>
__device__ __forceinline__ void tileBarrier() {
  if (WARPS == 1) __syncwarp();
  else __syncthreads();
}

// y = M^-1 * prologue for every tile.
template <class MV, class W, int NT, int WARPS, int DEPTH, bool DILU>
__global__ void __launch_bounds__(32 * WARPS) iluDirectKernel(DirectView V, SPro<W> pro, W* __restrict__ y, bool vec) {
  constexpr int THREADS = 32 * WARPS;
  using Rec = DirectRec<MV, NT>;
  extern __shared__ __align__(16) unsigned char smem[];
  const KState* st = pro.state();
  if (st && st->done) return;
  const int T = blockIdx.x, tid = threadIdx.x;
  const int base = V.tileStart[T], nRows = V.tileStart[T + 1] - base;
  using Steps = DirectSteps<MV, W, NT, WARPS, DEPTH>;
  unsigned char* x = smem + Steps::S::x;
  W* xs = reinterpret_cast<W*>(x);
  uint32_t* steps = reinterpret_cast<uint32_t*>(xs + V.xSlots);
  Steps sweep(V, smem, T, steps + kDirectHead);
  const int t0 = V.stepStart[T], words = V.stepStart[T + 1] - t0;
  for (int i = tid; i < words; i += THREADS) steps[i] = __ldg(V.steps + t0 + i);
  tilePrologue<THREADS>(pro, base, nRows, vec, xs);
  if (tid == 0) xs[nRows] = W(0);
  sweep.start();
  tileBarrier<WARPS>();
  const uint32_t nForward = steps[1], nSteps = steps[2];
  // Forward substitution (ilu/Solver.cpp:380-411); its last DEPTH steps copy
  // records of the backward sweep.
  auto forward = [&](auto isLong) {
    constexpr bool LONG = decltype(isLong)::value;
    auto begin = [](const Rec&, W was) { return was; };
    auto end = [](const Rec& r, W, W sum) { return DILU ? mul(sum, cvt<W>(r.diag())) : sum; };
    const uint32_t last = min(nForward, static_cast<uint32_t>(DEPTH));
    sweep.template run<LONG, DILU, LONG>(nForward - last, x, begin, end);
    sweep.template run<LONG, true, NT == 2>(last, x, begin, end);
  };
  if (NT == 2 && V.longForward) forward(std::bool_constant<NT == 2>{});
  else forward(std::false_type{});
  // Backward substitution (ilu/Solver.cpp:413-442).
  sweep.template run<NT == 2, true, NT == 2>(
      nSteps - nForward, x, [](const Rec&, W) { return W(0); },
      [](const Rec& r, W was, W sum) {
        const W iv = cvt<W>(r.diag());
        return DILU ? add(was, mul(sum, iv)) : mul(add(was, sum), iv);
      });
  tileStore<THREADS>(y, base, nRows, vec, xs);
}

// Vectors are stored in X; rows are computed in W, each new value rounded to
// X as it is stored (the working type of gauss-seidel/Solver.cpp:65-84).
template <class X, class W>
__device__ __forceinline__ W roundTo(W v) {
  return cvt<W>(cvt<X>(v));
}

// One Gauss-Seidel sweep of every tile (gauss-seidel/Solver.cpp:45-86): rows
// in ascending tile-local order, as the lower levels, each x_i = (seed_i -
// sum_j a_ij x_j) / d_i in tile-local order. The tile's x is [this sweep's
// values, the sweep-start values (unless they can be overwritten in place),
// halo, zero], the right-hand side follows in shared memory.
template <class MV, class X, class W, int NT, int WARPS, int DEPTH>
__global__ void __launch_bounds__(32 * WARPS) gsDirectKernel(DirectView V, SPro<X> pro, bool seedB,
                                                             const int* __restrict__ haloStart,
                                                             const int* __restrict__ haloSrc,
                                                             const X* __restrict__ xin, bool xinZero, bool inPlace,
                                                             bool dropHalo, X* __restrict__ xout, bool vec) {
  constexpr int THREADS = 32 * WARPS;
  using Rec = DirectRec<MV, NT>;
  using Steps = DirectSteps<MV, W, NT, WARPS, DEPTH>;
  extern __shared__ __align__(16) unsigned char smem[];
  const KState* st = pro.state();
  if (st && st->done) return;
  const int T = blockIdx.x, tid = threadIdx.x;
  const int base = V.tileStart[T], nRows = V.tileStart[T + 1] - base;
  const int h0 = haloStart[T], nHalo = haloStart[T + 1] - h0;
  unsigned char* x = smem + Steps::S::x;
  W* xs = reinterpret_cast<W*>(x);
  W* rhs = xs + V.xSlots;
  uint32_t* steps = reinterpret_cast<uint32_t*>(rhs + (V.maxRows + 3) / 4 * 4);
  Steps sweep(V, smem, T, steps + kDirectHead);
  const int t0 = V.stepStart[T], words = V.stepStart[T + 1] - t0;
  for (int i = tid; i < words; i += THREADS) steps[i] = __ldg(V.steps + t0 + i);
  W* start = xs + (inPlace ? 0 : nRows);
  W* halo = start + nRows;
  // Halo cells, four a thread: their source indices, then their values.
  for (int h = tid; h < nHalo; h += 4 * THREADS) {
    int src[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) src[j] = h + j * THREADS < nHalo ? __ldg(haloSrc + h0 + h + j * THREADS) : -1;
    W hv[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) hv[j] = src[j] >= 0 && !xinZero && !dropHalo ? cvt<W>(xin[src[j]]) : W(0);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (src[j] >= 0) halo[h + j * THREADS] = hv[j];
  }
  if (seedB || pro.kind != static_cast<int>(Prologue::Plain)) tilePrologue<THREADS>(pro, base, nRows, vec, rhs);
  if (xinZero) {
    for (int i = tid; i < nRows; i += THREADS) start[i] = W(0);
  } else {
    tilePrologue<THREADS>(SPro<X>{static_cast<int>(Prologue::Plain), xin, nullptr, nullptr, nullptr, nullptr}, base,
                          nRows, vec, start);
  }
  if (tid == 0) halo[nHalo] = W(0);
  sweep.start();
  tileBarrier<WARPS>();
  unsigned char* rhsBytes = reinterpret_cast<unsigned char*>(rhs);
  sweep.template run<NT == 2, true, NT == 2>(
      steps[2], x, [&](const Rec& r, W) { return seedB ? slotOf<W>(rhsBytes, r.row()) : cvt<W>(r.diag()); },
      [](const Rec& r, W, W sum) { return roundTo<X>(dvd(sum, cvt<W>(r.diag()))); });
  tileStore<THREADS>(xout, base, nRows, vec, xs);
}

// A solver's blocks from a plan's sources, the factor (or matrix) values F in
// tile-local CRS order and the diagonal inv in tile order; a record's row
// gives its diagonal. gridDim.y blocks a tile; a warp a step, or eight lanes
// (whose 16-byte words fill a line) where steps have less than 16 rows: a
// step is a chain of three loads, so what counts is steps in flight. Both
// plans of a Gauss-Seidel solver, with its wait, with one block a tile and a
// warp a step -> now: a chain of 4096 rows a tile, 16 tiles, 1018 us -> 35; a
// 96^3 grid in 148 tiles 147 us -> 57. An eight-lane step of 128 rows is
// slower than a warp's (16^3 in one tile: 48 us, 30).
template <class MV>
__global__ void __launch_bounds__(256) directPackKernel(const int* __restrict__ tileStart,
                                                        const int* __restrict__ stepStart,
                                                        const uint32_t* __restrict__ steps,
                                                        const uint32_t* __restrict__ stepRecord,
                                                        const uint32_t* __restrict__ stepUnit,
                                                        const int4* __restrict__ src, const int4* __restrict__ src2,
                                                        const uint32_t* __restrict__ tail,
                                                        const uint32_t* __restrict__ tail2, const MV* __restrict__ F,
                                                        const MV* __restrict__ inv, uint4* __restrict__ data,
                                                        int lanesLog2) {
  const int base = tileStart[blockIdx.x], lanes = 1 << lanesLog2, lane = threadIdx.x & (lanes - 1);
  auto val = [&](int e) { return e >= 0 ? F[e] : MV(0); };
  auto put = [&](char* out, uint32_t plane, const int4 s, uint32_t last) {
    if constexpr (sizeof(MV) == 4) {
      *reinterpret_cast<uint4*>(out) = make_uint4(__float_as_uint(val(s.x)), __float_as_uint(val(s.y)),
                                                  __float_as_uint(val(s.z)), static_cast<uint32_t>(s.w));
    } else {
      const double v0 = val(s.x), v1 = val(s.y), v2 = val(s.z);
      *reinterpret_cast<uint4*>(out) =
          make_uint4(__double2loint(v0), __double2hiint(v0), __double2loint(v1), __double2hiint(v1));
      *reinterpret_cast<uint4*>(out + plane) =
          make_uint4(__double2loint(v2), __double2hiint(v2), static_cast<uint32_t>(s.w), last);
    }
  };
  for (int i = stepStart[blockIdx.x] + kDirectHead + static_cast<int>((blockIdx.y * blockDim.x + threadIdx.x) >> lanesLog2);
       i < stepStart[blockIdx.x + 1]; i += static_cast<int>((gridDim.y * blockDim.x) >> lanesLog2)) {
    const uint32_t w = steps[i], rows = w & 0xFFu, nLong = (w >> kDirectLongShift) & 0xFFu;
    const DirectBlock<sizeof(MV)> at(w, (w & kDirectDiag) != 0);
    char* blk = reinterpret_cast<char*>(data + stepUnit[i]);
    for (uint32_t q = lane; q < rows; q += lanes) {
      const size_t p = stepRecord[i] + q;
      const uint32_t t = tail[p];
      put(blk + 16 * q, at.plane, src[p], t);
      const MV d = inv[base + (t >> 18)];  // the row, stored as 4 x row << 16
      char* tails = blk + at.tail;
      if constexpr (sizeof(MV) == 8) {
        if (w & kDirectDiag) reinterpret_cast<double*>(tails)[q] = d;
      } else {
        if (w & kDirectDiag) reinterpret_cast<uint2*>(tails)[q] = make_uint2(t, __float_as_uint(d));
        else reinterpret_cast<uint32_t*>(tails)[q] = t;
      }
      if (q < nLong) {
        put(blk + at.second + 16 * q, at.plane2, src2[p], tail2[p]);
        if (sizeof(MV) == 4) reinterpret_cast<uint32_t*>(blk + at.third)[q] = tail2[p];
      }
    }
  }
}

// ILU(0) / DILU factorisation of every tile (ilu/Solver.cpp:167-218) for
// patterns in which no entry (k, j) exists beside (i, k) and (i, j), written
// straight into the solver's blocks. Row i then takes, for its lower entries
// k in order, F_ik = A_ik / D_k and D_i -= F_ik F_ki; its other entries j only
// lose F_ik times an absent entry's 0, which is 0 or, for an F_ik that is not
// finite, NaN. The tile's D lies in shared memory, with each row's sum of
// those zeros (z: +0, -0 or NaN). Rows run level by level in the forward
// sweep's order, each thread a row; every gather is an index the host fixed.
// It replaces a factorisation that searched global memory for each F_ki and
// F_kj, a copy of the values, an inversion and a packing pass: on B200, 97 x
// 96 x 95 rows in 432 tiles, 535 + 5 + 49 us for those kernels, 123 us for
// this one (155 without the indices and values fetched ahead). What is left
// is the chain of a level: up to three dependent divisions and a barrier.
template <class MV, bool DILU>
__global__ void __launch_bounds__(128) iluFactorDirectKernel(
    const int* __restrict__ tileStart, const int* __restrict__ stepStart, const uint32_t* __restrict__ steps,
    const uint32_t* __restrict__ stepRecord, const uint32_t* __restrict__ stepUnit, const int* __restrict__ levelStart,
    const int4* __restrict__ levels, int stepShift, int maxRows, const int4* __restrict__ src,
    const int4* __restrict__ src2, const uint32_t* __restrict__ tail, const uint32_t* __restrict__ tail2,
    const int4* __restrict__ transposed, const int4* __restrict__ transposed2, const MV* __restrict__ A,
    const MV* __restrict__ diag, uint4* __restrict__ data) {
  extern __shared__ __align__(16) unsigned char smem[];
  MV* D = reinterpret_cast<MV*>(smem);
  MV* z = D + maxRows;
  const int T = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  const int base = tileStart[T], nRows = tileStart[T + 1] - base;
  for (int i = tid; i < nRows; i += 128) {
    D[i] = diag[base + i];
    z[i] = MV(0);
  }
  __syncthreads();
  auto put = [&](char* out, uint32_t plane, const MV (&v)[3], int slots, uint32_t last) {
    if constexpr (sizeof(MV) == 4) {
      *reinterpret_cast<uint4*>(out) = make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]),
                                                  static_cast<uint32_t>(slots));
    } else {
      *reinterpret_cast<uint4*>(out) =
          make_uint4(__double2loint(v[0]), __double2hiint(v[0]), __double2loint(v[1]), __double2hiint(v[1]));
      *reinterpret_cast<uint4*>(out + plane) =
          make_uint4(__double2loint(v[2]), __double2hiint(v[2]), static_cast<uint32_t>(slots), last);
    }
  };
  auto putTail = [&](char* tails, uint32_t q, uint32_t t, bool withDiag, MV inv) {
    if constexpr (sizeof(MV) == 8) {
      if (withDiag) reinterpret_cast<double*>(tails)[q] = inv;
    } else {
      if (withDiag) reinterpret_cast<uint2*>(tails)[q] = make_uint2(t, __float_as_uint(inv));
      else reinterpret_cast<uint32_t*>(tails)[q] = t;
    }
  };
  const int first = stepStart[T] + kDirectHead;
  const int nForward = static_cast<int>(steps[first - kDirectHead + 1]);
  const int4 none = make_int4(-1, -1, -1, 0);
  // Row q of a level: its indices, the values they gather, and its
  // elimination. Neither indices nor values depend on another row, so they
  // are fetched two and one levels ahead; only D and z wait for the barrier.
  struct Index {
    int4 s, r, s2, r2;
    uint32_t w, unit, t, t2;
  };
  struct Values {
    MV v[6], u[6];
  };
  auto index = [&](const int4 lv, int q, Index& x) {
    const bool on = q < (lv.y & 0xFFFF), two = q < (lv.y >> 16);
    const int step = lv.z + (q >> stepShift);
    x.w = on ? steps[step] : 0;
    x.unit = on ? stepUnit[step] : 0;
    x.t = on ? tail[lv.x + q] : 0;
    x.s = on ? src[lv.x + q] : none;
    x.r = on ? transposed[lv.w + q] : none;
    x.s2 = two ? src2[lv.x + q] : none;
    x.r2 = two ? transposed2[lv.w + q] : none;
    x.t2 = two ? tail2[lv.x + q] : 0;
  };
  auto gather = [&](const Index& x, Values& g) {
    const int e[6] = {x.s.x, x.s.y, x.s.z, x.s2.x, x.s2.y, x.s2.z}, et[6] = {x.r.x, x.r.y, x.r.z, x.r2.x, x.r2.y, x.r2.z};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      g.v[k] = e[k] >= 0 ? A[e[k]] : MV(0);
      g.u[k] = et[k] >= 0 ? A[et[k]] : MV(0);
    }
  };
  auto eliminate = [&](const int4 lv, int q, const Index& x, Values& g) {
    const int e[6] = {x.s.x, x.s.y, x.s.z, x.s2.x, x.s2.y, x.s2.z}, et[6] = {x.r.x, x.r.y, x.r.z, x.r2.x, x.r2.y, x.r2.z};
    const uint32_t sw = static_cast<uint32_t>(x.s.w), sw2 = static_cast<uint32_t>(x.s2.w);
    const uint32_t c[6] = {sw & 0xFFFFu, sw >> 16, x.t & 0xFFFFu, sw2 & 0xFFFFu, sw2 >> 16, x.t2};
    MV d = D[x.t >> 18], zi = MV(0);
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      if (e[k] < 0) continue;
      const MV dk = D[c[k] >> 2];
      if (DILU) {
        d = sub(d, dvd(mul(g.v[k], g.u[k]), dk));
      } else {
        g.v[k] = dvd(g.v[k], dk);
        const MV zk = mul(g.v[k], MV(0));
#pragma unroll
        for (int j = k + 1; j < 6; ++j)
          if (e[j] >= 0) g.v[j] = sub(g.v[j], zk);
        if (zi == zi && (zk != zk || signbit(zk))) zi = zk;
        d = sub(d, mul(g.v[k], et[k] >= 0 ? sub(g.u[k], z[c[k] >> 2]) : MV(0)));
      }
    }
    D[x.t >> 18] = d;
    z[x.t >> 18] = zi;
    const uint32_t at = static_cast<uint32_t>(q) & ((1u << stepShift) - 1);
    const DirectBlock<sizeof(MV)> blk(x.w, DILU);
    char* out = reinterpret_cast<char*>(data + x.unit);
    const MV lo[3] = {g.v[0], g.v[1], g.v[2]}, hi[3] = {g.v[3], g.v[4], g.v[5]};
    put(out + 16 * at, blk.plane, lo, x.s.w, x.t);
    putTail(out + blk.tail, at, x.t, DILU, DILU ? dvd(MV(1), d) : d);
    if (q < (lv.y >> 16)) {
      put(out + blk.second + 16 * at, blk.plane2, hi, x.s2.w, x.t2);
      if (sizeof(MV) == 4) reinterpret_cast<uint32_t*>(out + blk.third)[at] = x.t2;
    }
  };
  const int l0 = levelStart[T], l1 = levelStart[T + 1];
  auto level = [&](int l) { return l < l1 ? levels[l] : make_int4(0, 0, 0, 0); };
  int4 lv = level(l0), lv1 = level(l0 + 1);
  Index x, x1;
  Values g;
  index(lv, tid, x);
  index(lv1, tid, x1);
  gather(x, g);
  for (int l = l0; l < l1; ++l) {
    Values g1;
    gather(x1, g1);
    const int4 lv2 = level(l + 2);
    if (tid < (lv.y & 0xFFFF)) eliminate(lv, tid, x, g);
    x = x1;
    index(lv2, tid, x1);
    for (int q = tid + 128; q < (lv.y & 0xFFFF); q += 128) {  // wide levels
      Index xq;
      Values gq;
      index(lv, q, xq);
      gather(xq, gq);
      eliminate(lv, q, xq, gq);
    }
    g = g1;
    lv = lv1;
    lv1 = lv2;
    __syncthreads();
  }
  for (int i = tid; i < nRows; i += 128) D[i] = dvd(MV(1), D[i]);
  __syncthreads();
  // The backward records: a warp per step.
  const int stop = stepStart[T + 1];
#pragma unroll 2
  for (int i = first + nForward + (tid >> 5); i < stop; i += 4) {
    const uint32_t w = steps[i], rows = w & 0xFFu, longs = (w >> kDirectLongShift) & 0xFFu;
    const DirectBlock<sizeof(MV)> blk(w, true);
    char* out = reinterpret_cast<char*>(data + stepUnit[i]);
    for (uint32_t q = lane; q < rows; q += 32) {
      const size_t p = stepRecord[i] + q;
      const uint32_t t = tail[p];
      const MV zi = DILU ? MV(0) : z[t >> 18];
      auto val = [&](int e) { return e < 0 ? MV(0) : DILU ? A[e] : sub(A[e], zi); };
      const int4 s = src[p];
      const MV lo[3] = {val(s.x), val(s.y), val(s.z)};
      put(out + 16 * q, blk.plane, lo, s.w, t);
      putTail(out + blk.tail, q, t, true, D[t >> 18]);
      if (q < longs) {
        const int4 s2 = src2[p];
        const MV hi[3] = {val(s2.x), val(s2.y), val(s2.z)};
        put(out + blk.second + 16 * q, blk.plane2, hi, s2.w, tail2[p]);
        if (sizeof(MV) == 4) reinterpret_cast<uint32_t*>(out + blk.third)[q] = tail2[p];
      }
    }
  }
}

}  // namespace dev

// ---------------------------------------------------------------------------
namespace {

constexpr i64 kDirectFetchUnits = (i64(32) << 20) / 16;

dev::DirectView directView(const DeviceMatrix& A, const DirectPlan& P, const DBuf& data) {
  return dev::DirectView{A.tileStart.as<int>(),
                         P.stepStart.as<int>(),
                         P.steps.as<uint32_t>(),
                         P.stepUnit.as<uint32_t>(),
                         data.as<uint4>(),
                         static_cast<int>((P.maxXSlots + 3) / 4 * 4),
                         static_cast<int>(P.maxRows),
                         P.units >= kDirectFetchUnits,
                         P.longForward};
}

bool aligned16(std::initializer_list<const void*> ps) {
  uintptr_t bits = 0;
  for (const void* p : ps) bits |= reinterpret_cast<uintptr_t>(p);
  return (bits & 15u) == 0;
}

}  // namespace

size_t directBytes(const DirectPlan& P) { return 16 * std::max<size_t>(1, static_cast<size_t>(P.units)); }

void launchDirectPack(DeviceMatrix& A, const DirectPlan& P, DBuf& data, const void* F, const void* inv,
                      cudaStream_t s) {
  const int perTile = std::clamp(8 * A.numSMs / std::max<int>(1, A.P), 1, 32);
  const i64 sweeps = P.kind == RingKind::Ilu ? 2 : 1;
  const int lanesLog2 = sweeps * P.maxRows >= 16 * P.maxSteps ? 5 : 3;
  auto go = [&](auto zero) {
    using MV = decltype(zero);
    dev::directPackKernel<MV><<<dim3(A.P, perTile), 256, 0, s>>>(
        A.tileStart.as<int>(), P.stepStart.as<int>(), P.steps.as<uint32_t>(), P.stepRecord.as<uint32_t>(),
        P.stepUnit.as<uint32_t>(), P.src.as<int4>(), P.second ? P.src2.as<int4>() : nullptr, P.tail.as<uint32_t>(),
        P.second ? P.tail2.as<uint32_t>() : nullptr, static_cast<const MV*>(F), static_cast<const MV*>(inv), data.as<uint4>(),
        lanesLog2);
  };
  if (A.vt == DType::F32) go(0.0f);
  else go(0.0);
  checkLaunch("direct_pack");
}

size_t directFactorSmem(const DirectPlan& P, DType vt) { return 2 * static_cast<size_t>(P.maxRows) * dtypeSize(vt); }

void launchIluFactorDirect(DeviceMatrix& A, const DirectPlan& P, DBuf& data, bool dilu, cudaStream_t s) {
  if (!P.factors || P.dilu != dilu) fail(GR_EINVAL, "the plan does not factorise this matrix");
  const size_t smem = directFactorSmem(P, A.vt);
  const int stepShift = P.warps == 1 ? 5 : P.warps == 2 ? 6 : 7;
  auto go = [&](auto zero) {
    using MV = decltype(zero);
    auto kernel = dilu ? dev::iluFactorDirectKernel<MV, true> : dev::iluFactorDirectKernel<MV, false>;
    ensureDynamicSmem(reinterpret_cast<const void*>(kernel), smem);
    preferSharedCarveout(reinterpret_cast<const void*>(kernel));
    kernel<<<A.P, 128, smem, s>>>(
        A.tileStart.as<int>(), P.stepStart.as<int>(), P.steps.as<uint32_t>(), P.stepRecord.as<uint32_t>(),
        P.stepUnit.as<uint32_t>(), P.levelStart.as<int>(), P.levels.as<int4>(), stepShift, static_cast<int>(P.maxRows),
        P.src.as<int4>(), P.second ? P.src2.as<int4>() : nullptr, P.tail.as<uint32_t>(),
        P.second ? P.tail2.as<uint32_t>() : nullptr, P.transposed.as<int4>(),
        P.longForward ? P.transposed2.as<int4>() : nullptr, A.offDiag.as<MV>(), A.diag.as<MV>(), data.as<uint4>());
  };
  if (A.vt == DType::F32) go(0.0f);
  else go(0.0);
  checkLaunch("ilu_factor_direct");
}

namespace {
template <class MV, class W, int NT, bool DILU, int DEPTH>
auto iluDirectFor(int warps) {
  static_assert(dev::DirectShape<MV, NT, 32, DEPTH>::x ==
                    32 * DEPTH * (sizeof(MV) == 4 ? (NT == 2 ? 44 : 24) : (NT == 2 ? 72 : 40)),
                "directSmem's record size");
  return warps == 1   ? dev::iluDirectKernel<MV, W, NT, 1, DEPTH, DILU>
         : warps == 2 ? dev::iluDirectKernel<MV, W, NT, 2, DEPTH, DILU>
                      : dev::iluDirectKernel<MV, W, NT, 4, DEPTH, DILU>;
}
template <class MV, class W, int NT, bool DILU>
void iluDirectT(DeviceMatrix& A, const DirectPlan& P, i32 depth, const DBuf& data, const PrologueArgs& p, void* y,
                cudaStream_t s) {
  const size_t smem = directSmem(P, dtypeOf<MV>(), dtypeOf<W>(), depth);
  auto kernel = depth == 4 ? iluDirectFor<MV, W, NT, DILU, 4>(P.warps) : iluDirectFor<MV, W, NT, DILU, 8>(P.warps);
  ensureDynamicSmem(reinterpret_cast<const void*>(kernel), smem);
  preferSharedCarveout(reinterpret_cast<const void*>(kernel));
  dev::SPro<W> pro{static_cast<int>(p.kind), static_cast<const W*>(p.b), static_cast<const W*>(p.r),
                   static_cast<W*>(p.pOrS), static_cast<const W*>(p.v), p.st, p.stIndex};
  const bool vec = p.kind == Prologue::Plain ? aligned16({p.b, y}) : aligned16({p.r, p.pOrS, p.v, y});
  kernel<<<A.P, 32 * P.warps, smem, s>>>(directView(A, P, data), pro, static_cast<W*>(y), vec);
  checkLaunch("ilu_direct");
}
}  // namespace

void launchIluDirect(DeviceMatrix& A, const DirectPlan& P, i32 depth, const DBuf& data, bool dilu,
                     const PrologueArgs& pro, void* y, DType W, cudaStream_t s) {
  if (depth != 4 && depth != 8) fail(GR_EINVAL, "direct sweeps copy 4 or 8 steps ahead");
  auto go = [&](auto mv, auto w) {
    using MV = decltype(mv);
    using Wt = decltype(w);
    if (P.second) {
      if (dilu) iluDirectT<MV, Wt, 2, true>(A, P, depth, data, pro, y, s);
      else iluDirectT<MV, Wt, 2, false>(A, P, depth, data, pro, y, s);
    } else {
      if (dilu) iluDirectT<MV, Wt, 1, true>(A, P, depth, data, pro, y, s);
      else iluDirectT<MV, Wt, 1, false>(A, P, depth, data, pro, y, s);
    }
  };
  if (A.vt == DType::F32 && W == DType::F32) go(0.0f, 0.0f);
  else if (A.vt == DType::F32 && W == DType::F64) go(0.0f, 0.0);
  else if (A.vt == DType::F64 && W == DType::F64) go(0.0, 0.0);
  else fail(GR_EUNSUPPORTED, "ILU apply with float64 coefficients and float32 vectors");
}

namespace {
template <class MV, class X, class W, int NT>
auto gsDirectFor(int warps) {
  return warps == 1   ? dev::gsDirectKernel<MV, X, W, NT, 1, kDirectGsDepth>
         : warps == 2 ? dev::gsDirectKernel<MV, X, W, NT, 2, kDirectGsDepth>
                      : dev::gsDirectKernel<MV, X, W, NT, 4, kDirectGsDepth>;
}
template <class MV, class X, class W, int NT>
void gsDirectT(DeviceMatrix& A, const DirectPlan& P, const DBuf& data, const PrologueArgs& p, bool seedB,
               const void* xin, bool xinZero, void* xout, cudaStream_t s, bool dropHalo) {
  const size_t smem = directSmem(P, dtypeOf<MV>(), dtypeOf<W>(), kDirectGsDepth);
  auto kernel = gsDirectFor<MV, X, W, NT>(P.warps);
  ensureDynamicSmem(reinterpret_cast<const void*>(kernel), smem);
  preferSharedCarveout(reinterpret_cast<const void*>(kernel));
  dev::SPro<X> pro{static_cast<int>(p.kind), static_cast<const X*>(p.b), static_cast<const X*>(p.r),
                   static_cast<X*>(p.pOrS), static_cast<const X*>(p.v), p.st, p.stIndex};
  const bool vec = (p.kind == Prologue::Plain ? aligned16({p.b}) : aligned16({p.r, p.pOrS, p.v})) &&
                   aligned16({xinZero ? nullptr : xin, xout});
  kernel<<<A.P, 32 * P.warps, smem, s>>>(directView(A, P, data), pro, seedB, P.haloStart.as<int>(),
                                         P.haloSrc.as<int>(), static_cast<const X*>(xin), xinZero, P.gsInPlace,
                                         dropHalo, static_cast<X*>(xout), vec);
  checkLaunch("gs_direct");
}
}  // namespace

void launchGsDirect(DeviceMatrix& A, const DirectPlan& P, const DBuf& data, const PrologueArgs& pro, bool seedB,
                    const void* xin, bool xinZero, void* xout, DType X, DType W, cudaStream_t s, bool dropHalo) {
  if (P.kind == RingKind::Ilu) fail(GR_EINVAL, "not a Gauss-Seidel plan");
  if (P.kind == RingKind::GaussSeidelLower && !xinZero)
    fail(GR_EINVAL, "a lower-only Gauss-Seidel plan sweeps from x = 0 only");
  auto go = [&](auto mv, auto x, auto w) {
    using MV = decltype(mv);
    using Xt = decltype(x);
    using Wt = decltype(w);
    if (P.second) gsDirectT<MV, Xt, Wt, 2>(A, P, data, pro, seedB, xin, xinZero, xout, s, dropHalo);
    else gsDirectT<MV, Xt, Wt, 1>(A, P, data, pro, seedB, xin, xinZero, xout, s, dropHalo);
  };
  if (A.vt == DType::F32 && X == DType::F32 && W == DType::F32) go(0.0f, 0.0f, 0.0f);
  else if (A.vt == DType::F32 && X == DType::F32 && W == DType::F64) go(0.0f, 0.0f, 0.0);
  else if (A.vt == DType::F32 && X == DType::F64 && W == DType::F64) go(0.0f, 0.0, 0.0);
  else if (A.vt == DType::F64 && X == DType::F64 && W == DType::F64) go(0.0, 0.0, 0.0);
  else
    fail(GR_EUNSUPPORTED, "Gauss-Seidel: float64 coefficients need float64 vectors, and the working type must be "
                          "the vectors' type or float64 over float32 vectors");
}

}  // namespace gr
